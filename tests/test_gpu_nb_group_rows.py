"""LJ + Coulomb j-atom groups of rows of many and few blocks: one CTA a row has 16
warps up to 1,216 blocks, 8 above, and a row's entries keep their order either way,
so copies of a system in a batch get the forces it gets alone, bit for bit (the
sums are in fixed point and the groups of a row do not depend on other rows)."""
import numpy as np
import pytest

from test_gpu_nb_bodies import MODES, _lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,copies,periodic", [(2500, 15, 0), (2500, 16, 0), (2500, 16, 1), (2511, 16, 0)])
def test_groups_of_copies_equal_the_single_system(n, copies, periodic):
    torch = pytest.importorskip("torch")
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    pos, excl, box, par = _lattice(n, 5, periodic)
    kw = dict(Cutoff=9.0, Vdw14Scaling=0.5, Elec14Scaling=0.8, Dielectric=1.0, DoVdw=1, **MODES["same"])
    im = SystemImage([n], box, par["charge"], par["radius"], par["epsilon"], np.full(n, 2e-26), excl, pos=pos)
    out = []
    for image, k in ((im, 1), (SystemImage.concat([im] * copies), copies)):
        ctx = DeviceContext(image)
        ctx.set_list(1.0)
        ctx.set_nb(**kw)
        ctx.set_nb_groups(1)
        ctx.set_positions(np.tile(pos, (k, 1)))
        fd = torch.zeros((n * k, 3), dtype=torch.float64, device="cuda")
        ctx.compute_device(ffi.NB, fd.data_ptr())
        ctx.synchronize()
        assert ctx.nb_groups()[1] > 0
        out.append(fd.cpu().numpy())
        ctx.close()
    for c in range(copies):
        assert np.array_equal(out[1][c * n:(c + 1) * n], out[0])
