"""Where the list build leaves the NB j-atom groups out (periodic boxes whose tiles nearly
all need an image per pair) and where it builds them: the same forces as on tiles alone on
both sides of the line, cubic and thin boxes (FP32 sums over the same pairs in another
order: 1e-5 relative RMS, the parity tests' force tolerance)."""
import numpy as np
import pytest

from conftest import rel_rms

pytestmark = pytest.mark.gpu


# list radius 8 A: half of a cubic box's block pairs share an image from L = 29.8 A on
@pytest.mark.parametrize("edges,built", [((24.0, 24.0, 24.0), False), ((28.0, 28.0, 28.0), False), ((33.0, 33.0, 33.0), True),
                                         ((20.0, 60.0, 60.0), False), ((40.0, 40.0, 26.0), True)])
def test_forces_on_both_sides_of_the_rule(edges, built):
    torch = pytest.importorskip("torch")
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    rng = np.random.default_rng(int(sum(edges)))
    m = [int(e / 2.6) for e in edges]
    g = np.stack(np.meshgrid(*[np.arange(k) for k in m], indexing="ij"), -1).reshape(-1, 3)
    n = len(g)
    pos = g * (np.array(edges) / m) + rng.uniform(-0.3, 0.3, (n, 3))
    im = SystemImage([n], np.array(edges), rng.uniform(-0.6, 0.6, n), rng.uniform(0.0, 1.6, n), rng.uniform(1, 3, n) * 1e-11,
                     np.full(n, 2e-26), np.zeros((0, 3), np.int32), pos=pos)
    kw = dict(Cutoff=7.0, InnerCutoff=5.5, VdwCutoff=7.0, VdwInnerCutoff=5.5, EnergySwitch=1, ForceSwitch=0, DoVdw=1, DoElec=1,
              Vdw14Scaling=0.5, Elec14Scaling=0.8, Dielectric=1.0)
    out = []
    for on in (1, 0):
        ctx = DeviceContext(im)
        ctx.set_list(1.0)
        ctx.set_nb(**kw)
        ctx.set_nb_groups(on)
        ctx.set_positions(pos)
        fd = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
        ctx.compute_device(ffi.NB, fd.data_ptr())
        ctx.synchronize()
        assert (ctx.nb_groups()[1] > 0) == bool(on and built)
        out.append(fd.cpu().numpy())
        ctx.close()
    assert rel_rms(out[0], out[1]) <= 1e-5
