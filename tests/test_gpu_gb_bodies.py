"""The packed GB tile bodies at the sizes where they can go wrong: blocks with one
atom, exactly full and one over, odd and even tile counts per row, masked and
unmasked single tiles, near and far tile pairs, all pairs and switched cutoffs,
force-only and energy passes, against the FP64 oracle.  Tolerances as the parity
tests' (FP32 pair arithmetic): energies 1e-6, forces 1e-5 relative RMS."""
import numpy as np
import pytest

from conftest import rel_err, rel_rms

pytestmark = pytest.mark.gpu


def _chain(n, seed):
    """n atoms along a slowly turning chain, 1.5 A apart, bonded as a polymer: with n
    in the hundreds its ends lie beyond any exp threshold, its neighbours in contact."""
    rng = np.random.default_rng(seed)
    t = np.arange(n)
    pos = np.stack([1.2 * t, 4.0 * np.sin(0.35 * t), 4.0 * np.cos(0.35 * t)], 1) + rng.uniform(-0.1, 0.1, (n, 3))
    pos = pos[rng.permutation(n)] if n % 2 else pos      # slots and atom order unrelated, or alike
    d = np.linalg.norm(pos[:, None] - pos[None], axis=-1)
    i, j = np.nonzero(np.triu(d < 4.6, 1))
    bo = np.where(d[i, j] < 2.4, 1, np.where(d[i, j] < 3.6, 2, 3))
    par = dict(charge=rng.uniform(-0.6, 0.6, n), radius=rng.uniform(0.6, 1.9, n), epsilon=rng.uniform(1, 3, n) * 1e-11,
               gb_radius=rng.uniform(1.1, 1.9, n), gb_vj=rng.uniform(5.0, 20.0, n),
               gb_terms123=rng.uniform(-95.0, -80.0, n))
    return pos, np.stack([i, j, bo], 1).astype(np.int32), par


@pytest.mark.parametrize("cut", [None, 12.0])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 96, 129, 300])
def test_gb_bodies_match_oracle(n, cut):
    torch = pytest.importorskip("torch")
    from oracle import pdoracle as O
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    pos, excl, par = _chain(n, n)
    c, i, still = (999.0, 998.0, 999.0) if cut is None else (cut, cut - 3.0, 8.0)
    kw = dict(Cutoff=c, InnerCutoff=i, VdwCutoff=c, VdwInnerCutoff=i, Vdw14Scaling=0.5, Elec14Scaling=0.8,
              DielectricSolute=1.0, DielectricSolvent=80.0, GbsaStillCutoff=still, ExpApproxThreshold=-4.0,
              BornRadiusOffset=0.0)
    im = SystemImage([n], np.zeros(3), par["charge"], par["radius"], par["epsilon"], np.full(n, 2e-26), excl,
                     gb_radius=par["gb_radius"], gb_vj=par["gb_vj"], gb_terms123=par["gb_terms123"], pos=pos)
    ctx = DeviceContext(im)
    ctx.set_list(1.0)
    ctx.set_gb(P4=15.236, P5=1.254, **kw)
    ctx.set_positions(pos)
    f = np.zeros((n, 3))
    e = ctx.compute(ffi.GB, f)[0]
    fd = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    ctx.compute_device(ffi.GB, fd.data_ptr())       # the force-only pass
    ctx.synchronize()
    born = ctx.born_radii()
    ctx.close()
    s = O.OracleSystem(pos, par["charge"], par["radius"], par["epsilon"], excl)
    gp = O.gb_params(P1=0.073, P2=0.921, P3=6.211, P4=15.236, P5=1.254, ListCutoff=c + 1.0, **kw)
    re, rf, rb = O.gb_forces(s, gp, par["gb_radius"], par["gb_vj"], par["gb_terms123"])
    assert np.max(np.abs(born / rb - 1)) < 1e-6
    for key, r in (("vdw", re[1]), ("elec", re[2]), ("pol", re[3])):
        assert abs(e[key] - r) <= 1e-6 * (abs(re[1]) + abs(re[2]) + abs(re[3])), (key, e[key], r)
    if n > 1:
        assert rel_rms(f, rf) <= 1e-5 and rel_rms(fd.cpu().numpy(), rf) <= 1e-5
