"""Born sums of atoms of one type: the errors of their pairs average out.

P4 V is chosen to lie in the middle between two FP32 numbers, so that a volume rounded
with the factor P4 in it would shift every sum of every atom by 5.9e-8 of itself.
Rounded pair by pair, a sum of some 200 terms is off by 4e-7 at most and the mean over
216 atoms, whose errors are independent, by 1e-8; 2.5e-8 is allowed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("check_skin", [True, False])
def test_mean_error_of_the_born_sums(check_skin):
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    rng = np.random.default_rng(1)
    g = np.stack(np.meshgrid(*[np.arange(6)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = 3.5 * g + rng.uniform(-0.2, 0.2, g.shape)       # no pair in close contact: CCF = 1
    n = len(pos)
    P4 = 15.25
    v = (16.8 + 0.1 * rng.random(4000)).astype(np.float32)     # (P4 V just above 256: the widest spacing)
    pv = P4 * v.astype(np.float64)
    V = float(v[np.argmax(np.abs(pv.astype(np.float32) - pv) / pv)])
    assert abs(float(np.float32(P4 * V)) - P4 * V) / (P4 * V) > 5.5e-8
    terms = np.full(n, -60.0)
    im = SystemImage([n], np.zeros(3), rng.uniform(-0.5, 0.5, n), np.full(n, 1.5), np.full(n, 2e-11), np.full(n, 2e-26),
                     np.zeros((0, 3), np.int32), gb_radius=np.full(n, 1.4), gb_vj=np.full(n, V), gb_terms123=terms, pos=pos)
    ctx = DeviceContext(im)
    ctx.set_list(1.0, check_skin=check_skin)
    ctx.set_gb(Cutoff=999.0, InnerCutoff=998.0, VdwCutoff=999.0, VdwInnerCutoff=998.0, Vdw14Scaling=0.5, Elec14Scaling=0.8,
               DielectricSolute=1.0, DielectricSolvent=80.0, GbsaStillCutoff=999.0, ExpApproxThreshold=-4.0,
               BornRadiusOffset=0.0, P4=P4, P5=1.254)
    ctx.set_positions(pos)
    ctx.compute(ffi.GB)
    born = ctx.born_radii()
    ctx.close()
    econv = (6.0221418e23 / 4184.0) * 1.60217645e-19 ** 2 / (4.0 * np.pi * 8.854187817e-12 * 1e-10)
    got = -0.5 * econv / born - terms
    d = pos[:, None] - pos[None]
    r2 = (d * d).sum(-1)
    np.fill_diagonal(r2, np.inf)
    ref = P4 * V * (1.0 / r2 ** 2).sum(1)
    err = (got - ref) / ref
    assert np.abs(err).max() <= 4e-7 and abs(err.mean()) <= 2.5e-8, (err.mean(), np.abs(err).max())
