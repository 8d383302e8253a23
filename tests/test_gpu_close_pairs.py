"""Forces of close pairs in an evaluation with energies: r^2 is rounded once.

Isolated pairs of uncharged atoms 1.5 to 3 A apart, chosen so that a sum of squares
rounded term by term comes out too large by 0.75 units in its last place or more.  The
repulsion goes with r^-14, so such a sum would leave every force too small, by 7 x 0.75
x 6e-8 (the smallest such unit) = 3e-7 of it on average.  Rounded once, r^2 is as often
too large as too small, and half a unit at most: the mean error of the forces is then
that of the reciprocal root and the products behind it, which do not know of the choice;
1.2e-7 is allowed for them (14 x 2^-24 / sqrt(N), and a bias of the root of 1e-8 x 12)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32


def _plain_r2(d):
    """d: FP32 components -> fl(fma(z, z, fma(y, y, fl(x x))))"""
    x, y, z = (d[:, k].astype(np.float64) for k in range(3))
    s = (x * x).astype(F).astype(np.float64)
    s = (y * y + s).astype(F).astype(np.float64)
    return (z * z + s).astype(F).astype(np.float64)


def test_mean_force_error_of_close_pairs():
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    rng = np.random.default_rng(5)
    u = rng.standard_normal((400_000, 3))
    u = (u / np.linalg.norm(u, axis=1)[:, None] * rng.uniform(1.5, 3.0, (len(u), 1)))
    # components on a grid of 2^-21 A: exact in FP32, and as differences of the positions below
    u = np.round(u * 2.0 ** 21) / 2.0 ** 21
    r2 = (u * u).sum(1)
    ulp = np.spacing(r2.astype(F)).astype(np.float64)
    u = u[(_plain_r2(u.astype(F)) - r2) / ulp >= 0.75][:600]
    assert len(u) == 600
    m = 9
    site = np.stack(np.unravel_index(np.arange(len(u)), (m, m, m)), 1) * 20.0
    pos = np.empty((2 * len(u), 3))
    pos[0::2] = site
    pos[1::2] = site + u
    n = len(pos)
    radius, eps = np.full(n, 1.75), np.full(n, 2.0e-11)
    im = SystemImage([n], np.zeros(3), np.zeros(n), radius, eps, np.full(n, 2e-26), np.zeros((0, 3), np.int32),
                     gb_radius=np.full(n, 0.1), gb_vj=np.zeros(n), gb_terms123=np.full(n, -60.0), pos=pos)
    ctx = DeviceContext(im)
    ctx.set_list(1.0)
    ctx.set_gb(Cutoff=12.0, InnerCutoff=10.0, VdwCutoff=12.0, VdwInnerCutoff=10.0, Vdw14Scaling=0.5, Elec14Scaling=0.8,
               DielectricSolute=1.0, DielectricSolvent=80.0, GbsaStillCutoff=10.0, ExpApproxThreshold=-4.0,
               BornRadiusOffset=0.0, P4=15.236, P5=1.254)
    ctx.set_positions(pos)
    f = np.zeros((n, 3))
    ctx.compute(ffi.GB, f)
    ctx.close()
    r2 = (u * u).sum(1)
    B = (3.5 * 3.5 / r2) ** 3
    # eps (A - 2B) in kcal/mol, force in N along u on the second atom; the parameters as the
    # kernel holds them (FP32)
    se2 = np.float64(F(eps[0] * np.sqrt(6.0221418e23 / 4184.0))) ** 2
    g = 12.0 * se2 * (B * B - B) / r2 * (4184.0 / 6.0221418e23) / 1e-10
    keep = np.abs(B - 1.0) > 0.3                       # (not where repulsion and attraction cancel)
    got = (f[1::2] * u).sum(1) / r2
    err = ((got - g) / g)[keep]
    assert keep.sum() > 400 and abs(err.mean()) <= 1.2e-7, (err.mean(), err.std(), keep.sum())
