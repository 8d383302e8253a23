"""The packed gradient bodies at the sizes where they can go wrong (one atom, full
and part blocks, masked and plain tiles), with all-inside tiles found by the list
(displacement check on) and at run time (check off), all pairs and switched
cutoffs: central differences of the oracle's FP64 energy.  Tolerance as the
gradient tests': |g - fd| <= 1e-4 |fd| + 1e-6 max|g|."""
import numpy as np
import pytest

from test_gpu_adjoint import ABS, REL, STEP
from test_gpu_gb_bodies import _chain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cut", [None, 12.0])
@pytest.mark.parametrize("check", [True, False])
@pytest.mark.parametrize("n", [1, 2, 33, 64, 97, 200])
def test_gb_gradient_bodies_match_finite_differences(n, check, cut):
    from oracle import pdoracle as O
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    pos, excl, par = _chain(n, n)
    c, i, still = (999.0, 998.0, 999.0) if cut is None else (cut, cut - 3.0, 8.0)
    # (every pair above the exp threshold: differences across its jump do not converge)
    kw = dict(Cutoff=c, InnerCutoff=i, VdwCutoff=c, VdwInnerCutoff=i, Vdw14Scaling=0.5, Elec14Scaling=0.8,
              DielectricSolute=1.0, DielectricSolvent=80.0, GbsaStillCutoff=still, ExpApproxThreshold=-1e30,
              BornRadiusOffset=0.0)
    im = SystemImage([n], np.zeros(3), par["charge"], par["radius"], par["epsilon"], np.full(n, 2e-26), excl,
                     gb_radius=par["gb_radius"], gb_vj=par["gb_vj"], gb_terms123=par["gb_terms123"], pos=pos)
    ctx = DeviceContext(im)
    ctx.set_list(1.0, check_skin=check)
    ctx.set_gb(P4=15.236, P5=1.254, **kw)
    ctx.set_positions(pos)
    E, g = ctx.param_grad(ffi.GB)
    ctx.close()

    def energy(p):
        s = O.OracleSystem(pos, p["charge"], p["radius"], p["epsilon"], excl)
        gp = O.gb_params(P1=0.073, P2=0.921, P3=6.211, P4=15.236, P5=1.254, ListCutoff=c + 1.0, **kw)
        e = O.gb_forces(s, gp, p["gb_radius"], p["gb_vj"], p["gb_terms123"])[0]
        return e[1] + e[2] + e[3]

    e0 = energy(par)
    assert abs(E[0]["vdw"] + E[0]["elec"] + E[0]["pol"] - e0) <= 2e-6 * abs(e0)
    rng = np.random.default_rng(n)
    for name in STEP:
        scale = np.abs(g[name]).max()
        for a in rng.choice(n, min(n, 3), replace=False):
            h = STEP[name][0] * (abs(par[name][a]) if STEP[name][1] else 1.0)
            d = []
            for s in (1.0, -1.0):
                p = {k: v.copy() for k, v in par.items()}
                p[name][a] += s * h
                d.append(energy(p))
            fd = (d[0] - d[1]) / (2.0 * h)
            # (FP64 differences carry the rounding of the whole energy)
            assert abs(g[name][a] - fd) <= REL * abs(fd) + ABS * scale + 1e-15 * abs(e0) / h, (name, int(a), g[name][a], fd)
