"""FF_NonBonded energies in double-float arithmetic against the oracle's FP64 sums.

A pair's energy carries a few roundings of 2^-46 of its terms (|terms| below 100
kcal/mol outside clashes), a work item's sum one rounding to 2^-32 kcal/mol: with
at most 8e5 pairs and 5e3 items, 8e5 x 100 x 2^-44 + 5e3 x 2^-32 < 6e-6 kcal/mol
even if every rounding had one sign.
"""
import numpy as np
import pytest

from helpers import nb_kwargs, nb_params, oracle_system

pytestmark = pytest.mark.gpu

KCAL = 4184.0 / 6.0221418e23
TOL = 6e-6 * KCAL


@pytest.mark.parametrize("groups", [1, 0])
@pytest.mark.parametrize("name,tag", [("water_c1", "nb"), ("water_c1", "nbfswitch"), ("water_c1", "nbnormal"),
                                      ("water_c1", "nbvdwsplit"), ("peptide30_ap", "nb"), ("peptide120", "nb")])
def test_nb_energies_match_fp64(goldens, name, tag, groups):
    from oracle import pdoracle as O
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    d = goldens[name]
    ctx = DeviceContext(SystemImage._from_fixture(d))
    ctx.set_list(float(d["cfg_padding"][0]))
    ctx.set_positions(d["pos"])
    ctx.set_nb(**nb_kwargs(d, tag))
    ctx.set_nb_groups(groups)
    e = ctx.compute(ffi.NB)[0]
    ctx.close()
    ref = O.nonbonded(oracle_system(d), nb_params(d, tag))[0]
    # fixtures with clashing atoms hold a few larger terms: 2^-44 of the energies' own size covers them
    for key, r in (("vdw", ref[1]), ("elec", ref[2]), ("virial", ref[7])):
        assert abs(e[key] - r) <= TOL + 2.0 ** -40 * abs(r), (key, e[key] / KCAL, r / KCAL)


def test_nb_energies_at_exact_cutoffs():
    """Pairs exactly at unswitched cutoffs: r = Cutoff counts (r^2 <= Cutoff^2), r = VdwCutoff
    does not (r < VdwCutoff), as PD decides in FP64."""
    from oracle import pdoracle as O
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    n = 70                                   # three blocks, the last one padded
    pos = np.zeros((n, 3))
    pos[:, 0] = 3.0 * np.arange(n)
    q = np.where(np.arange(n) % 3 == 0, 0.4, -0.2)
    rad, eps = np.full(n, 1.7), np.full(n, 3.0e-11)
    kw = dict(Cutoff=12.0, InnerCutoff=12.0, VdwCutoff=9.0, VdwInnerCutoff=9.0, Vdw14Scaling=1.0, Elec14Scaling=1.0,
              Dielectric=1.0, EnergySwitch=0, ForceSwitch=0)
    im = SystemImage([n], np.zeros(3), q, rad, eps, np.full(n, 2e-26), np.zeros((0, 3), np.int32), pos=pos)
    ctx = DeviceContext(im)
    ctx.set_list(1.0)
    ctx.set_nb(DoVdw=1, DoElec=1, **kw)
    ctx.set_positions(pos)
    e = ctx.compute(ffi.NB)[0]
    ctx.close()
    ref = O.nonbonded(O.OracleSystem(pos, q, rad, eps, np.zeros((0, 3), np.int32)), O.nb_params(ListCutoff=13.0, **kw))[0]
    assert abs(e["vdw"] - ref[1]) <= TOL and abs(e["elec"] - ref[2]) <= TOL
