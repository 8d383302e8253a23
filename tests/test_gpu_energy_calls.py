"""Energy calls that read no forces leave out the passes that only form forces: the
same energies, bit for bit, as the call with forces (the energies' passes are the
same launches), whatever ran before, and forces afterwards as without it."""
import numpy as np
import pytest

from helpers import gb_kwargs, nb_kwargs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,tag,what", [("water_c1", "nb", "NB"), ("water_c1", "nbfswitch", "NB"),
                                           ("peptide30", "gb", "GB"), ("peptide30", "gb", "GB|PD_ENERGIES"),
                                           ("peptide120", "gb", "GB|SA|BONDED")])
def test_energies_without_forces(goldens, name, tag, what):
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    flags = 0
    for w in what.split("|"):
        flags |= getattr(ffi, w)
    d = goldens[name]
    n = len(d["pos"])

    def context():
        ctx = DeviceContext(SystemImage._from_fixture(d))
        ctx.set_list(float(d["cfg_padding"][0]))
        if tag == "gb":
            ctx.set_gb(**gb_kwargs(d))
        else:
            ctx.set_nb(**nb_kwargs(d, tag))
        ctx.set_positions(d["pos"])
        return ctx

    ctx, ref = context(), context()
    f, f0 = np.zeros((n, 3)), np.zeros((n, 3))
    e0 = ref.compute(flags, f0)
    assert ctx.compute(flags) == e0
    assert ctx.compute(flags, f) == e0
    assert ctx.compute(flags) == e0
    assert np.array_equal(f, f0) and np.abs(f0).max() > 0
    ctx.close()
    ref.close()


@pytest.mark.parametrize("n,periodic,cutoff", [(2, 0, 9.0), (33, 0, 9.0), (65, 1, 9.0), (300, 1, 9.0), (2500, 1, 5.0),
                                              (2500, 0, 12.0)])
def test_energy_lists_of_any_length(n, periodic, cutoff):
    """Pair lists from a single pair to full parts, odd remainders passed on between an
    item's parts, tile path and groups, against the FP64 oracle: a few roundings of
    2^-46 per pair and one of 2^-32 kcal/mol per item (below 6e-6 kcal/mol in all,
    see test_gpu_energy_precision)."""
    from oracle import pdoracle as O
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    from test_gpu_energy_precision import TOL
    from test_gpu_nb_bodies import _lattice
    pos, excl, box, par = _lattice(n, 11 * n + periodic, periodic)
    kw = dict(Cutoff=cutoff, InnerCutoff=cutoff - 2.0, VdwCutoff=cutoff, VdwInnerCutoff=cutoff - 2.0, Vdw14Scaling=0.5,
              Elec14Scaling=0.8, Dielectric=1.0, DoVdw=1, DoElec=1, EnergySwitch=1, ForceSwitch=0)
    s = O.OracleSystem(pos, par["charge"], par["radius"], par["epsilon"], excl, tuple(box))
    ref = O.nonbonded(s, O.nb_params(ListCutoff=cutoff + 1.0, **kw))[0]
    im = SystemImage([n], box, par["charge"], par["radius"], par["epsilon"], np.full(n, 2e-26), excl, pos=pos)
    for groups in (1, 0):
        ctx = DeviceContext(im)
        ctx.set_list(1.0)
        ctx.set_nb(**kw)
        ctx.set_nb_groups(groups)
        ctx.set_positions(pos)
        e = ctx.compute(ffi.NB)[0]
        ctx.close()
        for key, r in (("vdw", ref[1]), ("elec", ref[2]), ("virial", ref[7])):
            assert abs(e[key] - r) <= TOL + 2.0 ** -40 * abs(r), (key, e[key], r)
