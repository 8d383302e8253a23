"""Monte Carlo energies after a move onto another atom: the partial update reports
what a full evaluation of the same positions reports, keeps its reference, and goes
on from it (PD's overlapping trial moves come back as a huge energy; here the fixed
point's range is a status)."""
import numpy as np
import pytest

from conftest import rel_err
from helpers import nb_kwargs

pytestmark = pytest.mark.gpu


def _context(d):
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    ctx = DeviceContext(SystemImage._from_fixture(d))
    ctx.set_list(2.0)
    ctx.set_nb(**nb_kwargs(d, "nb"))
    ctx.set_positions(d["pos"])
    return ctx


def _status(call):
    from pd_gb300 import ffi
    try:
        call()
    except ffi.PDGPUError as e:
        return e.status
    return 0


@pytest.mark.parametrize("name", ["water_c1", "peptide30"])
@pytest.mark.parametrize("gap", [0.02, 0.2, 0.4, 0.5])
@pytest.mark.parametrize("pairs", [1, 2])
def test_an_overlapping_move_reports_the_status_of_a_full_evaluation(goldens, name, gap, pairs):
    from pd_gb300 import ffi
    d = goldens[name]
    ctx = _context(d)
    e0 = ctx.nb_energy_full()[0]
    # atoms with an LJ core moved to `gap` A from others far away in the sequence
    core = np.flatnonzero((d["radius"] > 1.0) & (d["epsilon"] > 0))
    pos = d["pos"].copy()
    for k in range(pairs):
        pos[core[k]] = d["pos"][core[-1 - 10 * k]] + gap / np.sqrt(3.0)
    ctx.set_positions(pos)
    full = _status(lambda: (ctx.rebuild_list(), ctx.compute(ffi.NB)))
    assert full != 0
    for _ in range(2):
        assert _status(ctx.nb_energy_update) == full
    # back: the reference is the old one
    ctx.set_positions(d["pos"])
    e1, n = ctx.nb_energy_update()
    assert n == 0 and e1[0] == e0
    # and an ordinary move is again what a full evaluation gives
    pos = d["pos"].copy()
    pos[core[0]] += 0.05
    ctx.set_positions(pos)
    e2, n = ctx.nb_energy_update()
    ctx.rebuild_list()
    f2 = ctx.compute(ffi.NB)[0]
    assert n == 1 and rel_err(e2[0]["vdw"], f2["vdw"]) <= 1e-7 and rel_err(e2[0]["elec"], f2["elec"]) <= 1e-7
    ctx.close()


def test_a_move_to_a_non_finite_position_is_reported(goldens):
    d = goldens["peptide30"]
    ctx = _context(d)
    e0 = ctx.nb_energy_full()[0]
    pos = d["pos"].copy()
    pos[7, 1] = np.nan
    ctx.set_positions(pos)
    assert _status(ctx.nb_energy_update) == -5         # PDGPU_ERR_NAN
    ctx.set_positions(d["pos"])
    assert ctx.nb_energy_update()[0][0] == e0
    ctx.close()


def test_container_energies_after_an_overlapping_move(goldens):
    import pd_gb300 as pdg
    d = goldens["water_c1"]
    ws = pdg.WorkSpace(pdg.SystemImage._from_fixture(d))
    ws.Padding = 2.0
    ff = pdg.Forcefield(ws)
    nb = pdg.FF_NonBonded_GPU(ws)
    for k, v in nb_kwargs(d, "nb").items():
        setattr(nb, k, v)
    nb.AutoScaling14 = False
    nb.UsePartialRecalc = True
    ff.add(nb)
    ff.calcEnergies()
    e0 = ws.ene.epot
    old = ws.cur.p[0].copy()
    ws.cur.p[0] = ws.cur.p[300] + 0.1
    assert _status(ff.calcEnergies) != 0
    ws.cur.p[0] = old
    ff.calcEnergies()
    assert ws.ene.epot == e0
    ws.close()


def test_container_energies_after_new_parameters(goldens):
    """Per-atom parameters changed between two partial recalculations: the next energy is
    of the new ones (1e-9: both are sums of the same pairs)."""
    import pd_gb300 as pdg
    d = goldens["peptide30"]
    ws = pdg.WorkSpace(pdg.SystemImage._from_fixture(d))
    ws.Padding = 2.0
    ff = pdg.Forcefield(ws)
    nb = pdg.FF_NonBonded_GPU(ws)
    for k, v in nb_kwargs(d, "nb").items():
        setattr(nb, k, v)
    nb.AutoScaling14 = False
    nb.UsePartialRecalc = True
    ff.add(nb)
    ff.calcEnergies()
    e0 = ws.ene.epot
    ws.context().update_params(charge=0.9 * d["charge"])
    ws.cur.p[3] += 0.02
    ff.calcEnergies()
    e1 = ws.ene.epot
    nb.UsePartialRecalc = False
    ff.calcEnergies()
    assert e1 != e0 and rel_err(e1, ws.ene.epot) <= 1e-9
    ws.close()
