"""Successive Forcefield calls on one WorkSpace: the list and the settings are kept
between calls, and every call still gives what a fresh WorkSpace gives."""
import numpy as np
import pytest

from conftest import rel_err, rel_rms
from helpers import nb_kwargs

pytestmark = pytest.mark.gpu


def _nb(goldens, name, padding=1.0):
    import pd_gb300 as pdg
    d = goldens[name]
    ws = pdg.WorkSpace(pdg.SystemImage._from_fixture(d))
    ws.Padding = padding
    ff = pdg.Forcefield(ws)
    nb = pdg.FF_NonBonded_GPU(ws)
    for k, v in nb_kwargs(d, "nb").items():
        setattr(nb, k, v)
    nb.AutoScaling14 = False
    ff.add(nb)
    return ws, ff, nb


def _same(ws, goldens, name, settings=()):
    """this WorkSpace's results against a fresh one at the same positions and settings"""
    fresh, ff, nb = _nb(goldens, name, ws.Padding)
    for k, v in settings:
        setattr(nb, k, v)
    fresh.cur.p[:] = ws.cur.p
    ff.calcForces()
    assert rel_err(ws.ene.epot_vdw, fresh.ene.epot_vdw) <= 1e-9 and rel_err(ws.ene.epot_elec, fresh.ene.epot_elec) <= 1e-9
    assert rel_rms(ws.cur.f, fresh.cur.f) <= 5e-6          # FP32 rounding about other block centres
    fresh.close()


@pytest.mark.parametrize("name", ["peptide30", "water_c1"])
def test_moves_of_any_size_between_calls(goldens, name):
    ws, ff, nb = _nb(goldens, name)
    rng = np.random.default_rng(2)
    for amplitude in (0.0, 0.05, 0.05, 0.4, 0.0, 2.0, 0.3, 0.02, 0.02):
        # (rigid shifts per block of atoms: no two atoms come onto one another)
        ws.cur.p += amplitude * rng.uniform(-1, 1, 3)
        ff.calcForces()
        _same(ws, goldens, name)


def test_list_is_kept_and_results_do_not_enter_the_checksum(goldens):
    ws, ff, nb = _nb(goldens, "peptide30")
    ff.calcForces()
    before = nb.calcCheckSum()
    slots = ws.context().list_slots()
    n0 = ws.context().kernel_launches()
    ff.calcForces()
    assert nb.calcCheckSum() == before and nb.epot_vdw != 0.0
    assert ws.context().kernel_launches() - n0 <= 6          # pack, records, pairs, forces: no list build
    assert np.array_equal(ws.context().list_slots(), slots)


def test_settings_changed_between_calls(goldens):
    ws, ff, nb = _nb(goldens, "peptide30")
    ff.calcForces()
    nb.Cutoff = nb.VdwCutoff = 11.0
    ff.calcForces()
    _same(ws, goldens, "peptide30", [("Cutoff", 11.0), ("VdwCutoff", 11.0)])
    ws.context().set_nb(**dict(nb._nb_kwargs(), Cutoff=8.0, InnerCutoff=6.0))   # behind the container's back
    ff.calcForces()
    _same(ws, goldens, "peptide30", [("Cutoff", 11.0), ("VdwCutoff", 11.0)])
    ws.close()
    ff.calcForces()
    _same(ws, goldens, "peptide30", [("Cutoff", 11.0), ("VdwCutoff", 11.0)])


def test_partial_recalculation_with_two_containers(goldens):
    """Two containers with different settings take turns on one WorkSpace: each
    energy is that of its own settings, whoever took the last reference."""
    import pd_gb300 as pdg
    ws, ff, nb = _nb(goldens, "peptide30")
    ff2 = pdg.Forcefield(ws)
    nb2 = pdg.FF_NonBonded_GPU(ws)
    for k, v in nb_kwargs(goldens["peptide30"], "nb").items():
        setattr(nb2, k, v)
    nb2.AutoScaling14 = False
    nb2.Cutoff = nb2.VdwCutoff = 10.5
    ff2.add(nb2)
    rng = np.random.default_rng(3)
    for k, (f, n) in enumerate([(ff, nb), (ff, nb), (ff2, nb2), (ff, nb), (ff2, nb2), (ff2, nb2)]):
        ws.cur.p[5 * k:5 * k + 3] += 0.1 * rng.standard_normal((3, 3))
        n.UsePartialRecalc = True
        f.calcEnergies()
        e = ws.ene.epot
        n.UsePartialRecalc = False
        f.calcEnergies()
        assert rel_err(e, ws.ene.epot) <= 1e-9
