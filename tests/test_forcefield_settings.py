"""Settings changed between two calls of a Forcefield reach the device context
whatever their type; the context here is a stand-in that records what it is given."""
import numpy as np
import pytest

import pd_gb300 as pdg
from pd_gb300 import ffi


class _Context:
    def __init__(self, nsystems):
        self.settings = self.updates = 0
        self.nsystems = nsystems
        self.nb, self.gb, self.lists, self.calls = [], [], [], []

    def set_nb(self, **kw):
        self.settings += 1
        self.nb.append(kw)

    def set_gb(self, **kw):
        self.settings += 1
        self.gb.append(kw)

    def set_gb_mode(self, fast_mode, **kw):
        self.settings += 1

    def set_list(self, padding, check_skin=True):
        self.settings += 1
        self.lists.append(padding)

    def set_positions(self, pos):
        pass

    def compute(self, what, forces=None):
        self.calls.append("compute")
        e = {k: float(len(self.calls)) for k, _ in ffi.Energies._fields_}
        return [dict(e) for _ in range(self.nsystems)]

    def nb_energy_full(self):
        self.calls.append("full")
        return self.compute(ffi.NB)

    def nb_energy_update(self):
        self.calls.append("update")
        return self.compute(ffi.NB), 1

    def close(self):
        pass


@pytest.fixture
def workspace(goldens, monkeypatch):
    ws = pdg.WorkSpace(pdg.SystemImage._from_fixture(goldens["peptide30"]))
    made = []

    def context():
        if ws._ctx is None:
            ws._ctx = _Context(ws.image.nsystems)
            made.append(ws._ctx)
        return ws._ctx
    monkeypatch.setattr(ws, "context", context)
    ws.made = made
    return ws


def _container(ws, kind):
    ff = pdg.Forcefield(ws)
    c = kind(ws)
    c.AutoScaling14 = False
    ff.add(c)
    return ff, c


@pytest.mark.parametrize("values", [[9, 10, 11, 12], list(np.arange(9, 13)), list(np.arange(9.0, 13.0, dtype=np.float32)),
                                    [np.array(9.0), np.array(10.5)], [np.float16(9), np.float64(10), 11]])
def test_a_cutoff_scan_reaches_the_context(workspace, values):
    ff, nb = _container(workspace, pdg.FF_NonBonded_GPU)
    nb.InnerCutoff = nb.VdwInnerCutoff = 8.0
    for v in values:
        nb.Cutoff = nb.VdwCutoff = v
        ff.calcForces()
        ff.calcForces()
    ctx = workspace.context()
    assert [k["Cutoff"] for k in ctx.nb] == [float(v) for v in values]
    assert ctx.settings == 2 * len(values)                  # once a value: nb and list


def test_settings_of_other_types(workspace):
    torch = pytest.importorskip("torch")
    ff, nb = _container(workspace, pdg.FF_NonBonded_GPU)
    nb.InnerCutoff = nb.VdwInnerCutoff = 8.0
    nb.notes = {"a": [1, np.arange(3)]}
    nb.table, nb.callback = torch.arange(4), print          # (no settings: kept, not compared element by element)
    cut = torch.tensor(9.0)
    for v in (9.0, 11.5):
        cut.fill_(v)
        nb.Cutoff = nb.VdwCutoff = cut
        ff.calcForces()
        ff.calcForces()
    ctx = workspace.context()
    assert [k["Cutoff"] for k in ctx.nb] == [9.0, 11.5] and ctx.settings == 4


def test_values_of_one_hash(workspace):
    ff, gb = _container(workspace, pdg.FF_GeneralizedBorn_Still_GPU)
    values = [-4.0, -1.0, -2.0, np.float32(-1), np.int64(-2)]
    for v in values:
        gb.ExpApproxThreshold = v
        ff.calcForces()
    assert [k["ExpApproxThreshold"] for k in workspace.context().gb] == [float(v) for v in values]


def test_the_surface_tension_reaches_the_image(workspace):
    ff = pdg.Forcefield(workspace)
    sa = pdg.FF_SASA_LCPO_GPU(workspace)
    ff.add(sa)
    for v in (0.005, np.float32(0.25), -1.0, -2.0):
        sa.GlobalASP = v
        ff.calcForces()
        assert np.allclose(workspace.image.lcpo_sigma, float(v) / 6.0221418E23 * 4184.0, rtol=1e-12, atol=0.0)


def test_flags_padding_and_tables(workspace):
    ff, nb = _container(workspace, pdg.FF_NonBonded_GPU)
    ff.calcForces()
    ctx = workspace.context()
    n = ctx.settings
    ff.calcForces()
    assert ctx.settings == n
    nb.DoElec = np.bool_(False)
    ff.calcForces()
    assert ctx.nb[-1]["DoElec"] == 0
    workspace.Padding = np.float32(1.25)
    ff.calcForces()
    assert ctx.lists[-1] == 1.25
    nb.AutoScaling14 = True
    workspace.image.scaling14 = np.array([0.25, 0.5])
    ff.calcForces()
    assert (ctx.nb[-1]["Vdw14Scaling"], ctx.nb[-1]["Elec14Scaling"]) == (0.25, 0.5)
    workspace.image.scaling14[0] = 0.75                     # in place
    ff.calcForces()
    assert ctx.nb[-1]["Vdw14Scaling"] == 0.75


def test_partial_recalculation_starts_anew_with_its_settings(workspace):
    ff, nb = _container(workspace, pdg.FF_NonBonded_GPU)
    nb.UsePartialRecalc = True
    ctx = workspace.context()
    for k in range(3):
        ff.calcEnergies()
    for v in (np.float32(11), np.int64(10)):
        nb.Cutoff = nb.VdwCutoff = v
        nb.InnerCutoff = nb.VdwInnerCutoff = 8.0
        ff.calcEnergies()
        ff.calcEnergies()
    assert [c for c in ctx.calls if c != "compute"] == ["full", "update", "update", "full", "update", "full", "update"]
    ctx.updates += 1                                        # (new per-atom parameters)
    ff.calcEnergies()
    ff.calcEnergies()
    assert [c for c in ctx.calls if c != "compute"][-2:] == ["full", "update"]
