"""Forcefield calls on a WorkSpace without list padding: nothing tells a stale list by
its atoms' displacement then, so every call builds its own and gives what a fresh
WorkSpace gives."""
import pytest

from test_gpu_forcefield_calls import _nb, _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["peptide30", "peptide120"])
def test_moves_without_padding(goldens, name):
    ws, ff, nb = _nb(goldens, name, padding=0.0)
    x = ws.cur.p.copy()
    for scale in (1.06, 1.03, 1.0, 1.02, 1.6, 1.0):    # (spread out and drawn together: pairs enter the cutoff)
        ws.cur.p[:] = x.mean(0) + scale * (x - x.mean(0))
        ff.calcForces()
        _same(ws, goldens, name)
    ws.cur.p[:] = x
    nb.UsePartialRecalc = True
    ff.calcEnergies()
    e = ws.ene.epot
    nb.UsePartialRecalc = False
    ff.calcEnergies()
    assert abs(e - ws.ene.epot) <= 1e-9 * abs(e)
    ws.close()
