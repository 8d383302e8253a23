"""List builds with many atoms in one grid cell (an open system with atoms far apart:
32 cells over its bounding box along each axis): the slots hold each cell's atoms
together and in ascending order, whatever its size, and every system its own atoms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KW = dict(Cutoff=6.0, InnerCutoff=5.0, VdwCutoff=6.0, VdwInnerCutoff=5.0, Vdw14Scaling=1.0, Elec14Scaling=1.0, Dielectric=1.0,
          EnergySwitch=1, ForceSwitch=0, DoVdw=1, DoElec=1)


def _system(sizes, rng):
    """Clusters of the given sizes, a cell each (100 A apart on the diagonal), atoms numbered at random."""
    cluster = rng.permutation(np.repeat(np.arange(len(sizes)), sizes))
    return 100.0 * cluster[:, None] + rng.uniform(0.0, 2.0, (len(cluster), 3)), cluster


# 64 atoms stay with a cell's thread in systems of up to 32,768 atoms, 78 in one of 40,000
@pytest.mark.parametrize("systems", [[[1, 2, 63, 64, 65, 66, 128] + [1] * 25],
                                     [[3000, 1] + [1] * 30, [5] * 32, [200, 64, 65, 1, 700] + [3] * 27],
                                     [[40000 - 310, 78, 79, 80, 64, 9]]])
def test_slots_hold_each_cells_atoms_in_order(systems):
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    rng = np.random.default_rng(len(systems[0]))
    pos, cluster = zip(*[_system(s, rng) for s in systems])
    n = [len(p) for p in pos]
    N = sum(n)
    im = SystemImage(n, np.zeros(3 * len(n)), np.zeros(N), np.full(N, 1.5), np.zeros(N), np.full(N, 2e-26),
                     np.zeros((0, 3), np.int32), pos=np.concatenate(pos))
    ctx = DeviceContext(im)
    ctx.set_list(1.0)
    ctx.set_nb(**KW)
    ctx.set_positions(im.pos)
    for build in range(2):
        slots, first = ctx.list_slots(), 0
        for s, c in enumerate(cluster):
            npad = (n[s] + 31) // 32 * 32
            a = slots[first:first + npad] - sum(n[:s])
            assert np.all(slots[first + n[s]:first + npad] == -1)
            a = a[:n[s]]
            assert np.array_equal(np.sort(a), np.arange(n[s]))
            # one run a cluster, ascending inside it
            cut = np.flatnonzero(np.diff(c[a])) + 1
            assert len(cut) == len(systems[s]) - 1
            assert all(np.all(np.diff(run) > 0) for run in np.split(a, cut))
            first += npad
        ctx.rebuild_list()                # (from the state the first build left)
    ctx.close()
