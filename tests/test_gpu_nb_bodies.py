"""The packed LJ + Coulomb force pass (switched laws) against the FP64 oracle: every
law (one switch, split radii, force switch, LJ alone), open space and periodic
boxes with and without per-pair images, tile path and j-atom groups, blocks with
one atom to many, bonded pairs.  Tolerance as the parity tests': forces 1e-5
relative RMS (FP32 pair arithmetic)."""
import numpy as np
import pytest

from conftest import rel_rms

pytestmark = pytest.mark.gpu

MODES = {"same": dict(InnerCutoff=7.0, VdwCutoff=9.0, VdwInnerCutoff=7.0, EnergySwitch=1, ForceSwitch=0, DoElec=1),
         "split": dict(InnerCutoff=6.5, VdwCutoff=8.0, VdwInnerCutoff=5.5, EnergySwitch=1, ForceSwitch=0, DoElec=1),
         "force": dict(InnerCutoff=6.0, VdwCutoff=9.0, VdwInnerCutoff=7.5, EnergySwitch=0, ForceSwitch=1, DoElec=1),
         "vdw": dict(InnerCutoff=7.0, VdwCutoff=9.0, VdwInnerCutoff=7.0, EnergySwitch=1, ForceSwitch=0, DoElec=0)}


def _lattice(n, seed, periodic):
    rng = np.random.default_rng(seed)
    m = int(np.ceil(n ** (1.0 / 3.0)))
    L = max(20.0, 3.0 * m)
    a = L / m if periodic else 3.0
    g = rng.permutation(m ** 3)[:n]
    pos = np.stack([g // (m * m), g // m % m, g % m], 1) * a + rng.uniform(-0.3, 0.3, (n, 3))
    d = pos[:, None] - pos[None] if n <= 400 else None
    excl = np.zeros((0, 3), np.int32)
    if d is not None:
        i, j = np.nonzero(np.triu((d ** 2).sum(-1) < 3.4 ** 2, 1))
        excl = np.stack([i, j, rng.integers(1, 4, len(i))], 1).astype(np.int32)
    return pos, excl, np.full(3, L if periodic else 0.0), dict(
        charge=rng.uniform(-0.6, 0.6, n), radius=rng.uniform(0.0, 1.7, n), epsilon=rng.uniform(1, 3, n) * 1e-11)


@pytest.mark.parametrize("mode", sorted(MODES))
@pytest.mark.parametrize("n,periodic", [(1, 0), (2, 1), (33, 0), (64, 1), (300, 0), (300, 1), (2500, 0), (2500, 1)])
def test_nb_force_bodies_match_oracle(n, periodic, mode):
    torch = pytest.importorskip("torch")
    from oracle import pdoracle as O
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    pos, excl, box, par = _lattice(n, 7 * n + periodic, periodic)
    kw = dict(Cutoff=9.0, Vdw14Scaling=0.5, Elec14Scaling=0.8, Dielectric=1.0, DoVdw=1, **MODES[mode])
    s = O.OracleSystem(pos, par["charge"], par["radius"], par["epsilon"], excl, tuple(box))
    ref = O.nonbonded(s, O.nb_params(ListCutoff=10.0, **kw))[1]
    out = []
    for groups in (1, 0):
        im = SystemImage([n], box, par["charge"], par["radius"], par["epsilon"], np.full(n, 2e-26), excl, pos=pos)
        ctx = DeviceContext(im)
        ctx.set_list(1.0)
        ctx.set_nb(**kw)
        ctx.set_nb_groups(groups)
        ctx.set_positions(pos)
        ctx.compute_device(ffi.NB)
        moved = pos + 0.2                       # inside the skin: the packed boxes follow the atoms
        moved[::7] -= 0.35
        # (a block as wide as half the box may not move: the skin check sees its image flip)
        for p in (pos, moved, pos) if not periodic or n > 1000 else (pos,):
            ctx.set_positions(p)
            fd = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
            ctx.compute_device(ffi.NB, fd.data_ptr())
            ctx.synchronize()
        out.append(fd.cpu().numpy())
        ctx.close()
    scale = np.sqrt((ref ** 2).sum(1).mean())
    for f in out:
        assert (rel_rms(f, ref) if scale > 0 else np.abs(f).max()) <= 1e-5


def test_nb_force_of_moved_atoms_matches_oracle():
    """Forces after a move inside the skin, the list (groups, classes) from before it."""
    torch = pytest.importorskip("torch")
    from oracle import pdoracle as O
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    n = 2500
    pos, excl, box, par = _lattice(n, 3, 1)
    kw = dict(Cutoff=9.0, Vdw14Scaling=0.5, Elec14Scaling=0.8, Dielectric=1.0, DoVdw=1, **MODES["same"])
    im = SystemImage([n], box, par["charge"], par["radius"], par["epsilon"], np.full(n, 2e-26), excl, pos=pos)
    ctx = DeviceContext(im)
    ctx.set_list(2.0)
    ctx.set_nb(**kw)
    ctx.set_positions(pos)
    ctx.compute_device(ffi.NB)
    d = np.random.default_rng(1).standard_normal((n, 3))
    moved = pos + 0.95 * d / np.linalg.norm(d, axis=1)[:, None] * np.random.default_rng(2).random((n, 1))
    ctx.set_positions(moved)
    fd = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    ctx.compute_device(ffi.NB, fd.data_ptr())
    ctx.synchronize()
    ctx.close()
    s = O.OracleSystem(moved, par["charge"], par["radius"], par["epsilon"], excl, tuple(box))
    assert rel_rms(fd.cpu().numpy(), O.nonbonded(s, O.nb_params(ListCutoff=11.0, **kw))[1]) <= 1e-5
