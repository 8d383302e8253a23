"""Dynamics past its first steps, where runs of plain steps are captured as one
graph and the integrator packs the next step's positions: bit for bit the same
trajectory, energies and kinetic energies as direct launches of single steps,
whatever step counts the caller uses (no tolerance: the sums are in fixed point
and both forms do the same arithmetic per atom)."""
import numpy as np
import pytest

from helpers import gb_kwargs, nb_kwargs

pytestmark = pytest.mark.gpu


def _dynamics(d, case, use_graph):
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.md import maxwell_boltzmann
    from pd_gb300.workspace import SystemImage
    ctx = DeviceContext(SystemImage._from_fixture(d))
    ctx.set_list(2.0)
    kind, integrator, nlist, sasa = case
    if kind == "nb":
        ctx.set_nb(**nb_kwargs(d, "nb"))
        what = ffi.NB | ffi.BONDED
    else:
        ctx.set_gb(**gb_kwargs(d))
        what = ffi.GB | ffi.BONDED | (ffi.SA if kind == "gbsa" else 0)
    ctx.set_positions(d["pos"])
    ctx.md_setup([300.0], integrator=integrator, timestep=5e-16, fric=1e13, update_nlist=nlist, update_sasa=sasa,
                 what=what, seed=7, use_graph=use_graph)
    ctx.set_velocities(maxwell_boltzmann(d["mass"], 300.0, 3))
    ring = ctx.md_set_trajectory(7, nslots=4) if kind == "gbsa" else None
    out = []
    # 70 steps reach the runs; then every remainder of the run lengths, with and
    # without energies on the last step
    for n, energy in ((70, False), (20, False), (1, False), (3, False), (7, True), (40, False), (33, True), (2, False)):
        ctx.md_run(n, energy_on_last=energy)
        out += [ctx.get_positions(), ctx.get_velocities(), np.array(ctx.kinetic())]
        if energy:
            out.append(np.array([ctx.energies()[0]["epot"]]))
    if ring is not None:
        out += [np.array([ctx.md_trajectory_frames()]), np.array(ring)]
    ctx.close()
    return out


@pytest.mark.parametrize("case", [("nb", 0, 5, 1), ("nb", 1, 1, 1), ("nb", 1, 3, 1), ("gbsa", 1, 20, 5), ("gb", 0, 50, 1)])
def test_captured_runs_equal_single_steps(goldens, case):
    d = goldens["water_c1" if case[0] == "nb" else "peptide30"]
    a, b = _dynamics(d, case, False), _dynamics(d, case, True)
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
