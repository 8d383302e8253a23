"""Settings changed between runs of one trajectory: steps captured before the change
are not replayed after it, whichever evaluation rebuilt the list in between.  Bit for
bit the trajectory of direct launches (no tolerance: the same kernels, sums in fixed
point)."""
import numpy as np
import pytest

from helpers import gb_kwargs, nb_kwargs

pytestmark = pytest.mark.gpu


def _dynamics(d, kind, changes, use_graph):
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.md import maxwell_boltzmann
    from pd_gb300.workspace import SystemImage
    ctx = DeviceContext(SystemImage._from_fixture(d))
    # (short cutoffs in the 27.5 A box: the list build makes NB j-atom groups)
    cut = lambda c: dict(Cutoff=c, InnerCutoff=c - 1.0, VdwCutoff=c, VdwInnerCutoff=c - 1.0)
    setters = {"nb": lambda c: ctx.set_nb(**dict(nb_kwargs(d, "nb"), **cut(c))),
               "gb": lambda c: ctx.set_gb(**dict(gb_kwargs(d), **cut(c))),
               "list": lambda padding, check: ctx.set_list(padding, check_skin=check)}
    setters["list"](1.0, True)
    setters[kind](5.0 if kind == "nb" else 12.0)
    what = ffi.NB if kind == "nb" else ffi.GB
    ctx.set_positions(d["pos"])
    ctx.md_setup([300.0], integrator=1, timestep=2.5e-16, fric=1e13, update_nlist=1000, what=what | ffi.BONDED, seed=7,
                 use_graph=use_graph)
    ctx.set_velocities(maxwell_boltzmann(d["mass"], 300.0, 3))
    ctx.md_run(6)
    out = []
    for name, args, evaluate in changes:
        setters[name](*args)
        if evaluate:
            ctx.compute_device(what)            # (builds the list outside the dynamics)
        ctx.md_run(4)
        out += [ctx.get_positions(), ctx.get_velocities(), np.array(ctx.kinetic())]
    ctx.close()
    return out


@pytest.mark.parametrize("kind,changes", [
    ("nb", [("list", (1.0, False), True), ("nb", (6.5,), True), ("list", (1.0, True), False), ("nb", (5.0,), True)]),
    ("nb", [("nb", (9.0,), True), ("list", (2.0, True), True)]),
    ("gb", [("gb", (9.0,), True), ("list", (2.0, True), True), ("gb", (12.0,), False)]),
])
def test_settings_between_runs(goldens, kind, changes):
    d = goldens["water_c1" if kind == "nb" else "peptide30"]
    a, b = _dynamics(d, kind, changes, False), _dynamics(d, kind, changes, True)
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
