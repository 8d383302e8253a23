"""What the context knows of its list after a replayed step has rebuilt it."""
import numpy as np
import pytest

from conftest import golden
from helpers import nb_kwargs

pytestmark = pytest.mark.gpu


def _context(d, im, pos, **nb):
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    ctx = DeviceContext(im)
    ctx.set_list(2.0)
    ctx.set_nb(**(nb or nb_kwargs(d, "nb")))
    ctx.set_positions(pos)
    ctx.md_setup([300.0], integrator=1, timestep=1e-18, fric=1e13, update_nlist=1000, what=ffi.NB, seed=7)
    return ctx


def test_a_replayed_rebuild_counts_as_a_list_build(goldens):
    """A rebuild asked for by the host (here by setting the list parameters anew) is
    made once, by the next step, also where that step is replayed from a graph."""
    from pd_gb300.workspace import SystemImage
    d = goldens["water_c1"]
    ctx = _context(d, SystemImage._from_fixture(d), d["pos"])
    launches = lambda: (lambda n: (ctx.md_run(1), ctx.kernel_launches() - n)[1])(ctx.kernel_launches())
    ctx.md_run(2)
    plain = launches()
    for _ in range(3):
        ctx.set_list(2.0)
        assert launches() > plain
        assert launches() == plain
        assert len(ctx.list_slots()) >= len(d["pos"])
    ctx.close()


def test_an_evaluation_after_a_step_whose_list_outgrew_its_arrays(goldens):
    """A replayed rebuild that finds more tiles than the arrays hold reports it, and
    the next evaluation grows them instead of using the short list."""
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import load_workload
    d = golden("cfg_c4_large")
    im = load_workload(str(d["image"])).subset(int(d["system"][0]))
    centre = im.pos.mean(0)
    nb = dict(Cutoff=12.0, InnerCutoff=10.0, VdwCutoff=12.0, VdwInnerCutoff=10.0, Vdw14Scaling=0.5, Elec14Scaling=0.83333,
              Dielectric=1.0, EnergySwitch=1, ForceSwitch=0, DoVdw=1, DoElec=1)
    ctx = _context(d, im, centre + (im.pos - centre) * 2.0, **nb)
    ctx.md_run(2)
    for _ in range(2):                       # the rebuilding step: captured, then replayed
        ctx.set_list(2.0)
        ctx.md_run(1)
    ctx.set_list(2.0)
    ctx.set_positions(im.pos)
    with pytest.raises(ffi.PDGPUError) as err:
        ctx.md_run(1)
    assert err.value.status == -3            # PDGPU_ERR_LIST_OVERFLOW
    ctx.set_positions(im.pos)
    f = np.zeros((im.natom, 3))
    e = ctx.compute(ffi.NB, f)[0]
    ctx.close()
    ref = DeviceContext(im)
    ref.set_list(2.0)
    ref.set_nb(**nb)
    ref.set_positions(im.pos)
    f0 = np.zeros((im.natom, 3))
    e0 = ref.compute(ffi.NB, f0)[0]
    ref.close()
    assert e["vdw"] == e0["vdw"] and e["elec"] == e0["elec"] and np.array_equal(f, f0)
