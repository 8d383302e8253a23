"""A context's first list and later ones of the same positions: the same work items,
so the same results bit for bit (a pair of tiles rounds the row block's Born sums
once, two single tiles twice)."""
import numpy as np
import pytest

from helpers import gb_kwargs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cutoff", [999.0, 80.0])
def test_first_and_second_build_give_the_same_gradients(goldens, cutoff):
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    d = goldens["peptide120"]
    ctx = DeviceContext(SystemImage._from_fixture(d))
    ctx.set_list(2.0, check_skin=False)
    kw = dict(Cutoff=cutoff, InnerCutoff=cutoff - 1.0, VdwCutoff=cutoff, VdwInnerCutoff=cutoff - 1.0, GbsaStillCutoff=cutoff)
    ctx.set_gb(**dict(gb_kwargs(d), **kw))
    ctx.set_positions(d["pos"])
    out = []
    for _ in range(2):
        E, g = ctx.param_grad(ffi.GB)
        out.append((E, g, ctx.born_radii()))
        ctx.rebuild_list()
    # other cutoffs in between: the next build decides by its own
    ctx.set_gb(**dict(gb_kwargs(d), Cutoff=12.0, InnerCutoff=10.0, VdwCutoff=12.0, VdwInnerCutoff=10.0, GbsaStillCutoff=10.0))
    ctx.param_grad(ffi.GB)
    ctx.set_gb(**dict(gb_kwargs(d), **kw))
    E, g = ctx.param_grad(ffi.GB)
    out.append((E, g, ctx.born_radii()))
    ctx.close()
    for E, g, born in out[1:]:
        assert np.array_equal(born, out[0][2]) and E == out[0][0]
        assert all(np.array_equal(g[k], out[0][1][k]) for k in g)
