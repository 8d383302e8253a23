"""The block-grid path of the list build (systems of more than 8,192 blocks)."""
import numpy as np
import pytest

from test_gpu_list_build import NB_OPEN, _blocks, _box_distance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("periodic", [0, 1])
def test_block_grid_list_of_a_large_system_matches_all_pairs_scan(periodic):
    """More blocks than a row tests directly (8,192): the block-grid path, its row
    totals and a sample of whole rows against a scan of all block boxes."""
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    n, L, R = 270_001, 140.0, 6.0
    rng = np.random.default_rng(3)
    pos = rng.uniform(0.0, L, (n, 3))
    z = np.zeros(n)
    im = SystemImage([n], np.full(3, L if periodic else 0.0), z, np.full(n, 1.5), z, np.full(n, 2e-26),
                     np.stack([np.arange(0, n - 1, 2), np.arange(1, n, 2), np.ones(n // 2, np.int64)], 1), pos=pos)
    ctx = DeviceContext(im)
    ctx.set_list(1.0)
    ctx.set_nb(**dict(NB_OPEN, Cutoff=R - 1.0, InnerCutoff=R - 2.0, VdwCutoff=R - 1.0, VdwInnerCutoff=R - 2.0))
    ctx.set_positions(pos)
    tiles, _, _ = ctx.list_tiles()
    centre, half, _, _ = _blocks(ctx, im)
    ctx.close()
    nb = len(centre)
    assert nb > 8192
    key = np.unique(tiles[:, 0].astype(np.int64) * nb + tiles[:, 1])
    assert len(key) == len(tiles)
    for b in np.r_[0, nb - 1, rng.choice(nb, 200, replace=False)]:
        cols = np.arange(b, nb)
        d = _box_distance(centre, half, im.box[0], np.full(len(cols), b), cols)
        got = set(tiles[tiles[:, 0] == b, 1].tolist())
        assert set(cols[d < R - 1e-3].tolist()) <= got
        assert got <= set(cols[d < R + 2e-3].tolist())
