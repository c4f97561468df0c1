"""The visibility pass cuts the rows into whole rounds of equal tiles (4 CTAs an
SM, 8 to 20 rows a thread of 256): row counts at the edges of a warp's run, of
the smallest tile, of its growth, and of a second and third round give the
visible pairs of the oracle, in its order."""
from __future__ import annotations

import numpy as np
import pytest

from gamesplat_b200 import Renderer, _lib as L
from gamesplat_b200 import renderer as RR
from gamesplat_b200 import scene
from oracle import oracle as O

from helpers import small_cam

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

CELLS = 4 * 256   # rows of one row a thread, per SM


@pytest.fixture(scope="module")
def pool():
    """Rows of which a part is behind the camera or off the screen; alternating
    long runs of the two kinds, so that whole tiles are empty or full."""
    raw = np.tile(scene.small_scene(4, 4099), (12, 1))
    raw[:, 0] += np.where((np.arange(raw.shape[0]) // 5000) % 3 == 1, 9.0, 0.0)
    return RR.pack_raw(raw)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 257, 2047, 2048, 2049, 40_001, "8", "8+", "20", "20+", "40+"])
def test_visible_pairs_in_order(pool, n):
    if isinstance(n, str):
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        n = int(n.rstrip("+")) * CELLS * sms + (1 if n.endswith("+") else 0)
    rows = np.ascontiguousarray(np.resize(pool, (n, pool.shape[1])))
    cam = small_cam(64, 64)
    ids, keys, _, visible, _ = O.cull(rows, cam)
    ks, si = O.sort_pairs(keys, ids)
    with Renderer(0) as r:
        r.set(splat_render_mode="alpha", sh_degree=0)
        r.upload_gaussians(rows)
        r.draw_frame(cam)
        assert r.stats().visible_count == visible
        assert np.array_equal(r.debug_read(L.GS_DEBUG_IDS, n), ids)
        assert np.array_equal(r.debug_read(L.GS_DEBUG_KEYS, n), keys)
        assert np.array_equal(r.debug_read(L.GS_DEBUG_SORTED_IDS, n), si)
        assert np.array_equal(r.debug_read(L.GS_DEBUG_SORTED_KEYS, n), ks)
