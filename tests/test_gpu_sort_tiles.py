"""The sorts' tiles: a pass is cut into equal tiles by its element count, and
look-backs go over groups of 16 tiles.  gs_sort_pairs at counts around the tile
sizes (1280 to 5120 pairs), one and many groups, one and several waves of the
grid, bit ranges that end inside a digit, and few distinct keys: exactly numpy's
stable sort.  Frames whose tile entries take one pass (at most 256 tiles), two,
or the (id, position) pairs (more than 65 536 tiles), and whose depths reach past
the three depth-key digits: order and counts exact, images within the gate."""
from __future__ import annotations

import numpy as np
import pytest

from gamesplat_b200 import Renderer, _lib as L
from gamesplat_b200 import renderer as RR
from gamesplat_b200 import scene
from oracle import oracle as O

from helpers import image_gate
from test_gpu_sort import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 1279, 1280, 1281, 2304, 20_479, 20_481, 81_921, 568_320, 568_321, 2_273_281,
                               6_000_001])
@pytest.mark.parametrize("kind", ["random", "few", "range"])
def test_pairs_at_tile_edges(n, kind):
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 2 ** 32, size=n, dtype=np.uint64).astype(np.uint32)
    begin, end = 0, 32
    if kind == "few":
        keys = (keys % np.uint32(3)) << np.uint32(13)
    if kind == "range":
        begin, end = 5, 18
    vals = rng.permutation(n).astype(np.uint32)
    k, v = _run(keys, vals, begin, end)
    order = np.argsort((keys >> np.uint32(begin)) & np.uint32((1 << (end - begin)) - 1), kind="stable")
    assert np.array_equal(k, keys[order]) and np.array_equal(v, vals[order])


def _check_frame(rows, cam, w, h):
    ids, keys, proj, vc, _ = O.cull(rows, cam)
    sk, si = O.sort_pairs(keys, ids)
    ref, _ = O.composite_alpha(si, proj, w, h, cam, bg=0.0)
    with Renderer(0) as r:
        r.set(splat_render_mode="alpha", black_background=1)
        r.upload_gaussians(rows)
        for _ in range(2):      # the second frame finds the first one's look-back words
            img = r.draw_frame(cam)
        assert r.stats().visible_count == vc
        assert np.array_equal(r.debug_read(L.GS_DEBUG_SORTED_IDS, rows.shape[0]), si)
        assert np.array_equal(r.debug_read(L.GS_DEBUG_SORTED_KEYS, rows.shape[0]), sk)
    gate = image_gate(img, ref.astype(np.float16))
    assert gate["ok"], gate


@pytest.mark.parametrize("n,w,h", [(1, 16, 16), (5_000, 256, 256), (5_000, 257, 255), (70_000, 640, 480),
                                   (3_000, 4112, 4096)])
def test_frames_by_tile_count(n, w, h):
    rows = RR.pack_raw(scene.small_scene(n, n))
    _check_frame(rows, RR.camera_uniforms(*scene.small_camera_pose(), w, h), w, h)


def test_frame_with_far_depths():
    """Depths from the near test's 0.2 to 1e6: the keys' upper digit is not constant."""
    raw = scene.small_scene(5, 20_000)
    rng = np.random.default_rng(5)
    depth = 10.0 ** rng.uniform(np.log10(0.2), 6.0, 20_000)
    raw[:, 0:2] *= depth[:, None] * 0.3
    raw[:, 2] = 3.0 - depth                       # the camera stands at z = 3 and looks down -z
    raw[:, 52:55] += np.log(depth)[:, None] * 0.9
    rows = RR.pack_raw(raw)
    cam = RR.camera_uniforms(*scene.small_camera_pose(), 320, 180, far_plane=4.0e6)
    _check_frame(rows, cam, 320, 180)
