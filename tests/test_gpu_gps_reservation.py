"""GPS work items are reserved a warp at a time: at a budget that holds a frame's
items exactly, the frame equals the one with room to spare; one item less (a
budget that ends inside a warp's reservation), one item in all and far fewer
report the overflow and the same requested count, and the context draws the
whole frame again afterwards."""
from __future__ import annotations

import numpy as np
import pytest

from gamesplat_b200 import Renderer
from gamesplat_b200 import renderer as RR
from gamesplat_b200 import scene

pytestmark = pytest.mark.gpu


def _frame(rows, cam, budget):
    with Renderer(0) as r:
        r.set(splat_render_mode="gps", gps_supersample_factor=1)
        r.upload_gaussians(rows)
        assert r.set_gps_work_budget(budget)
        img = r.draw_frame(cam)
        st = r.stats()
        assert r.set_gps_work_budget(16 << 20)
        r.reset_stochastic_accumulation()      # a changed budget resets it, the same one does not
        again = r.draw_frame(cam)
        return img, int(st.gps_requested_work_items), int(st.gps_budget_exhausted), again


@pytest.mark.parametrize("n", [1, 33, 20_001])
def test_budget_at_the_requested_count(n):
    raw = scene.small_scene(n, n)
    raw[:, 51] = 2.0
    raw[:, 52:55] = -2.5        # several items a splat
    rows = RR.pack_raw(raw)
    cam = RR.camera_uniforms(*scene.small_camera_pose(), 320, 180)
    full, items, over, again = _frame(rows, cam, 16 << 20)
    assert items > n and not over
    img, got, over, second = _frame(rows, cam, items)
    assert (got, over) == (items, 0)
    assert np.array_equal(img.view(np.uint16), full.view(np.uint16))
    assert np.array_equal(second.view(np.uint16), again.view(np.uint16))
    for budget in {items - 1, max(items // 3, 1), 1}:
        _, got, over, second = _frame(rows, cam, budget)
        assert (got, over) == (items, 1)
        assert np.array_equal(second.view(np.uint16), again.view(np.uint16))
