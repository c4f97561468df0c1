"""gsanim state batches are drawn in groups of frames that share the alpha work
(8 frames, the last group 4 where that holds the rest): for every split of a
batch into groups, every tile shape, SH degree and kind of state (base, one
state, blends with and without the base) each image has the bits of gs_render
after gs_set_anim_state."""
from __future__ import annotations

import numpy as np
import pytest

from gamesplat_b200 import Renderer
from gamesplat_b200 import _lib as L
from gamesplat_b200 import renderer as RR
from gamesplat_b200 import scene

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

N, STATES, W, H = 9_001, 4, 149, 83


@pytest.mark.parametrize("frames,shape,degree,lod", [(1, (16, 16), 3, 0.0), (4, (32, 8), 3, 2.9), (5, (16, 16), 2, 0.0),
                                                     (8, (8, 32), 1, 0.0), (9, (16, 16), 3, 0.0),
                                                     (13, (32, 8), 0, 0.0), (19, (16, 16), 3, 3.0)])
def test_state_groups_equal_single_frames(frames, shape, degree, lod):
    rng = np.random.default_rng(frames)
    deltas = rng.integers(-128, 128, (STATES, N, 48)).astype(np.int8)
    scales = rng.uniform(0.0, 0.01, 48).astype(np.float32)
    sa = rng.integers(0, STATES + 1, frames)
    sb = rng.integers(0, STATES + 1, frames)
    wt = np.where(rng.random(frames) < 0.4, 0.0, rng.random(frames)).astype(np.float32)
    cam = RR.camera_uniforms(*scene.small_camera_pose(), W, H)
    with Renderer(0) as r:
        r.set(splat_render_mode="alpha", sh_degree=degree, sh_lod_distance=lod)   # background 0.1
        L.check(L.lib().gs_set_tile_shape(r._ctx, *shape), "gs_set_tile_shape")
        r.upload_gaussians(RR.pack_raw(scene.small_scene(frames, N)))
        r.upload_animation(deltas, scales)
        outs = [torch.full((H, W, 4), float("nan"), dtype=torch.float16, device="cuda") for _ in range(frames)]
        r.render_anim_batch(cam, sa, [o.data_ptr() for o in outs], sb, wt)
        for k in range(frames):
            r.set_animation_state(int(sa[k]), int(sb[k]), float(wt[k]))
            one = torch.empty(H, W, 4, dtype=torch.float16, device="cuda")
            r.draw_frame(cam, out_ptr=one.data_ptr())
            torch.cuda.synchronize()
            assert torch.equal(one.view(torch.int16), outs[k].view(torch.int16)), k
