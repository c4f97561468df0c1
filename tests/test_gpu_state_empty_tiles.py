"""State batches over tiles without entries: such a tile goes through the group
rasterizer without a batch of records, so nothing but its own barrier stands
between the warp that lays out the group's images and the warps that store into
them.  A few Gaussians in a wide image, or none in view: every image, the
background included, has the bits of gs_render after gs_set_anim_state, with
other kernels' shared memory left on the SMs between the batches."""
from __future__ import annotations

import numpy as np
import pytest

from gamesplat_b200 import Renderer
from gamesplat_b200 import _lib as L
from gamesplat_b200 import renderer as RR
from gamesplat_b200 import scene

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

STATES, W, H = 3, 640, 384


@pytest.mark.parametrize("shape", [(16, 16), (32, 8), (8, 32)])
@pytest.mark.parametrize("frames,n,behind", [(3, 60, False), (8, 60, False), (11, 60, False), (13, 1, False),
                                             (16, 60, True)])
def test_states_over_empty_tiles(frames, n, behind, shape):
    rng = np.random.default_rng(frames + n)
    raw = scene.small_scene(frames, n)
    if behind:
        raw[:, 2] += 9.0
    deltas = rng.integers(-128, 128, (STATES, n, 48)).astype(np.int8)
    scales = rng.uniform(0.0, 0.01, 48).astype(np.float32)
    sa = rng.integers(0, STATES + 1, frames)
    sb = rng.integers(0, STATES + 1, frames)
    wt = np.where(rng.random(frames) < 0.4, 0.0, rng.random(frames)).astype(np.float32)
    cam = RR.camera_uniforms(*scene.small_camera_pose(), W, H)
    with Renderer(0) as r:
        r.set(splat_render_mode="alpha")   # background 0.1
        L.check(L.lib().gs_set_tile_shape(r._ctx, *shape), "gs_set_tile_shape")
        r.upload_gaussians(RR.pack_raw(raw))
        r.upload_animation(deltas, scales)
        outs = [torch.empty(H, W, 4, dtype=torch.float16, device="cuda") for _ in range(frames)]
        ones = []
        for k in range(frames):
            r.set_animation_state(int(sa[k]), int(sb[k]), float(wt[k]))
            ones.append(torch.empty(H, W, 4, dtype=torch.float16, device="cuda"))
            r.draw_frame(cam, out_ptr=ones[-1].data_ptr())
        assert r.stats().tile_entries < (W * H) // 256 // 2   # most tiles hold nothing
        for _ in range(4):
            for o in outs:
                o.fill_(float("nan"))
            r.draw_frame(cam, out_ptr=ones[-1].data_ptr())   # its kernels' shared memory stays behind
            r.render_anim_batch(cam, sa, [o.data_ptr() for o in outs], sb, wt)
            torch.cuda.synchronize()
            for k in range(frames):
                assert torch.equal(ones[k].view(torch.int16), outs[k].view(torch.int16)), k
