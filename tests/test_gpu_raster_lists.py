"""Each warp of a rasterizer lists the staged splats it shades (batches of 128)
and takes them 8, 4 or 2 to a trip (alpha, stochastic, two samples): lists that
end at every remainder of a trip and batches that end at every edge, in one tile
and in two, with splats too faint for a pixel to be done before its last one.
Alpha within the image gate of the oracle; the stochastic samples bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from gamesplat_b200 import Renderer, _lib as L
from gamesplat_b200 import renderer as RR
from gamesplat_b200 import scene
from oracle import oracle as O

from helpers import image_gate, oracle_alpha, small_cam

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

W, H = 18, 10


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 8, 9, 15, 16, 17, 127, 128, 129, 131, 256, 263])
def test_list_and_batch_remainders(n):
    raw = scene.small_scene(n, n)
    raw[:, 51] = -4.0        # opacity 0.018
    raw[:, 52:55] += 2.5     # wide: most reach every warp of both tiles
    rows, cam = RR.pack_raw(raw), small_cam(W, H)
    ref, _ = oracle_alpha(rows, cam, W, H)
    ids, _, proj, _, _ = O.cull(rows, cam)
    with Renderer(0) as r:
        r.set(splat_render_mode="alpha", black_background=1)
        r.upload_gaussians(rows)
        gate = image_gate(r.draw_frame(cam), ref)
        assert gate["ok"], gate
        r.set(splat_render_mode="stochastic", stochastic_taa_enabled=0, stochastic_accumulation_enabled=0,
              stochastic_samples_per_frame=1)
        r.draw_frame(cam)
        sample = r.debug_read(L.GS_DEBUG_SAMPLE, W * H * 4, np.float32, (H, W, 4))
        depth = r.debug_read(L.GS_DEBUG_DEPTH, W * H, np.float32, (H, W))
        one, one_depth, _ = O.stochastic_sample(ids, proj, W, H, 1.0, cam, bg=0.0, rgba8=True)
        assert np.array_equal(sample.view(np.uint32), one.view(np.uint32))
        assert np.array_equal(depth.view(np.uint32), one_depth.view(np.uint32))
    with Renderer(0) as r:
        r.set(splat_render_mode="denoised", black_background=1)
        r.upload_gaussians(rows)
        feats = torch.zeros(H, W, 16, dtype=torch.bfloat16, device="cuda")
        r.render_features(cam, feats.data_ptr())
        sample = r.debug_read(L.GS_DEBUG_SAMPLE, W * H * 4, np.float32, (H, W, 4))
        depth = r.debug_read(L.GS_DEBUG_DEPTH, W * H, np.float32, (H, W))
        s = [O.stochastic_sample(ids, proj, W, H, seed, cam, bg=0.0, rgba8=False) for seed in (1.0, 2.0)]
        half = np.float32(0.5)
        assert np.array_equal(sample.view(np.uint32), ((s[0][0] + s[1][0]) * half).view(np.uint32))
        assert np.array_equal(depth.view(np.uint32), ((s[0][1] + s[1][1]) * half).view(np.uint32))
