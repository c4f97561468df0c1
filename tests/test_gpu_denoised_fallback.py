"""The denoised mode's fallback draws, of all tiles in the frame's order, those
at or above the error budget: a budget between the tiles' errors gives each tile
the network's or the sorted-alpha pixels, and a viewport of as many pixels but
more tiles has room for all its errors."""
from __future__ import annotations

import numpy as np
import pytest

from gamesplat_b200 import Renderer
from gamesplat_b200 import renderer as RR
from gamesplat_b200 import scene
from gamesplat_b200.denoiser import Denoiser

from helpers import image_gate, oracle_alpha

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _draw(rows, cam, budget, fallback, d):
    with Renderer(0) as r:
        r.set(splat_render_mode="denoised", black_background=1)
        r.upload_gaussians(rows)
        r.set_denoiser(d)
        r.set_denoise_budget(budget, fallback)
        img = r.draw_frame(cam)
        return img.view(np.uint16), r.stats().denoise_fallback_tiles


@pytest.mark.parametrize("w,h", [(16, 16), (50, 34), (320, 180)])
def test_budget_between_the_tiles_errors(w, h):
    rows = RR.pack_raw(scene.small_scene(3, 20_000))
    cam = RR.camera_uniforms(*scene.small_camera_pose(), w, h)
    tx, ty = (w + 15) // 16, (h + 15) // 16
    with Denoiser(0) as d:
        head, none = _draw(rows, cam, 0.0, False, d)
        alpha, every = _draw(rows, cam, 0.0, True, d)
        assert (none, every) == (0, tx * ty)
        counts = []
        for budget in (1e-7, 1e-6, 1e-5, 3e-5, 1e-4, 3e-4, 1e-3):
            img, count = _draw(rows, cam, budget, True, d)
            drawn = 0
            for ty0 in range(ty):   # tile rows from the bottom
                rs = slice(max(h - 16 * (ty0 + 1), 0), h - 16 * ty0)
                for tx0 in range(tx):
                    cs = slice(16 * tx0, 16 * tx0 + 16)
                    is_alpha = np.array_equal(img[rs, cs], alpha[rs, cs])
                    assert is_alpha or np.array_equal(img[rs, cs], head[rs, cs])
                    drawn += is_alpha and not np.array_equal(alpha[rs, cs], head[rs, cs])
            assert drawn <= count
            counts.append(count)
    assert counts == sorted(counts, reverse=True)


def test_as_many_pixels_in_more_tiles():
    rows = RR.pack_raw(scene.small_scene(3, 20_000))
    with Denoiser(0) as d, Renderer(0) as r:
        r.set(splat_render_mode="denoised", black_background=1)
        r.upload_gaussians(rows)
        r.set_denoiser(d)
        r.set_denoise_budget(0.0, True)
        for w, h in ((64, 64), (2048, 2)):   # 16 tiles, then 128
            cam = RR.camera_uniforms(*scene.small_camera_pose(), w, h)
            img = r.draw_frame(cam)
            assert r.stats().denoise_fallback_tiles == ((w + 15) // 16) * ((h + 15) // 16)
            ref, _ = oracle_alpha(rows, cam, w, h)
            gate = image_gate(img, ref)
            assert gate["ok"], gate
