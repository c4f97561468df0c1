"""The training loss works on 32 x 16 pixel tiles with a 5-pixel halo: its value
and gradient against torch (fp32) at sizes around the tile edges, on images too
small for the SSIM window, and with an output tensor that is not 16-byte
aligned (read element by element).  Tolerances as for whole images: the bf16
gradient within 1e-2 of its scale, sums within 1e-4."""
from __future__ import annotations

import pytest

from gamesplat_b200 import denoiser as DN

from test_gpu_denoiser import _features, _torch_loss

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n,h,w", [(1, 1, 1), (1, 10, 40), (1, 11, 11), (2, 16, 32), (1, 17, 33), (2, 31, 65)])
def test_loss_at_tile_edges(n, h, w, offset):
    g = torch.Generator(device="cuda").manual_seed(100 * h + w)
    x = _features(n, h, w, h)
    out = torch.randn(n, h, w, 16, device="cuda", generator=g) * 0.1
    store = torch.zeros(out.numel() + offset, device="cuda")
    store[offset:] = out.flatten()
    target = torch.rand(n, h, w, 4, device="cuda", generator=g)
    dout = torch.full((n, h, w, 16), 7.0, device="cuda", dtype=torch.bfloat16)
    ssim_w = 0.2 if h > 10 and w > 10 else 0.0    # smaller images have no SSIM term
    with DN.Denoiser(0) as d:
        parts = d.loss(x.data_ptr(), store.data_ptr() + 4 * offset, target.data_ptr(), n, h, w, dout.data_ptr(), 0.2, 0.01)
    o = out.clone().requires_grad_(True)
    if ssim_w:
        total, l1, ssim, le = _torch_loss(o, x, target, ssim_w, 0.01)
        assert abs(parts[1] - float(ssim)) <= 1e-4
    else:
        pred = torch.cat([x[..., 5:8].float() + o[..., 0:3], x[..., 3:4].float() + o[..., 3:4]], dim=-1)
        l1 = (pred - target).abs().mean()
        le = ((o[..., 4] - 1000.0 * ((pred - target).detach() ** 2).mean(dim=-1)) ** 2).mean()
        total = l1 + 0.01 * le
        assert parts[1] == 1.0
    total.backward()
    assert abs(parts[0] - float(l1)) <= 1e-5
    assert abs(parts[2] - float(le)) <= 1e-4 * max(1.0, float(le))
    got, ref = dout.float(), o.grad
    for c in range(5):
        assert float((got[..., c] - ref[..., c]).abs().max()) <= 1e-2 * float(ref[..., c].abs().max()), c
    assert float(got[..., 5:].abs().max()) == 0.0
