"""The forward convolution in runs of one and two rows, dozens of them a CTA: each
run adds two halo rows to the ring, so here the multiplications run furthest
ahead of the epilogues.  Images of one row (and the half-size layers of crops
of two rows), several thousand row strips, every pair of channel counts, with
and without a mask, and transposed; tolerances as for the larger images in
test_gpu_denoiser."""
from __future__ import annotations

import pytest

from gamesplat_b200 import _lib as L
from gamesplat_b200 import denoiser as DN

from test_gpu_denoiser import _bf, _conv_ref, _features, _p, _random_params, _torch_net

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("cin,cout", [(16, 32), (32, 32), (32, 16)])
@pytest.mark.parametrize("n,h,w", [(6000, 1, 9), (1500, 1, 520), (4001, 2, 17)])
@pytest.mark.parametrize("masked", [False, True])
def test_short_runs(cin, cout, n, h, w, masked):
    g = torch.Generator(device="cuda").manual_seed(cin + 5 * cout + n)
    x = torch.randn(n, h, w, cin, device="cuda", generator=g).bfloat16()
    wt = (torch.randn(3, 3, cin, cout, device="cuda", generator=g) * 0.2).float()
    mask = torch.randn(n, h, w, cout, device="cuda", generator=g).bfloat16() if masked else None
    out = torch.full((n, h, w, cout), float("nan"), device="cuda")
    out16 = torch.full((n, h, w, cout), float("nan"), device="cuda", dtype=torch.bfloat16)
    scratch = torch.empty(L.lib().gs_conv3x3_scratch_bytes(cin, cout), dtype=torch.uint8, device="cuda")
    err = torch.zeros(4, dtype=torch.int32, device="cuda")
    L.check(L.lib().gs_conv3x3_bf16(_p(x), None, n, h, w, cin, cout, _p(wt), None, 0, 0, _p(mask), _p(out16), _p(out),
                                    _p(scratch), _p(err), None), "gs_conv3x3_bf16")
    torch.cuda.synchronize()
    assert int(err[0]) == 0
    ref = _conv_ref(x.float(), _bf(wt))
    if masked:
        ref = torch.where(mask.float() > 0, ref, torch.zeros_like(ref))
    scale = float(ref.abs().max())
    assert float((out - ref).abs().max()) <= 1e-4 * scale + 1e-6
    assert float((out16.float() - ref).abs().max()) <= 8e-3 * scale


def test_network_on_crops_of_two_rows():
    n, h, w = 4000, 2, 12
    x = _features(n, h, w, 3)
    flat = _random_params(4)
    o = 0
    flat_bf = flat.copy()
    for cin, cout in DN.LAYERS:
        k = 9 * cin * cout
        flat_bf[o:o + k] = torch.from_numpy(flat[o:o + k]).bfloat16().float().numpy()
        o += k + cout
    out = torch.full((n, h, w, 16), float("nan"), device="cuda")
    with DN.Denoiser(0) as d:
        d.set_params(flat)
        d.forward(x.data_ptr(), n, h, w, out.data_ptr())
        torch.cuda.synchronize()
        d.status()
    ref = _torch_net(x.float(), flat_bf)
    assert float((out - ref).abs().max()) <= 1e-2 * float(ref.abs().max())
