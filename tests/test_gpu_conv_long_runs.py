"""The forward convolution where a CTA walks dozens of rows and crosses from one
column strip or image to the next: the rings of halo rows and accumulators wrap
(also in the middle of an MMA over three output rows), both epilogue groups take
turns, and the pooled output's row pairs meet a strip's end.  Every channel pair,
with and without a mask, the two-input layer, the input gradient, and the
network with its pooled first layer; tolerances as for the smaller images in
test_gpu_denoiser."""
from __future__ import annotations

import pytest

from gamesplat_b200 import _lib as L
from gamesplat_b200 import denoiser as DN

from test_gpu_denoiser import _bf, _conv_ref, _features, _p, _random_params, _torch_net, _up2

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

N, H, W = 3, 700, 520   # 15 strips of 128 pixels: 35 rows a CTA on 148 SMs


def _run(x, xh, cin, cout, wt, mask, transposed, outs):
    scratch = torch.empty(L.lib().gs_conv3x3_scratch_bytes(cin, cout), dtype=torch.uint8, device="cuda")
    err = torch.zeros(4, dtype=torch.int32, device="cuda")
    n, h, w = x.shape[:3]
    L.check(L.lib().gs_conv3x3_bf16(_p(x), _p(xh), n, h, w, cin, cout, _p(wt), None, 0, transposed, _p(mask),
                                    _p(outs[0]), _p(outs[1]), _p(scratch), _p(err), None), "gs_conv3x3_bf16")
    torch.cuda.synchronize()
    assert int(err[0]) == 0


def _check(outs, ref):
    scale = float(ref.abs().max())
    assert float((outs[1] - ref).abs().max()) <= 1e-4 * scale + 1e-6
    assert float((outs[0].float() - ref).abs().max()) <= 8e-3 * scale


def _outs(channels):
    return (torch.full((N, H, W, channels), float("nan"), device="cuda", dtype=torch.bfloat16),
            torch.full((N, H, W, channels), float("nan"), device="cuda"))


@pytest.mark.parametrize("cin,cout,half", [(16, 32, False), (32, 32, False), (32, 16, False), (32, 32, True)])
@pytest.mark.parametrize("masked", [False, True])
def test_long_runs(cin, cout, half, masked):
    g = torch.Generator(device="cuda").manual_seed(3 * cin + cout + half)
    x = torch.randn(N, H, W, cin, device="cuda", generator=g).bfloat16()
    xh = torch.randn(N, H // 2, W // 2, cin, device="cuda", generator=g).bfloat16() if half else None
    wt = (torch.randn(3, 3, cin, cout, device="cuda", generator=g) * 0.2).float()
    mask = torch.randn(N, H, W, cout, device="cuda", generator=g).bfloat16() if masked else None
    outs = _outs(cout)
    _run(x, xh, cin, cout, wt, mask, 0, outs)
    ref = _conv_ref(_bf(x.float() + _up2(xh.float())) if half else x.float(), _bf(wt))
    _check(outs, torch.where(mask.float() > 0, ref, torch.zeros_like(ref)) if masked else ref)


@pytest.mark.parametrize("cin,cout", [(16, 32), (32, 32), (32, 16)])
def test_long_runs_of_the_input_gradient(cin, cout):
    g = torch.Generator(device="cuda").manual_seed(cin + 7 * cout)
    dy = torch.randn(N, H, W, cout, device="cuda", generator=g).bfloat16()
    wt = (torch.randn(3, 3, cin, cout, device="cuda", generator=g) * 0.2).float()
    outs = _outs(cin)
    _run(dy, None, cin, cout, wt, None, 1, outs)
    flipped = _bf(wt).flip(0, 1).transpose(2, 3)   # [tap'][cout][cin]
    _check(outs, _conv_ref(dy.float(), flipped))


def test_long_runs_of_the_network():
    x = _features(N, H, W, 5)
    flat = _random_params(6)
    flat_bf = flat.copy()
    o = 0
    for cin, cout in DN.LAYERS:
        k = 9 * cin * cout
        flat_bf[o:o + k] = torch.from_numpy(flat[o:o + k]).bfloat16().float().numpy()
        o += k + cout
    out = torch.full((N, H, W, 16), float("nan"), device="cuda")
    with DN.Denoiser(0) as d:
        d.set_params(flat)
        d.forward(x.data_ptr(), N, H, W, out.data_ptr())
        torch.cuda.synchronize()
        d.status()
    ref = _torch_net(x.float(), flat_bf)
    assert float((out - ref).abs().max()) <= 1e-2 * float(ref.abs().max())
