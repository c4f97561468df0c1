"""The weight-gradient kernel's strips (128 pixels by up to 4 rows, fewer rows on
small images): against torch at sizes where strips, K-steps of 16 pixels and row
bands end raggedly, from one pixel to more strips than the GPU has SMs, with and
without a bias gradient and with a dw that is not 16-byte aligned.  The operands
are bf16, products exact in fp32, sums fp32: 1e-3 of the scale, as for whole
images."""
from __future__ import annotations

import ctypes as C

import pytest

from gamesplat_b200 import _lib as L

from test_gpu_denoiser import _bf, _up2

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("cin,cout,half", [(16, 32, False), (32, 32, False), (32, 16, False), (32, 32, True)])
@pytest.mark.parametrize("n,h,w,shift", [(1, 2, 2, 0), (1, 3, 17, 1), (2, 5, 129, 0), (1, 7, 255, 1), (3, 130, 140, 0),
                                         (8, 301, 33, 0)])
def test_weight_gradient_strips(cin, cout, half, n, h, w, shift):
    g = torch.Generator(device="cuda").manual_seed(cin + 3 * cout + h)
    x = torch.randn(n, h, w, cin, device="cuda", generator=g).bfloat16()
    xh = torch.randn(n, h // 2, w // 2, cin, device="cuda", generator=g).bfloat16() if half else None
    dy = torch.randn(n, h, w, cout, device="cuda", generator=g).bfloat16()
    store = torch.zeros(9 * cin * cout + shift, device="cuda")
    db = None if shift else torch.zeros(cout, device="cuda")
    err = torch.zeros(4, dtype=torch.int32, device="cuda")

    def p(t):
        return None if t is None else C.c_void_p(t.data_ptr())

    L.check(L.lib().gs_conv3x3_wgrad_bf16(p(x), p(xh), n, h, w, cin, cout, p(dy),
                                          C.c_void_p(store.data_ptr() + 4 * shift), p(db), p(err), None),
            "gs_conv3x3_wgrad_bf16")
    torch.cuda.synchronize()
    assert int(err[0]) == 0
    dw = store[shift:].view(3, 3, cin, cout)
    xin = _bf(x.float() + _up2(xh.float(), h, w)) if half else x.float()
    ref = torch.nn.grad.conv2d_weight(xin.double().permute(0, 3, 1, 2), (cout, cin, 3, 3),
                                      dy.double().permute(0, 3, 1, 2), padding=1).permute(2, 3, 1, 0)
    assert float((dw - ref).abs().max()) <= 1e-3 * float(ref.abs().max())
    if db is not None:
        dbr = dy.double().sum(dim=(0, 1, 2))
        assert float((db - dbr).abs().max()) <= 1e-3 * float(dbr.abs().max())
