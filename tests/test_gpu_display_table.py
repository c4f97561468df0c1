"""The display LUT's float table is made in place of the uploaded lattice, in
launches that shrink towards its end: LUT sizes around the last launch's 1024
points and with many launches give the oracle's bits, and the largest LUT holds
16 bytes a lattice point."""
from __future__ import annotations

import numpy as np
import pytest

from gamesplat_b200 import Renderer
from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [3, 10, 11, 14, 65, 129, 256])
def test_table_of_every_point(n):
    rng = np.random.default_rng(n)
    lut = rng.integers(0, 65536, (n, n, n, 3), dtype=np.uint16)
    lut[0, 0, 0] = (0, 1, 65535)
    lut[-1, -1, -1] = (65535, 0, 1)
    img = (2.0 ** rng.uniform(-7.0, 3.0, (96, 128, 4))).astype(np.float16)
    img[0, 0, :3] = 0.0
    img[0, 1, :3] = np.float16(60000.0)
    ref = O.display(img, lut, -6.0, 2.0, 0.25)
    src = torch.from_numpy(img.view(np.uint16).copy()).cuda()
    dst = torch.empty((96, 128, 4), dtype=torch.float32, device="cuda")
    with Renderer(0) as r:
        r.set_display_lut(lut, -6.0, 2.0)
        r.display(src.data_ptr(), dst.data_ptr(), 128, 96, 0.25)
        torch.cuda.synchronize()
    assert np.array_equal(dst.cpu().numpy().view(np.uint32), ref.view(np.uint32))


def test_table_holds_16_bytes_a_point():
    n = 256
    lut = np.zeros((n, n, n, 3), np.uint16)
    with Renderer(0) as r:
        r.set_display_lut(np.zeros((2, 2, 2, 3), np.uint16), 0.0, 1.0)
        before = torch.cuda.mem_get_info()[0]
        r.set_display_lut(lut, 0.0, 1.0)
        held = before - torch.cuda.mem_get_info()[0]
    assert held <= 16 * n ** 3 + (4 << 20)   # and the allocator's 2 MiB granules
