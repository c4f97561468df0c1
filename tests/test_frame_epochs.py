"""The tags of the look-back words, compiled from the library's header on the
host: over the wrap of the epochs no frame has epoch 0 or its predecessor's, and
no (epoch, pass) of the sorts has the tag 0 of memory that was never written, or
another's tag."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CUDA = Path("/usr/local/cuda/include")

SOURCE = r"""
#include <cstdio>
#include "gs_internal.h"
int main() {
    // the first epochs, the last ones, and the first of the next round
    uint32_t e = 0;
    for (int frame = 0; frame < 8192; ++frame) {
        const uint32_t n = frame == 4096 ? gs::kEpochs - 2048u : gs::next_epoch(e);
        for (uint32_t p = 0; p < 4; ++p) {
            const uint32_t t = gs::sort_tag(n, p);
            if (n == 0u || n == e || t == 0u || (t >> 2) != n || (t & 3u) != p)
                return std::printf("epoch %u after %u, pass %u: tag %u\n", n, e, p, t), 1;
        }
        e = n;
    }
    if (e != 2048u) return std::printf("epoch %u at the end\n", e), 1;
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not CUDA.exists(), reason="g++ and the CUDA headers are needed")
def test_tags_over_the_wrap(tmp_path):
    (tmp_path / "tags.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", str(ROOT / "gamesplat_b200" / "csrc"), "-I", str(CUDA),
                    str(tmp_path / "tags.cpp"), "-o", str(tmp_path / "tags")], check=True)
    run = subprocess.run([str(tmp_path / "tags")], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout
