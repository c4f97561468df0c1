"""The launchers raise a kernel's shared-memory limit on every device a process
launches on (the limit is an attribute per device): the helper they share,
compiled from the library's header on the host, runs its action once on each
device, every time on devices beyond its 64 bits, and never lets a thread pass
before the action has run for the thread's device."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CUDA = Path("/usr/local/cuda/include")

SOURCE = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "gs_internal.h"
int main() {
    gs::OncePerDevice once;
    int runs[66] = {};
    for (int pass = 0; pass < 3; ++pass)
        for (int dev = -1; dev < 65; ++dev) once(dev, [&] { ++runs[dev + 1]; });
    for (int dev = -1; dev < 65; ++dev)
        if (runs[dev + 1] != (dev < 0 || dev > 63 ? 3 : 1)) return std::printf("device %d: %d runs\n", dev, runs[dev + 1]), 1;
    for (int round = 0; round < 200; ++round) {
        gs::OncePerDevice shared;
        std::atomic<int> set[2] = {{0}, {0}};
        std::atomic<int> early{0};
        std::vector<std::thread> threads;
        for (int t = 0; t < 8; ++t)
            threads.emplace_back([&, t] {
                shared(t & 1, [&] { std::this_thread::yield(); set[t & 1] = 1; });
                if (!set[t & 1]) ++early;
            });
        for (auto& t : threads) t.join();
        if (early) return std::printf("%d threads went on without the attribute\n", early.load()), 1;
    }
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not CUDA.exists(), reason="g++ and the CUDA headers are needed")
def test_once_per_device(tmp_path):
    (tmp_path / "once.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I", str(ROOT / "gamesplat_b200" / "csrc"), "-I", str(CUDA),
                    str(tmp_path / "once.cpp"), "-o", str(tmp_path / "once")], check=True)
    run = subprocess.run([str(tmp_path / "once")], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout
