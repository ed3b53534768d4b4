"""Step counts past 2^32: the Philox step counter has 32 bits, a cap on the
accepted steps 63."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

SOURCE = r"""
#include "tl_shared.h"
int main() {
    uint32_t step = 0xfffffffdu, epochs = 0;
    const uint32_t rej = 7;
    long long want = 0xfffffffdll - rej;
    for (int q = 0; q < 6; ++q) {
        if (tl::accepted(epochs, step, rej) != want + q) return 1;
        const uint32_t from = step++;
        epochs += tl::wrapped_past(step, from);
    }
    // right after a wrap, more rejections than the counter shows
    if (tl::accepted(epochs, step, rej) != (1ll << 32) + 3 - 7) return 2;
    epochs = 5;
    if (tl::accepted(epochs, 0u, 0xffffffffu) != (5ll << 32) - 0xffffffffll) return 3;
    // a block of direct-method steps over the wrap
    epochs = 1;
    step = 0xfffffff0u;
    for (int q = 1; q <= 40; ++q) {
        ++step;
        if (tl::accepted(epochs + tl::wrapped(step, q), step, 3u) != (1ll << 32) + 0xfffffff0ll - 3 + q) return 4;
    }
    return 0;
}
"""


def test_accepted_steps_past_the_counter(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    (tmp_path / "counts.cpp").write_text(SOURCE)
    exe = tmp_path / "counts"
    r = subprocess.run([gxx, "-std=c++17", "-I", str(ROOT / "tau_leaping_gb300" / "csrc"), str(tmp_path / "counts.cpp"),
                        "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert subprocess.run([str(exe)]).returncode == 0
