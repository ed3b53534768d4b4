"""The kernel that bench.py names is that of the plan that ran."""
import sys
from pathlib import Path
from types import SimpleNamespace

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT))

import bench  # noqa: E402


def test_kernel_is_named_from_the_plan():
    def plan(variant, grid, block):
        return SimpleNamespace(variant=variant, grid=grid, block_threads=block)

    # dimer: four lanes a realization up to one wave, one lane past it
    assert bench.kernel_of(plan(1, 313, 128), 10_000) == "k_tiny"
    assert bench.kernel_of(plan(1, 16, 32), 32) == "k_tiny"  # idle lanes count
    assert bench.kernel_of(plan(1, 907, 128), 29_000) == "k_tiny"
    assert bench.kernel_of(plan(1, 469, 128), 60_000) == "k_fast"
    assert bench.kernel_of(plan(1, 782, 128), 100_000) == "k_fast"
    # lane, warp and CTA groups
    assert bench.kernel_of(plan(8, 608, 256), 100_000) == "k_fast"
    assert bench.kernel_of(plan(2, 572, 224), 4000) == "k_fast"
    assert bench.kernel_of(plan(3, 1216, 128), 65_536) == "k_fast"
