"""Calls that choose between builds and plans: whatever is launched, the
results are those of the same group kind launched directly."""
import numpy as np
import pytest

from tau_leaping_gb300 import Model, _ffi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 152, 1000, 1217])
@pytest.mark.parametrize("bits", [32, 64])
def test_measured_mode_launches_the_plan_that_it_chose(n, bits):
    """Small ensembles of a warp-group model are planned as teams first; the
    measured plan is another kind's, with its own block and slots."""
    m = Model.generate("toy", pop_bits=bits)
    kw = dict(t_final=0.0005, n=n, seed=3, tracked=[0, 1], keep_samples=True)
    for _ in range(2):  # measured, then from the handle's cache
        r = m.simulate(flags=_ffi.FLAG_AUTOTUNE_MEASURE, **kw)
        same = m.simulate(variant=r.variant, block_threads=r.block_threads, **kw)
        assert np.array_equal(r.samples, same.samples)
        assert (r.leaps, r.ssa_steps, r.rejections) == (same.leaps, same.ssa_steps, same.rejections)


def test_measured_mode_is_no_slower_than_the_planned_launch():
    """Teams are planned, never asked for by a block: 152 toy realizations take
    9.8 ms on them and 10.7 ms on the fastest launch that a block asks for."""
    m = Model.generate("toy")
    kw = dict(t_final=0.002, n=152, seed=3, tracked=[0])
    planned = min(m.simulate(**kw).kernel_ms for _ in range(5))
    measured = min(m.simulate(flags=_ffi.FLAG_AUTOTUNE_MEASURE, **kw).kernel_ms for _ in range(5))
    assert measured <= 1.05 * planned, (measured, planned)
