"""Calls that choose between builds and plans: whatever is launched, the
results are those of the same group kind launched directly."""
import numpy as np
import pytest

from tests.test_gpu_group_builds import KINDS, assert_same, network

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


@pytest.mark.parametrize("kind", ["thread", "lanes8", "warp", "cta"])
@pytest.mark.parametrize("bits", [32, 64])
def test_direct_steps_below_zero_match_the_general_build(kind, bits):
    """A channel that lists a species twice as a reactant S + S takes two of
    it while one is left; the propensities of the steps that follow are
    products of |x| in every build."""
    cols = [[(0, -1), (0, -1), (1, 1)], [(1, -1), (0, 1)], [(0, -1), (2, 1)], [(2, -2), (0, 3)], [(3, -1), (0, 1)]]
    cols += [[(i, -1), ((i + 1) % 20, 1)] for i in range(4, 20)]
    cp = np.cumsum([0] + [len(c) for c in cols])
    x0 = [5, 4, 3, 2] + [2] * 16
    m = Model.from_arrays(x0, [0.5, 0.2, 0.3, 0.1, 0.2] + [0.1] * 16, cp, [i for c in cols for i, _ in c],
                          [v for c in cols for _, v in c], pop_bits=bits)
    kw = dict(t_final=50.0, n=200, seed=3, intervals=3, keep_samples=True, max_steps=150, allow_truncation=True,
              ssa_factor=10**9, n_critical=1, variant=KINDS[kind])
    a, b = m.simulate(**kw), m.simulate(flags=_ffi.FLAG_COMPAT_G, **kw)
    assert (b.samples < 0).any()
    assert np.array_equal(a.samples, b.samples)
    assert (a.leaps, a.ssa_steps, a.truncated) == (b.leaps, b.ssa_steps, b.truncated)


@pytest.mark.parametrize("kind", ["thread", "lanes8", "warp", "cta"])
def test_a_leap_from_below_zero_is_rejected_not_an_overflow(kind):
    """Direct-method steps take S below zero (S + S from one species), then
    births of A make the steps leaps: a leap that adds to S without lifting it to
    zero is rejected until its halvings run out, in every build."""
    cols = [[(0, -1), (0, -1)], [(0, 1)], [(1, 5)], [(1, -1)]] + [[(2 + i, -1), (2 + (i + 1) % 18, 1)] for i in range(18)]
    cp = np.cumsum([0] + [len(c) for c in cols])
    m = Model.from_arrays([1, 0] + [3] * 18, [20.0, 300.0, 1000.0, 1.0] + [0.01] * 18, cp, [i for c in cols for i, _ in c],
                          [v for c in cols for _, v in c], pop_bits=32)
    kw = dict(t_final=5.0, n=2000, seed=3, max_steps=150, allow_truncation=True, ssa_factor=1, variant=KINDS[kind])
    for flags in (0, _ffi.FLAG_COMPAT_CRIT):
        with pytest.raises(_ffi.TLError) as e:
            m.simulate(flags=flags, **kw)
        assert e.value.status == 12, (flags, str(e.value))


@pytest.mark.parametrize("kind", ["thread", "lanes8", "warp", "cta"])
@pytest.mark.parametrize("n_critical", [2**30 - 1, 2**30, 2**30 + 2**29, 2**31 - 1])
def test_thresholds_near_the_end_of_int32(kind, n_critical):
    """Twice the threshold leaves int32 from 2^30 on."""
    for bits in (32, 64):
        m, general = network(12, 16, 5, bits, two_s=True)
        r = assert_same(m, general, variant=KINDS[kind], n_critical=n_critical)
        assert r is not None


@pytest.mark.parametrize("variant,family,kw,t,n", [
    (_ffi.VARIANT_AUTO, "chain", dict(n_species=32), 0.5, 50000), (_ffi.VARIANT_AUTO, "chain", dict(n_species=64, pop_bits=64), 0.5, 50000),
    (_ffi.VARIANT_LANES2, "dimer", {}, 1.0, 4000), (_ffi.VARIANT_LANES4, "toy", {}, 0.001, 4000),
    (_ffi.VARIANT_LANES4, "chain", dict(n_species=128), 0.3, 4000), (_ffi.VARIANT_LANES16, "chain", dict(n_species=1024), 0.3, 30000)])
def test_narrow_groups_are_no_slower_than_the_general_build(variant, family, kw, t, n):
    """Narrow groups take the build that runs faster; on the fast one these runs
    took 1.2 to 3 times the general build's time."""
    m = Model.generate(family, **kw)
    run = dict(seed=3, tracked=[0], max_steps=200, allow_truncation=True, variant=variant, keep_samples=n <= 4000)
    a = [m.simulate(t, n, **run) for _ in range(5)]
    b = [m.simulate(t, n, flags=_ffi.FLAG_COMPAT_CRIT if family != "dimer" else _ffi.FLAG_COMPAT_G, **run) for _ in range(5)]
    assert min(r.kernel_ms for r in a) <= 1.1 * min(r.kernel_ms for r in b)
    assert np.allclose(a[0].mean, b[0].mean, rtol=0.02)
