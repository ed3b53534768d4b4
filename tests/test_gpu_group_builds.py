"""The fast and scores builds of the kernels against the general build.

The builds of a group kind run the same method on the same Philox streams,
and every sum in the same order, so on the same model their trajectories are
bit-identical; the general build keeps the direct form of each pass.  A
reference-compatibility switch selects it, one that changes nothing on the
model at hand: TL_FLAG_COMPAT_CRIT only concerns 2S reactions
(tau_leaping/functions.h:115), TL_FLAG_COMPAT_G reads a species' order from
the channel of its index (CSRMatrixPacked.cu:353), which is the right one
where that channel is 2S of it.  Sizes sit at the edges of the passes' tiles:
blocks of four channels, turns of a group's lanes, several turns and queues.
"""
import numpy as np
import pytest

from tau_leaping_gb300 import Model, _ffi
from tau_leaping_gb300.model import simulate_batch

pytestmark = pytest.mark.gpu

KINDS = {"thread": _ffi.VARIANT_THREAD, "lanes2": _ffi.VARIANT_LANES2, "lanes8": _ffi.VARIANT_LANES8,
         "lanes16": _ffi.VARIANT_LANES16, "warp": _ffi.VARIANT_WARP, "cta": _ffi.VARIANT_CTA}


def network(N, M, seed, pop_bits=32, x_max=3000, two_s=False):
    """M channels on N species: no reactant, S or S + S' (or first 2S of every
    species); 0-5 products of stoichiometry 1-3; rates over four decades, so
    that the leaps' means lie on both sides of 10 and far below 1, and a few
    populations are critical.  Returns the model and the switch that selects
    the general build."""
    rng = np.random.default_rng(seed)
    cols = []
    for j in range(M):
        if two_s and j < N:
            order, re, most = 2, [(j, -2)], 1
        else:
            order = int(rng.choice([0, 1, 1, 2])) if N > 1 else int(rng.choice([0, 1]))
            re, most = [(int(i), -1) for i in rng.choice(N, size=order, replace=False)], 3 if j else 5
        rest = [i for i in range(N) if i not in [i for i, _ in re]]
        n_prod = int(rng.integers(0, min(most, len(rest)) + 1))
        pr = rng.choice(rest, size=n_prod, replace=False) if n_prod else []
        cols.append((sorted(re + [(int(i), int(rng.integers(1, 4))) for i in pr]), order))
    x0 = rng.integers(0, x_max, size=N)
    x0[rng.random(N) < 0.1] = 3
    rate = [10.0 ** rng.uniform(-2, 2) * (float(x_max) ** (1 - o)) for _, o in cols]
    cp = np.cumsum([0] + [len(c) for c, _ in cols])
    m = Model.from_arrays(x0, rate, cp, [i for c, _ in cols for i, _ in c], [v for c, _ in cols for _, v in c],
                          pop_bits=pop_bits)
    return m, _ffi.FLAG_COMPAT_G if two_s else _ffi.FLAG_COMPAT_CRIT


def assert_same(m, general, **kw):
    kw = dict(dict(t_final=0.05, n=70, seed=3, intervals=2, keep_samples=True, max_steps=250, allow_truncation=True), **kw)

    def outcome(flags):
        try:
            return m.simulate(flags=flags, **kw)
        except _ffi.TLError as e:  # a growing network can leave int32, in either build
            assert e.status == 4
            return None

    a, b = outcome(0), outcome(general)
    if a is None or b is None:
        assert a is None and b is None
        return None
    assert np.array_equal(a.samples, b.samples)
    assert (a.leaps, a.ssa_steps, a.rejections, a.truncated) == (b.leaps, b.ssa_steps, b.rejections, b.truncated)
    assert a.leaps + a.ssa_steps > 0
    return a


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("N,M,two_s", [(1, 1, False), (2, 3, False), (5, 4, False), (16, 16, True), (7, 33, False),
                                       (40, 64, True), (31, 127, False), (33, 257, False), (129, 1025, True)])
def test_builds_are_bit_identical(kind, N, M, two_s):
    if kind == "thread" and M > 33:
        pytest.skip("thread groups are for small models")
    for pop_bits in (32, 64):
        m, general = network(N, M, 100 * N + M, pop_bits, two_s=two_s)
        for eps in (0.03, 0.5):  # 0.5: larger leaps, some rejected
            assert_same(m, general, variant=KINDS[kind], eps=eps)


@pytest.mark.parametrize("kind", list(KINDS))
def test_direct_method_steps_are_bit_identical(kind):
    """A handful of molecules: every step is a direct-method step."""
    for N, M, two_s in ((4, 9, False), (12, 16, True)):
        m, general = network(N, M, N + M, x_max=12, two_s=two_s)
        r = assert_same(m, general, variant=KINDS[kind], t_final=3.0)
        assert r.ssa_steps > 0


@pytest.mark.parametrize("kind", ["lanes8", "warp", "cta"])
@pytest.mark.parametrize("pairs", [1, 16, 37, 300])
def test_leaps_that_fire_a_critical_channel(kind, pairs):
    """Pairs A <-> B of 10^5 molecules, which set the leap, and species of
    about five molecules each, which are born and decay: one critical channel
    fires in most leaps, from any lane."""
    cols = []
    for q in range(pairs):
        a, b, s = 3 * q, 3 * q + 1, 3 * q + 2
        cols += [[(a, -1), (b, 1)], [(a, 1), (b, -1)], [(s, 1)], [(s, -1)]]
    x0 = np.tile([100000, 100000, 5], pairs)
    rate = np.tile([1.0, 1.0, 1.0 + 200.0 / pairs, 40.0 / pairs], pairs)
    cp = np.cumsum([0] + [len(c) for c in cols])
    m = Model.from_arrays(x0, rate, cp, [i for c in cols for i, _ in c], [v for c in cols for _, v in c])
    r = assert_same(m, _ffi.FLAG_COMPAT_CRIT, variant=KINDS[kind], n=40, t_final=0.2)
    assert r is not None and r.leaps > 0


@pytest.mark.parametrize("kind", ["lanes8", "warp", "cta"])
def test_rejected_leaps_that_fire_a_critical_channel(kind):
    """eps = 3 on few molecules: a retry selects among the critical channels
    of the state before the rejected leap."""
    for N, M in ((16, 32), (20, 70)):
        m, general = network(N, M, N + M, x_max=60)
        r = assert_same(m, general, variant=KINDS[kind], n=1000, t_final=0.5, eps=3.0)
        assert r is not None and r.rejections > 0


@pytest.mark.parametrize("n", [3, 1500, 9000, 21000])
def test_thread_groups_of_every_ensemble_size(n):
    """Lanes per realization and realizations per warp follow the ensemble."""
    m, general = network(6, 11, 5)
    assert_same(m, general, variant=_ffi.VARIANT_THREAD, n=n, t_final=0.02)


@pytest.mark.parametrize("kind", ["lanes16", "warp"])
@pytest.mark.parametrize("n", [31, 1217, 2600, 4001, 4864, 4865])
def test_ensembles_of_one_wave_on_even_ctas(kind, n):
    """Smaller CTAs where they share an ensemble out more evenly: the same
    realizations as on CTAs of 256 threads."""
    m, _ = network(12, 20, 5)
    kw = dict(t_final=0.01, n=n, seed=3, keep_samples=True, variant=KINDS[kind], max_steps=100, allow_truncation=True)
    a, b = m.simulate(**kw), m.simulate(block_threads=256, **kw)
    assert np.array_equal(a.samples, b.samples)
    assert 32 <= a.block_threads <= 256 and a.leaps + a.ssa_steps == b.leaps + b.ssa_steps > 0


@pytest.mark.parametrize("kind", ["thread", "lanes8", "warp", "cta"])
def test_wide_leaps_are_bit_identical(kind):
    """More than 10^8 firings in a leap: sums past int32 in between."""
    for pop_bits in (32, 64):
        m = Model.from_arrays([3 * 10**8, 10**9], [1.0, 1.0], [0, 2, 4], [0, 1, 0, 1], [-1, 1, 1, -1], pop_bits=pop_bits)
        assert_same(m, _ffi.FLAG_COMPAT_CRIT, variant=KINDS[kind], eps=0.4, t_final=1.0, n=9)


def test_global_propensities_and_batches_are_bit_identical():
    m, general = network(33, 257, 8)
    a = assert_same(m, general, variant=_ffi.VARIANT_CTA)
    kw = dict(t_final=0.05, n=70, seed=3, intervals=2, keep_samples=True, max_steps=250, allow_truncation=True)
    g = m.simulate(variant=_ffi.VARIANT_CTA, **dict(kw, flags=_ffi.FLAG_GLOBAL_SLOTS))
    assert np.array_equal(a.samples, g.samples)
    small, _ = network(6, 11, 5)
    items = [dict(model=q, t_final=0.004, n=n, seed=9, tracked=[0, 1], keep_samples=True) for q, n in ((m, 20), (small, 45))]
    fast = simulate_batch(items)
    slow = simulate_batch([dict(it, flags=general) for it in items])
    for x, y in zip(fast, slow):
        assert np.array_equal(x["samples"], y["samples"]) and x["leaps"] == y["leaps"]


@pytest.mark.parametrize("n_small,n_big", [(300, 2431), (20000, 40), (9, 2600)])
def test_batches_of_more_units_than_two_ctas_hold(n_small, n_big):
    """The batch kernel's register budget follows the number of units; every
    item equals its own call."""
    big, _ = network(33, 60, 8)
    small, _ = network(6, 11, 5)
    kw = dict(t_final=0.002, seed=9, keep_samples=True, tracked=[0, 1, 2])
    out = simulate_batch([dict(kw, model=small, n=n_small), dict(kw, model=big, n=n_big)])
    for r, m, n, v in ((out[0], small, n_small, _ffi.VARIANT_THREAD), (out[1], big, n_big, _ffi.VARIANT_WARP)):
        one = m.simulate(n=n, variant=v, **kw)
        assert np.array_equal(r["samples"], one.samples) and r["leaps"] == one.leaps


@pytest.mark.parametrize("n,K,intervals,sets", [(64, 64, 1, 1), (1001, 33, 2, 3), (257, 130, 1, 2)])
def test_statistics_of_many_columns(n, K, intervals, sets):
    """Means and deviations of 64 columns and more: exact integer sums, so
    within FP64 rounding of numpy's on the same samples."""
    m, _ = network(K, 2 * K, 7)
    rates = np.tile(m.desc()["rate"], (sets, 1))
    r = m.simulate(0.01, n, seed=5, intervals=intervals, keep_samples=True, rate_sets=rates, max_steps=50,
                   allow_truncation=True)
    x = r.samples.astype(np.float64)
    assert np.allclose(r.mean, x.mean(axis=1), rtol=1e-13, atol=1e-13)
    assert np.allclose(r.stddev, x.std(axis=1, ddof=1), rtol=1e-11, atol=1e-11)
