"""The scores builds against the general build, and the cases that the tests of
the unscored builds leave out.

A scored run draws the same trajectories in every build of a group kind: final
means and step counts are equal.  Scores are FP32 sums of the same terms, one a
step, so two builds differ by rounding alone: a score by at most steps x 2^-23 of
its largest partial sum, some ten standard deviations sd at most, and a gradient,
the covariance with a population, by sd(x) times that.  Its standard error is about
sd(x) sd / sqrt(n): the tolerance is 10 sqrt(n) steps 2^-23 of it.
"""
import numpy as np
import pytest

from tau_leaping_gb300 import Model, _ffi
from tau_leaping_gb300.model import simulate_batch
from tests.test_gpu_group_builds import KINDS, assert_same, network

pytestmark = pytest.mark.gpu

GENERAL = _ffi.FLAG_COMPAT_CRIT


def closed_network(N, M, seed, bits=32, x_max=3000):
    """Conversions S -> S', S + S' -> S'' or S'' + S''', and a few births at a
    constant rate: populations do not grow on themselves, so that a run without a
    cap ends.  No 2S channel: the switch of GENERAL changes nothing."""
    rng = np.random.default_rng(seed)
    cols, rate = [], []
    for j in range(M):
        order = 0 if j % 16 == 15 else 2 if N > 2 and j % 3 == 2 else 1
        pick = [int(i) for i in rng.choice(N, size=min(N, order + int(rng.integers(1, 3))), replace=False)]
        re, pr = pick[:order], pick[order:][:max(order, 1)]
        cols.append(sorted([(i, -1) for i in re] + [(i, 1) for i in pr]))
        rate.append(10.0 ** rng.uniform(-1, 1) * float(x_max) ** (1 - order))
    x0 = rng.integers(x_max // 2, x_max, size=N)
    x0[rng.random(N) < 0.1] = 3
    cp = np.cumsum([0] + [len(c) for c in cols])
    return Model.from_arrays(x0, rate, cp, [i for c in cols for i, _ in c], [v for c in cols for _, v in c], pop_bits=bits)


def assert_same_gradients(a, b, n):
    assert np.array_equal(a["mean_final"], b["mean_final"])
    assert (a["leaps"], a["ssa_steps"]) == (b["leaps"], b["ssa_steps"])
    steps = (a["leaps"] + a["ssa_steps"]) / n
    assert steps > 0
    tol = 10 * np.sqrt(n) * steps * 2.0**-23
    assert np.all(np.abs(a["grad"] - b["grad"]) <= tol * b["stderr"])
    assert np.allclose(a["stderr"], b["stderr"], rtol=10 * tol, atol=0)
    assert (b["stderr"] > 0).any()


def assert_ends(m, n, **kw):
    """Scored runs take no cap: the same trajectories under one first."""
    assert m.simulate(n=n, max_steps=4000, allow_truncation=True, **kw).truncated == 0


def check(m, n, **kw):
    kw = dict(dict(seed=3, tracked=[0, m.n_species - 1]), **kw)
    assert_ends(m, n, **kw)
    a = m.sensitivity(n=n, **kw)
    assert_same_gradients(a, m.sensitivity(n=n, flags=GENERAL, **kw), n)
    return a


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("kind", ["thread", "lanes8", "warp", "cta"])
@pytest.mark.parametrize("N,M", [(3, 4), (4, 3), (7, 8), (5, 7), (16, 16), (13, 15), (20, 32), (20, 31), (40, 64), (33, 70), (60, 257)])
def test_scores_builds_match_the_general_build(kind, N, M, bits):
    """Four, eight and sixteen lanes, and one, for thread groups; M a multiple of
    four (scores four at a time) and not."""
    if kind == "thread" and M > 33:
        pytest.skip("thread groups are for small models")
    check(closed_network(N, M, 100 * N + M, bits), 80, t_final=0.3, variant=KINDS[kind])


@pytest.mark.parametrize("n", [80, 20000, 80000])
def test_scores_of_thread_groups_of_every_ensemble_size(n):
    """Four lanes a realization and, past one wave, one."""
    check(closed_network(4, 4, 5), n, t_final=0.1, variant=_ffi.VARIANT_THREAD)


@pytest.mark.parametrize("kind", ["thread", "warp", "cta"])
@pytest.mark.parametrize("N,M", [(4, 9), (12, 16), (14, 31), (30, 32), (33, 40)])
def test_scores_of_direct_method_steps(kind, N, M):
    m = closed_network(N, M, N + M, x_max=12)
    assert check(m, 60, t_final=0.5, variant=KINDS[kind])["ssa_steps"] > 0


@pytest.mark.parametrize("N", [128, 4096, 4099])
def test_scores_in_global_memory(N):
    """Slots past a quarter of shared memory leave their scores there."""
    check(closed_network(128, 256, 7) if N == 128 else Model.generate("chain", n_species=N), 60, t_final=0.1)


@pytest.mark.parametrize("N,M,x_max,t", [(64, 128, 3000, 0.2), (70, 131, 3000, 0.2), (150, 400, 3000, 0.1),
                                         (64, 128, 8, 0.2), (130, 141, 6, 0.2)])
@pytest.mark.parametrize("bits", [32, 64])
def test_teams_match_warps(N, M, x_max, t, bits):
    """Four warps a realization: leaps and direct-method steps, with scores and
    without."""
    m = closed_network(N, M, N + M, bits, x_max=x_max)
    kw = dict(t_final=t, n=50, seed=3, intervals=2, keep_samples=True, max_steps=200, allow_truncation=True)
    a, b = m.simulate(**kw), m.simulate(flags=GENERAL, variant=_ffi.VARIANT_WARP, **kw)
    assert (a.variant, a.block_threads, a.grid) == (_ffi.VARIANT_WARP, 128, 50)  # a team each
    assert np.array_equal(a.samples, b.samples) and (a.leaps, a.ssa_steps) == (b.leaps, b.ssa_steps)
    assert a.ssa_steps > 0 if x_max < 10 else a.leaps > 0
    s = check(m, 50, t_final=t / 4)
    assert s["ssa_steps"] > 0 if x_max < 10 else s["leaps"] > 0


@pytest.mark.parametrize("seeds", [(3, 3), (3, 4)])
@pytest.mark.parametrize("n_big", [20, 3000])
def test_scored_batches_match_their_own_runs(seeds, n_big):
    """Teams (few large realizations of one seed), warps, and lanes of small items."""
    big, small = closed_network(64, 130, 8), closed_network(6, 11, 5)
    items = [dict(model=big, t_final=0.02, n=n_big, seed=seeds[0], tracked=[0, 63], sensitivity=True),
             dict(model=small, t_final=0.2, n=300, seed=seeds[1], tracked=[0, 5], sensitivity=True),
             dict(model=small, t_final=0.1, n=45, seed=seeds[1], tracked=[1])]
    for it in items:
        assert_ends(it["model"], it["n"], t_final=it["t_final"], seed=it["seed"])
    out = simulate_batch(items)
    slow = simulate_batch([dict(it, flags=GENERAL) for it in items])
    for it, a, b in zip(items, out, slow):
        if it.get("sensitivity"):
            assert_same_gradients(a, b, it["n"])
            one = it["model"].sensitivity(it["t_final"], it["n"], seed=it["seed"], tracked=it["tracked"],
                                          variant=_ffi.VARIANT_WARP if it["model"] is big else _ffi.VARIANT_THREAD)
            assert_same_gradients(a, one, it["n"])
        else:
            assert np.array_equal(a["mean"], b["mean"]) and a["leaps"] == b["leaps"]


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("N,M,two_s", [(1, 1, False), (2, 3, False), (5, 4, False), (16, 16, True), (7, 33, False),
                                       (40, 64, True), (31, 127, False), (33, 257, False), (129, 1025, True)])
def test_builds_are_compared_on_runs_that_end(kind, N, M, two_s):
    """The sizes of the bit-identity test with a result in each: int64, and
    int32 over the few steps in which no population overflows."""
    if kind == "thread" and M > 33:
        pytest.skip("thread groups are for small models")
    for bits, steps in ((64, 250), (32, 12)):
        m, general = network(N, M, 100 * N + M, bits, two_s=two_s)
        for eps in (0.03, 0.5):
            assert assert_same(m, general, variant=KINDS[kind], eps=eps, max_steps=steps) is not None


@pytest.mark.parametrize("kind", list(KINDS))
def test_int32_overflow_is_an_error_in_every_build(kind):
    """Births past 2^31 - 1 in a leap."""
    n = 33 if kind != "thread" else 3
    cols = [[(0, 5)]] + [[(i, -1), ((i + 1) % n, 1)] for i in range(1, n)]
    cp = np.cumsum([0] + [len(c) for c in cols])
    m = Model.from_arrays([2**31 - 5000] + [1000] * (n - 1), [1e4] + [1.0] * (n - 1), cp, [i for c in cols for i, _ in c],
                          [v for c in cols for _, v in c], pop_bits=32)
    for flags in (0, GENERAL):
        with pytest.raises(_ffi.TLError) as e:
            m.simulate(1.0, 40, seed=3, variant=KINDS[kind], flags=flags, max_steps=500, allow_truncation=True)
        assert e.value.status == 4
