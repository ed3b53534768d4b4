"""Calls that choose between builds and plans: whatever is launched, the
results are those of the same group kind launched directly."""
import numpy as np
import pytest

from tests.test_gpu_group_builds import KINDS, assert_same, network

from tau_leaping_gb300 import Model, _ffi
from tau_leaping_gb300.model import simulate_batch

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
    kw = dict(t_final=0.002, n=152, seed=3, tracked=[0])
    models = [Model.generate("toy") for _ in range(3)]  # each handle measures for itself
    planned = min(m.simulate(**kw).kernel_ms for m in models for _ in range(3))
    measured = min(m.simulate(flags=_ffi.FLAG_AUTOTUNE_MEASURE, **kw).kernel_ms for m in models for _ in range(3))
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


def rate_sets_of(m, sets, seed=4):
    d = m.desc()["rate"]
    return d[None, :] * np.random.default_rng(seed).lognormal(0.0, 0.3, size=(sets, len(d)))


@pytest.mark.parametrize("N,M,two_s", [(3, 4, False), (5, 4, True), (12, 16, True), (31, 63, True), (40, 64, False)])
@pytest.mark.parametrize("bits", [32, 64])
def test_rate_sets_reach_every_build(N, M, two_s, bits):
    """The sets go to the device in the form that the build reads; with the
    model's own rates in a set, its realizations are the model's."""
    m, general = network(N, M, 5, bits, two_s=two_s)
    rs = rate_sets_of(m, 3)
    rs[0] = m.desc()["rate"]
    kw = dict(t_final=0.02, n=40, seed=3, keep_samples=True, max_steps=200, allow_truncation=True)
    a, b = m.simulate(rate_sets=rs, **kw), m.simulate(rate_sets=rs, flags=general, **kw)
    assert np.array_equal(a.samples, b.samples) and a.leaps + a.ssa_steps == b.leaps + b.ssa_steps > 0
    assert np.array_equal(a.samples[0], m.simulate(**kw).samples[0])
    c = m.simulate(rate_sets=rs, flags=_ffi.FLAG_AUTOTUNE_MEASURE, **kw)
    d = m.simulate(rate_sets=rs, variant=c.variant, block_threads=c.block_threads, **kw)
    assert np.array_equal(c.samples, d.samples)
    # rates that cannot be halved exactly take the general build
    rs[1] = rs[1] * 1e-38
    a, b = m.simulate(rate_sets=rs, **kw), m.simulate(rate_sets=rs, flags=general, **kw)
    assert np.array_equal(a.samples, b.samples)
    items = [dict(model=m, t_final=0.02, n=40, seed=3, tracked=[0], rate_sets=rate_sets_of(m, 3), sensitivity=q, max_steps=200)
             for q in (True, False)]
    try:
        out = simulate_batch(items)
    except _ffi.TLError as e:
        assert e.status in (4, 5)
        return
    assert np.array_equal(out[0]["mean"], out[1]["mean"]) and out[0]["leaps"] == out[1]["leaps"]


def test_bad_rates_are_found_in_any_set():
    m = Model.generate("toy")
    for bad in (np.nan, np.inf, -np.inf, -1e-300, -np.nan):
        for at in ((0, 0), (1, 17), (2, 255)):
            rs = rate_sets_of(m, 3)
            rs[at] = bad
            with pytest.raises(_ffi.TLError) as e:
                m.simulate(1e-5, 4, tracked=[0], rate_sets=rs)
            assert e.value.status == 12
    rs = rate_sets_of(m, 3)
    rs[1, 3], rs[2, 4] = -0.0, 0.0
    assert m.simulate(1e-5, 4, tracked=[0], rate_sets=rs).status == 0


def test_many_rate_sets_cost_the_host_one_pass():
    """20 000 sets of 256 rates: 0.8 ns of host time a rate in one pass, 2.4 ns
    where both forms were made, zeroed and copied."""
    m = Model.generate("toy")
    rs = rate_sets_of(m, 20000)
    host = min(r.total_ms - r.kernel_ms for r in (m.simulate(2e-6, 1, tracked=[0], rate_sets=rs) for _ in range(5)))
    assert host * 1e6 / rs.size < 1.6, host


@pytest.mark.parametrize("bits", [32, 64])
def test_small_models_past_one_wave_take_one_lane_each(bits):
    """60 000 dimer realizations to t = 5e-4 took 1.44 ms on four lanes each, of
    which 29 184 realizations are resident, and 1.17 ms on one; 29 000 stay on four.
    The realizations are the same on either."""
    m = Model.generate("dimer", pop_bits=bits)
    a, b = (m.simulate(5e-4, n, seed=3, tracked=[0, 1], keep_samples=True) for n in (29000, 60000))
    assert b.grid * b.block_threads < 60000 + b.block_threads  # a lane each
    assert a.grid * a.block_threads >= 4 * 29000
    assert np.array_equal(a.samples, b.samples[:, :29000])


@pytest.mark.parametrize("n_items,n", [(16, 3100), (16, 8192)])
def test_batches_of_small_items_on_one_lane_each(n_items, n):
    """49 600 and 131 072 realizations: the builds at three and four CTAs an SM;
    every set equals its part of a run of its own."""
    m = Model.generate("dimer")
    rs = rate_sets_of(m, n_items)
    for sens in (False, True):
        out = simulate_batch([dict(model=m, t_final=0.002, n=n, seed=9, tracked=[0, 1], rate_sets=rs, sensitivity=sens)])[0]
        one = m.simulate(0.002, n, seed=9, tracked=[0, 1], rate_sets=rs)
        assert np.array_equal(out["mean"], one.mean) and out["leaps"] == one.leaps


@pytest.mark.parametrize("N", [312, 320, 328, 332])
@pytest.mark.parametrize("bits", [32, 64])
def test_wide_models_at_the_edge_of_shared_memory(N, bits):
    """48 672 to 55 112 channels: a queue of fewer turns, then the propensities
    in global memory; the same realizations as with all of it there, from the
    static entry as well, which has no room for those slots.  At 0.6 to 0.75 of the
    general build's time, which these models had fallen back to."""
    m = Model.generate("colloid", n_species=N, pop_bits=bits)
    kw = dict(t_final=0.002, n=200, seed=3, tracked=[0, 1, N - 1])
    a = m.simulate(keep_samples=True, **kw)
    b = m.simulate(keep_samples=True, flags=_ffi.FLAG_GLOBAL_SLOTS, variant=_ffi.VARIANT_CTA, **kw)
    assert np.array_equal(a.samples, b.samples) and a.leaps + a.ssa_steps == b.leaps + b.ssa_steps > 0
    s = m.simulate_static(**kw)
    assert np.array_equal(s.mean, a.mean) and (s.leaps, s.ssa_steps) == (a.leaps, a.ssa_steps)
    # the general build in the same launch: populations far from critical, so the same trajectories
    t, u = (min(m.simulate(flags=f, **dict(kw, n=152, tracked=[0])).kernel_ms for _ in range(5)) for f in (0, _ffi.FLAG_COMPAT_CRIT))
    assert t <= 0.9 * u, (t, u)


@pytest.mark.parametrize("family,kw,t", [("dimer", {}, 0.01), ("toy", {}, 0.0005), ("colloid", dict(n_species=60), 0.002),
                                         ("toy", dict(n_species=33, n_channels=61, seed=4), 0.001)])
def test_tables_are_there_for_whatever_runs_first(family, kw, t):
    """Each build's tables go to the device with the first launch that reads
    them, from every entry and in any order; the static entry allocates nothing."""
    import torch

    def fresh():
        return Model.generate(family, **kw)

    run = dict(t_final=t, n=64, seed=3, tracked=[0, 1])
    compat = dict(run, flags=_ffi.FLAG_COMPAT_REFERENCE)
    want, want_c = fresh().simulate(**run), fresh().simulate(**compat)

    def same(r, w):
        assert np.array_equal(r.mean, w.mean) and (r.leaps, r.ssa_steps) == (w.leaps, w.ssa_steps)

    m = fresh()
    x = m.desc()["x0"]
    ev = m.eval_leap(x)
    m.simulate_static(**run)
    m = fresh()
    m.eval_leap(x)
    free = torch.cuda.mem_get_info(0)[0]
    same(m.simulate_static(**run), want)
    same(m.simulate_static(**compat), want_c)
    assert torch.cuda.mem_get_info(0)[0] == free
    m = fresh()
    same(m.simulate(**run), want)
    free = torch.cuda.mem_get_info(0)[0]
    same(m.simulate_static(**compat), want_c)
    assert torch.cuda.mem_get_info(0)[0] == free
    same(m.simulate(**compat), want_c)
    assert all(np.array_equal(ev[q], v) for q, v in m.eval_leap(x).items())
    m = fresh()
    same(m.simulate(**compat), want_c)
    same(m.simulate(**run), want)
    m = fresh()
    k = np.zeros((2, m.n_channels), np.int32)
    assert np.array_equal(m.replay(x, k), np.tile(x, (2, 1)))
    same(m.simulate(**run), want)
    m, q = fresh(), fresh()
    out = simulate_batch([dict(model=m, **run), dict(model=q, **run, sensitivity=True)])
    assert out[0]["leaps"] == out[1]["leaps"] and np.array_equal(out[0]["mean"], out[1]["mean"])
    m = fresh()
    r = m.simulate(**dict(run, flags=_ffi.FLAG_AUTOTUNE_MEASURE))
    same(m.simulate(variant=r.variant, block_threads=r.block_threads, **run), r)
    m = fresh()
    assert m.simulate(variant=_ffi.VARIANT_PLAIN, **dict(run, t_final=t / 10)).status == 0


def test_a_first_call_makes_only_the_tables_that_it_reads():
    """Colloid of 400 species: the first replay took 2.1 ms with both builds'
    tables and takes 1.1 ms with its own; the fast build's come with the first run."""
    import time

    def ms(f):
        t = time.perf_counter()
        f()
        return (time.perf_counter() - t) * 1e3

    first, later = [], []
    for _ in range(6):
        m = Model.generate("colloid", n_species=400)
        x, k = m.desc()["x0"], np.zeros((1, m.n_channels), np.int32)
        first.append(ms(lambda: m.replay(x, k)))
        a, b = (ms(lambda: m.simulate(1e-4, 32, tracked=[0])) for _ in range(2))
        later.append(a - b)
        m.close()
    assert min(first) <= 0.8 * (min(first) + min(later)), (first, later)
