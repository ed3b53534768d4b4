"""The fast and scores builds of the group kernels against the general build.

Both builds of a group kind run the same method on the same Philox streams,
and every sum in the same order, so on the same model their trajectories are
bit-identical; the general build keeps the direct form of each pass.  A
reference-compatibility switch selects it: TL_FLAG_COMPAT_CRIT changes only
the criticality of 2S reactions (tau_leaping/functions.h:115), and the
networks here have none.  Sizes sit at the edges of the passes' tiles: blocks
of four channels, turns of a group's lanes, several turns and queues.
"""
import numpy as np
import pytest

from tau_leaping_gb300 import Model, _ffi

pytestmark = pytest.mark.gpu

KINDS = {"lanes8": _ffi.VARIANT_LANES8, "lanes16": _ffi.VARIANT_LANES16, "warp": _ffi.VARIANT_WARP,
         "cta": _ffi.VARIANT_CTA}


def network(N, M, seed, pop_bits, x_max=3000):
    """M channels on N species: no reactant, S or S + S'; 0-3 products of
    stoichiometry 1-3; rates over four decades, so that the leaps' means lie
    on both sides of 10 and far below 1, and a few populations are critical."""
    rng = np.random.default_rng(seed)
    cols = []
    for j in range(M):
        order = int(rng.choice([0, 1, 1, 2])) if N > 1 else int(rng.choice([0, 1]))
        re = rng.choice(N, size=order, replace=False)
        rest = [i for i in range(N) if i not in re]
        n_prod = int(rng.integers(0, min(3, len(rest)) + 1))
        pr = rng.choice(rest, size=n_prod, replace=False) if n_prod else []
        col = sorted([(int(i), -1) for i in re] + [(int(i), int(rng.integers(1, 4))) for i in pr])
        cols.append((col, order))
    x0 = rng.integers(0, x_max, size=N)
    x0[rng.random(N) < 0.1] = 3
    rate = [10.0 ** rng.uniform(-2, 2) * (x_max ** (1 - o)) for _, o in cols]
    cp = np.cumsum([0] + [len(c) for c, _ in cols])
    return Model.from_arrays(x0, rate, cp, [i for c, _ in cols for i, _ in c], [v for c, _ in cols for _, v in c],
                             pop_bits=pop_bits)


@pytest.mark.parametrize("kind", list(KINDS))
@pytest.mark.parametrize("N,M", [(1, 1), (2, 3), (5, 4), (7, 33), (40, 64), (31, 127), (33, 257), (129, 1025)])
def test_builds_are_bit_identical(kind, N, M):
    for pop_bits in (32, 64):
        m = network(N, M, 100 * N + M, pop_bits)
        kw = dict(t_final=0.05, n=70, seed=3, intervals=2, variant=KINDS[kind], keep_samples=True, max_steps=250,
                  allow_truncation=True)
        for eps in (0.03, 0.5):  # 0.5: larger leaps, some rejected
            a = m.simulate(eps=eps, **kw)
            b = m.simulate(eps=eps, flags=_ffi.FLAG_COMPAT_CRIT, **kw)
            assert np.array_equal(a.samples, b.samples)
            assert (a.leaps, a.ssa_steps, a.rejections) == (b.leaps, b.ssa_steps, b.rejections)
            assert a.leaps + a.ssa_steps > 0
