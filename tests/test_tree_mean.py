"""The tree build's parallel form of the sampled mean's running sum (moves of the
sum within a binade, csrc/p2p_tree_kernels.cuh: MeanMoves) restated in numpy,
against the chain of FP64 additions it replaces, bit for bit."""
import math

import numpy as np
import pytest


def binade(s):
    if s == 0.0 or not math.isfinite(s):
        return None
    e = math.frexp(s)[1] - 1
    return (math.ldexp(1.0, e), math.ldexp(1.0, e - 53)) if -923 <= e <= 977 else None


def moves(x, s, half_u):
    """Cumulative sums of the samples' moves and their sizes, and which samples
    round by parity."""
    with np.errstate(all="ignore"):
        m = (s + x) - s
        return np.cumsum(m), np.cumsum(np.abs(m)), np.abs(x - m) == half_u


def parallel_sum(x, group):
    """Groups of samples at once; the group that holds a half or might leave
    the binade, sample by sample."""
    x = np.asarray(x, np.float64)
    s, i = 0.0, 0
    while i < len(x):
        b = binade(s)
        g = x[i:i + group]
        if b:
            total, size, half = moves(g, s, b[1])
            along = math.copysign(1.0, s) * total[-1]
            if (not half.any() and abs(s) - 0.5 * (size[-1] - along) > b[0]
                    and abs(s) + 0.5 * (size[-1] + along) < 2 * b[0]):
                s = s + float(total[-1])
                i += len(g)
                continue
        for v in g:
            s = s + float(v)
        i += len(g)
    return s


def chain(x):
    s = 0.0
    for v in x:
        s = s + float(v)
    return s


KINDS = {
    "uniform": lambda g, n: g.random(n),
    "ghosts": lambda g, n: g.random(n) * 1.1 - 0.05,
    "halves": lambda g, n: g.integers(-3, 9, n) * 2.0 ** -g.integers(30, 56, n),
    "signs": lambda g, n: g.normal(size=n),
    "scales": lambda g, n: g.random(n) * 10.0 ** g.integers(-18, 18, n),
    "equal": lambda g, n: np.full(n, 0.3),
    "nan": lambda g, n: np.where(np.arange(n) == n // 2, np.nan, g.random(n)),
    "inf": lambda g, n: np.where(np.arange(n) == n // 2, np.inf, g.random(n)),
    "tiny": lambda g, n: g.random(n) * 1e-300,
}


@pytest.mark.parametrize("kind", sorted(KINDS))
@pytest.mark.parametrize("n", [3, 31, 33, 513, 20000])
@pytest.mark.parametrize("group", [4, 16, 512])
def test_moves_give_the_chain_of_additions_bit_for_bit(kind, n, group):
    x = KINDS[kind](np.random.default_rng(n + group + len(kind)), n)
    a, b = parallel_sum(x, group), chain(x)
    assert a == b or (math.isnan(a) and math.isnan(b))
