"""The FP64 pair kernel with a fitted cutoff (pair_fp64_kernel) against the
plain-C oracle, at the sizes and settings where its branches differ.

Bound of one pair, relative, in half units in the last place (2^-53): with the
erfc / exp arithmetic (the oracle's, and the general kernel's) x carries up to 2
of them (r^2, the root, two products) and x^2 one more rounding, and exp(-x^2)
multiplies an error of x^2 by itself: 4.5 x^2. The fitted kernel rounds r^2 (2 of
them, multiplied by x^2 likewise) and is otherwise within 1e-15
(tests/test_fit64.py), as are the other factors' roundings."""
import numpy as np
import pytest

from oracle import oracle as O
from photons_p2p import abi
from photons_p2p.p2p import Session, make_params

pytestmark = pytest.mark.gpu

def pair_max(x, fitted):
    return (4.5 + (2.0 if fitted else 4.5)) * x * x * 2.0 ** -53 + 2e-15


SUM_MAX = 1e-12  # the FP64 form's bar for sums


def run(prm, pos, ip, npt, tt, ts, masses=None):
    with Session(0, prm) as s:
        return s.force_pass(pos, ip, npt, tt, ts, masses=masses)[0]


# every coefficient count of the far polynomial, and the general kernel
# (x_cut 0: none; 1, 4.5: out of the fit's range)
@pytest.mark.parametrize("x_cut", [0.0, 1.0, 1.25, 2.25, 2.8125, 3.5, 4.0, 4.5])
@pytest.mark.parametrize("soft", [abi.SOFT_CLAMP, abi.SOFT_PLUMMER])
def test_single_pairs_over_the_whole_range(gpu, x_cut, soft):
    rs, eps, n = 0.05, 1e-3, 4000
    g = np.random.default_rng(7)
    x = np.concatenate([np.geomspace(1e-4, 1.2 * (x_cut or 4.0), n - 400),
                        0.99 + np.linspace(-1e-2, 1e-2, 200),            # near / far
                        (x_cut or 4.0) * (1 + np.linspace(-1e-6, 1e-6, 200))])  # the cutoff's high word
    v = g.normal(size=(3, n))
    d = 2 * rs * x * v / np.linalg.norm(v, axis=0)
    pos = np.zeros((3, 2 * n))
    pos[:, 0::2] = g.random((3, n)) * 1e-3
    pos[:, 1::2] = pos[:, 0::2] + d
    leaf = np.arange(2 * n, dtype=np.int32)
    one = np.ones(2 * n, np.int32)
    tt, ts = leaf[0::2], leaf[1::2]
    acc = run(make_params(form=abi.FORM_PLAIN_FP64, soft_mode=soft, soften=eps, split_radius=rs, x_cut=x_cut,
                          mass=0.7), pos, leaf, one, tt, ts)
    ref, _ = O.p2p_lists(O.params(soft, eps, rs, x_cut, 0.7), pos, leaf, one, tt, ts)
    a, b = acc[:, 0::2], ref[:, 0::2]
    den = np.linalg.norm(b, axis=0)
    xr = np.linalg.norm(pos[:, 1::2] - pos[:, 0::2], axis=0) / (2 * rs)
    xs = np.sqrt(xr ** 2 + (eps / (2 * rs)) ** 2) if soft == abi.SOFT_PLUMMER else xr
    edge = np.abs(xs * xs - x_cut ** 2) < 1e-14 * x_cut ** 2  # rounding decides
    assert np.array_equal((den == 0) & ~edge, (np.linalg.norm(a, axis=0) == 0) & ~edge)
    use = (den > 0) & ~edge
    assert use.sum() > n // 2
    assert (np.linalg.norm(a - b, axis=0)[use] / den[use] / pair_max(xs[use], 1.25 <= x_cut <= 4.0)).max() <= 1.0


@pytest.mark.parametrize("warps", [1, 3, 8])
@pytest.mark.parametrize("stage", [32, 96, 512])
@pytest.mark.parametrize("masses", [False, True])
def test_leaf_sizes_rows_and_launch_shapes(gpu, warps, stage, masses):
    """Leaves of 0 to 70 particles (every group count, two and three slices),
    rows from one entry to all."""
    g = np.random.default_rng(warps * 100 + stage)
    npt = np.array([1, 2, 3, 4, 5, 8, 13, 29, 31, 32, 33, 64, 70, 0, 7, 40], np.int32)
    ip = np.concatenate([[0], np.cumsum(npt)[:-1]]).astype(np.int32)
    n = int(npt.sum())
    pos = g.random((3, n))
    tt = np.concatenate([np.full(k % 16 + 1, k % 16) for k in range(16)]).astype(np.int32)
    ts = np.concatenate([g.permutation(16)[:k % 16 + 1] for k in range(16)]).astype(np.int32)
    m = g.random(n) if masses else None
    prm = make_params(form=abi.FORM_PLAIN_FP64, soft_mode=abi.SOFT_PLUMMER, soften=0.01, split_radius=0.2,
                      x_cut=2.25, mass=0.3, warps_per_block=warps, stage_sources=stage)
    acc = run(prm, pos, ip, npt, tt, ts, m)
    ref, _ = O.p2p_lists(O.params(abi.SOFT_PLUMMER, 0.01, 0.2, 2.25, 0.3), pos, ip, npt, tt, ts, masses=m)
    den = np.linalg.norm(ref, axis=0)
    use = den > 0
    assert np.all(np.linalg.norm(acc, axis=0)[~use] == 0)
    assert (np.linalg.norm(acc - ref, axis=0)[use] / den[use]).max() <= SUM_MAX
    assert np.array_equal(acc, run(prm, pos, ip, npt, tt, ts, m))  # repeats bit for bit


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_a_position_that_is_not_finite_gives_what_the_general_kernel_gives(gpu, bad):
    """Only the sums that meet it are not finite, component by component as in
    the oracle's arithmetic."""
    pos = np.random.default_rng(1).random((3, 12))
    pos[1, 5] = bad
    ip, npt = np.array([0, 4, 8], np.int32), np.full(3, 4, np.int32)
    tt, ts = np.array([0, 0, 2, 2], np.int32), np.array([0, 1, 0, 2], np.int32)
    for soft in (abi.SOFT_CLAMP, abi.SOFT_PLUMMER):
        out = [run(make_params(form=abi.FORM_PLAIN_FP64, soft_mode=soft, soften=0.01, split_radius=0.2, x_cut=xc),
                   pos, ip, npt, tt, ts) for xc in (2.25, 1.2)]  # fitted; general kernel
        assert np.array_equal(np.isnan(out[0]), np.isnan(out[1]))
        assert np.isfinite(out[0][:, 8:]).all()


@pytest.mark.parametrize("soft", [abi.SOFT_CLAMP, abi.SOFT_PLUMMER])
def test_pairs_beyond_the_cutoff_add_nothing(gpu, soft):
    """Also where the pair's offset or the source's mass is infinite and the
    lane's other pairs are inside."""
    pos = np.full((3, 8), 0.5) + 0.01 * np.random.default_rng(2).random((3, 8))
    pos[2, 1] = np.inf  # a sink
    pos[0, 6] = 9.0     # a source with an infinite mass
    m = np.ones(8)
    m[6] = np.inf
    ip, npt = np.array([0, 4], np.int32), np.full(2, 4, np.int32)
    tt, ts = np.array([0], np.int32), np.array([1], np.int32)
    # (the clamp takes an infinite r^2 for 0 * inf = NaN, in the oracle's arithmetic too)
    fitted, general = (run(make_params(form=abi.FORM_PLAIN_FP64, soft_mode=soft, soften=0.01, split_radius=0.2,
                                       x_cut=xc), pos, ip, npt, tt, ts, masses=m) for xc in (2.25, 1.2))
    assert np.array_equal(np.isnan(fitted), np.isnan(general))
    for out in (fitted, general):
        assert np.isfinite(out[:, [0, 2, 3]]).all() and (out[:, [0, 2, 3]] != 0).any(axis=0).all()
        assert soft == abi.SOFT_CLAMP or (out[:, 1] == 0).all()
