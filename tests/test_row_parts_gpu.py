"""Rows cut into shares whose sums are kept apart (passes with few leaves),
against one warp per row: the same sums up to the grouping of FP32 partials,
the same on every run, over several chunks, with masses, and replayed."""
import numpy as np
import pytest

from photons_p2p import abi
from photons_p2p.p2p import Session, make_params

pytestmark = pytest.mark.gpu


def leaves(sizes, g):
    npt = np.asarray(sizes, np.int32)
    ip = np.concatenate([[0], np.cumsum(npt)[:-1]]).astype(np.int32)
    return g.random((3, int(npt.sum()))), ip, npt


@pytest.mark.parametrize("sizes", [[1], [33], [0, 5, 0, 64], [32] * 40, [7, 70, 1, 31, 33] * 6],
                         ids=["one", "two_slices", "empty_leaves", "even", "uneven"])
@pytest.mark.parametrize("form", [abi.FORM_SPLIT, abi.FORM_KAHAN_FP32, abi.FORM_NAIVE_FP32, abi.FORM_PLAIN_FP64])
@pytest.mark.parametrize("masses", [False, True])
def test_shares_give_the_sums_of_whole_rows(gpu, sizes, form, masses):
    g = np.random.default_rng(len(sizes))
    pos, ip, npt = leaves(sizes, g)
    n = len(sizes)
    tt, ts = (a.ravel().astype(np.int32) for a in np.meshgrid(np.arange(n), np.arange(n), indexing="ij"))
    keep = g.random(tt.size) < 0.7  # rows of every length, some empty
    tt, ts = tt[keep], ts[keep]
    m = g.random(pos.shape[1]) if masses else None
    out = []
    for warps in (0, 1):
        p = make_params(form=form, soft_mode=abi.SOFT_PLUMMER, soften=0.02, split_radius=0.15, x_cut=2.25, mass=0.5)
        p.warps_per_leaf = warps
        with Session(gpu, p) as s:
            runs = [s.force_pass(pos, ip, npt, tt, ts, masses=m, chunk=c)[0] for c in (0, 0, max(1, tt.size // 3))]
        assert np.array_equal(runs[0], runs[1])
        out.append(runs)
    # FP32 partial sums grouped otherwise: each rounds by 2^-24 of the terms' sizes
    tol = 1e-12 if form == abi.FORM_PLAIN_FP64 else 1e-5
    ref = np.linalg.norm(out[1][0], axis=0)
    scale = np.maximum(ref, ref.mean() if ref.size else 0.0)
    for a in (out[0][0], out[0][2]):
        assert np.all(np.linalg.norm(a - out[1][0], axis=0) <= tol * scale)


def test_replayed_pass_starts_from_zero_shares(gpu):
    import torch

    g = np.random.default_rng(3)
    pos, ip, npt = leaves([20] * 30, g)
    tt = np.repeat(np.arange(30, dtype=np.int32), 30)
    ts = np.tile(np.arange(30, dtype=np.int32), 30)
    with Session(gpu, make_params(form=abi.FORM_SPLIT, soft_mode=abi.SOFT_PLUMMER, soften=0.02, split_radius=0.15,
                                  x_cut=2.25)) as s:
        want, _ = s.force_pass(pos, ip, npt, tt, ts)
        d = [torch.from_numpy(np.ascontiguousarray(a)).to(f"cuda:{gpu}") for a in (pos, ip, npt, tt, ts)]
        torch.cuda.synchronize()
        for _ in range(3):
            s.run_device(pos.shape[1], d[0].data_ptr(), 30, d[1].data_ptr(), d[2].data_ptr(), tt.size, d[3].data_ptr(),
                         d[4].data_ptr())
            s.end()
            got = np.zeros_like(want)
            s.accumulate(got)
            assert np.array_equal(got, want)
