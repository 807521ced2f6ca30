"""A begin that is refused for lack of device memory leaves the session's counts as
they were: the result calls write as many numbers as the last pass had, and the
session runs the next pass."""
import ctypes

import numpy as np
import pytest

from photons_p2p import abi, lists as L, workloads as W
from photons_p2p.p2p import Session, params_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [abi.FORM_PLAIN_FP64, abi.FORM_SPLIT])
def test_result_keeps_the_last_pass_size(gpu, form):
    import torch

    # more than the device holds, so that no kernel sees these counts: 24 bytes a
    # particle for the sums (they are allocated) and 96 for the rows' shares
    huge = 2_100_000_000
    total = torch.cuda.get_device_properties(gpu).total_memory
    assert 24 * huge < total < 96 * huge
    cfg = W.c1_config()
    allpos, tag = W.with_ghosts(W.c1_positions(), cfg)
    tl = L.build_tree_lists(allpos, tag, cfg.maxleaf, cfg.box, cfg.cutoff_radius, cfg.open_angle)
    with Session(gpu, params_for(cfg, form, 1.0)) as s:
        want, _ = s.force_pass(tl.pos, tl.leaf_ipart, tl.leaf_npart, tl.task_t, tl.task_s)
        d = torch.zeros(64, dtype=torch.float64, device=f"cuda:{gpu}")
        assert s.lib.p2p_pass_begin_device(s.h, huge, d.data_ptr(), None, 4, d.data_ptr(),
                                           d.data_ptr()) == abi.P2P_ERR_NOMEM
        n3 = 3 * tl.npart
        out = np.full(n3 + 4096, 7.0)
        s.lib.p2p_pass_result(s.h, out.ctypes.data_as(ctypes.c_void_p))
        assert np.all(out[n3:] == 7.0)
        s.lib.p2p_pass_accumulate(s.h, out.ctypes.data_as(ctypes.c_void_p))
        assert np.all(out[n3:] == 7.0)
        got, _ = s.force_pass(tl.pos, tl.leaf_ipart, tl.leaf_npart, tl.task_t, tl.task_s)
    assert np.array_equal(got, want)
