"""The device walks when a pool of lists or rows runs out and the walk is repeated,
and when rows are counted first and written by a second walk: the same rows as the
serial walk's, the same far field as with the default sizes, whatever sizes the
session's earlier walks left behind."""
import numpy as np
import pytest

from photons_p2p import abi, lists as L, workloads as W
from photons_p2p.p2p import DeviceTree, DeviceWalkTree, FarField, P2PError, Session, params_for

pytestmark = pytest.mark.gpu


def particles(name):
    if name == "c1":
        cfg, pos = W.c1_config(), W.c1_positions()
    else:
        cfg, pos = W.scaled(W.c2_config(), n_side=48, mesh=48, eps=1 / (40 * 48)), W.c2_positions(48)
    return (cfg, *W.with_ghosts(pos, cfg))


# (chunks of lists, chunks of rows or tasks, bytes of rows kept)
LIMITS = [(16, 16, 0), (0, 0, 1), (16, 0, 1), (0, 16, 100000), (0, 0, 0)]


@pytest.mark.parametrize("name", ["c1", "clustered"])
def test_rows_do_not_depend_on_the_pools(gpu, name):
    cfg, allpos, tag = particles(name)
    with L.Tree(allpos, tag, cfg.maxleaf, cfg.box) as tree:
        tt, ts = tree.walk(cfg.cutoff_radius, cfg.open_angle)
        off = np.concatenate([[0], np.cumsum(np.bincount(tt, minlength=tree.nleaf))])
        src = ts[np.argsort(tt, kind="stable")]
        dev = DeviceWalkTree(tree, f"cuda:{gpu}")

        def check(s):
            s.begin(tree.pos, tree.leaf_ipart, tree.leaf_npart)
            assert s.submit_walk(dev, cfg.cutoff_radius, cfg.open_angle) == len(tt)
            s.end()
            got = s.rows()
            assert np.array_equal(got[0], off) and np.array_equal(got[1], src)
            return s.pair_count(), s.evaluated_pairs()

        counts = set()
        for limits in LIMITS:  # a session of its own: no buffers from before
            with Session(gpu, params_for(cfg, abi.FORM_SPLIT, 1.0)) as s:
                s.walk_limits(*limits)
                counts.add(check(s))
        with Session(gpu, params_for(cfg, abi.FORM_SPLIT, 1.0)) as s:  # and one for all
            for limits in LIMITS + LIMITS[::-1]:
                s.walk_limits(*limits)
                counts.add(check(s))
    assert len(counts) == 1


def test_a_size_that_cannot_be_allocated_is_forgotten(gpu):
    cfg, allpos, tag = particles("c1")
    with L.Tree(allpos, tag, cfg.maxleaf, cfg.box) as tree:
        dev = DeviceWalkTree(tree, f"cuda:{gpu}")
        with Session(gpu, params_for(cfg, abi.FORM_SPLIT, 1.0)) as s:
            s.walk_limits(list_chunks=2**31 - 1)  # 558 GB
            s.begin(tree.pos, tree.leaf_ipart, tree.leaf_npart)
            with pytest.raises(P2PError) as e:
                s.submit_walk(dev, cfg.cutoff_radius, cfg.open_angle)
            assert e.value.status == abi.P2P_ERR_NOMEM
            s.end()
            s.walk_limits()
            _, _, ntask = s.force_pass_walk(tree, dev, cfg.cutoff_radius, cfg.open_angle)
            assert ntask == len(tree.walk(cfg.cutoff_radius, cfg.open_angle)[0])


def test_far_field_does_not_depend_on_the_pools(gpu):
    import torch

    cfg, allpos, tag = particles("clustered")
    d_pos = torch.from_numpy(np.ascontiguousarray(allpos)).to(f"cuda:{gpu}")
    torch.cuda.synchronize()
    out = []
    for limits in [(0, 0), (16, 16), (16, 0), (0, 16)]:
        with Session(gpu) as s, DeviceTree(s, d_pos, None, cfg.maxleaf, cfg.box) as t:
            s.walk_limits(*limits)
            with FarField(s) as ff:
                p, _, ip, npt = t.device_arrays()
                for _ in range(2):
                    acc = torch.empty((3, t.npart), dtype=torch.float64, device=d_pos.device)
                    ff.far(t.struct, p, ip, npt, t.npart, 1.0 / t.npart, cfg.split_radius, cfg.cutoff_radius, 0.4, 1e-15,
                           acc.data_ptr())
                    st = ff.stats()
                    out.append((acc.cpu().numpy(), st["n_m2l"], st["n_applied"], st["levels"]))
    assert out[0][1] > 0 and np.abs(out[0][0]).max() > 0
    for o in out[1:]:
        assert o[1:] == out[0][1:] and np.array_equal(o[0], out[0][0])


def test_a_small_trees_walk_takes_little_memory(gpu):
    """500 leaves: the pools take some 8 MB for the lists and 5 for the rows, where
    pools for a GPU full of warps took 74."""
    import torch

    g = np.random.default_rng(1)
    with L.Tree(g.random((3, 4500)), np.ones(4500, np.int32), 16, 1.0) as tree:
        assert 300 < tree.nleaf < 700
        dev = DeviceWalkTree(tree, f"cuda:{gpu}")
        used = []
        for _ in range(2):  # (the first loads the kernels)
            with Session(gpu, params_for(W.c1_config(), abi.FORM_SPLIT, 1.0)) as s:
                s.begin(tree.pos, tree.leaf_ipart, tree.leaf_npart)
                before = torch.cuda.mem_get_info(gpu)[0]
                s.submit_walk(dev, 0.1, 0.0)
                used.append(before - torch.cuda.mem_get_info(gpu)[0])
                s.end()
    assert used[1] < 40e6
