"""Trees walked by sink leaf: chains of splits over particles at one point, whose
depth or waiting leaves outgrow the walk by depth, and ordinary trees sent that way.
The rows equal the serial walk's entry for entry, the M2L tasks its tasks."""
import numpy as np
import pytest

from photons_p2p import abi, lists as L, workloads as W
from photons_p2p.p2p import DeviceTree, DeviceWalkTree, FarField, P2PError, Session, params_for

pytestmark = pytest.mark.gpu


def particles(side, together):
    """Uniform particles, the first `together` of them at one point (dyadic
    coordinates, whose means are exact: the split peels off one at a time)."""
    g = np.random.default_rng(side + together)
    pos = g.random((3, side**3))
    pos[:, :together] = np.array([[0.25], [0.5], [0.375]])
    return pos, np.where(g.random(side**3) < 0.9, 1, 0).astype(np.int32)


def check(s, tree, cutoff, angle):
    tt, ts = tree.walk(cutoff, angle)
    s.begin(tree.pos, tree.leaf_ipart, tree.leaf_npart)
    assert s.submit_walk(DeviceWalkTree(tree, "cuda:0"), cutoff, angle) == len(tt)
    s.end()
    off, src = s.rows()
    assert np.array_equal(off, np.concatenate([[0], np.cumsum(np.bincount(tt, minlength=tree.nleaf))]))
    assert np.array_equal(src, ts[np.argsort(tt, kind="stable")])
    return len(tt)


@pytest.mark.parametrize("together", [40, 300, 1100, 2000])
@pytest.mark.parametrize("angle", [0.0, 0.4])
def test_particles_at_one_point(gpu, together, angle):
    pos, tag = particles(20, together)
    with L.Tree(pos, tag, 16, 1.0) as tree, Session(gpu, params_for(W.c1_config(), abi.FORM_SPLIT, 1.0)) as s:
        assert check(s, tree, 0.1, angle) > together**2 / 2
        assert check(s, tree, 0.0, angle) > 0


def test_the_deepest_trees(gpu):
    """About the deepest chain that the tree build makes is walked; one so long that a
    leaf's walk would take minutes is refused, and the session goes on."""
    with Session(gpu, params_for(W.c1_config(), abi.FORM_SPLIT, 1.0)) as s:
        pos, tag = particles(20, 6000)
        with L.Tree(pos, tag, 16, 1.0) as tree:
            assert check(s, tree, 0.05, 0.0) > 6000**2 / 2
        pos, tag = particles(25, 15000)
        with L.Tree(pos, tag, 16, 1.0) as tree:
            s.begin(tree.pos, tree.leaf_ipart, tree.leaf_npart)
            with pytest.raises(P2PError) as e:
                s.submit_walk(DeviceWalkTree(tree, f"cuda:{gpu}"), 0.05, 0.0)
            assert e.value.status == abi.P2P_ERR_CAPACITY
            assert s.lib.p2p_pass_end(s.h, None) == abi.P2P_ERR_CAPACITY
        pos, tag = particles(12, 0)
        with L.Tree(pos, tag, 16, 1.0) as tree:
            check(s, tree, 0.1, 0.0)


@pytest.mark.parametrize("name", ["c1", "clustered", "two_leaves"])
@pytest.mark.parametrize("depths", [1, 3, 96])
def test_depth_limit_changes_no_row(gpu, name, depths):
    if name == "c1":
        cfg, pos = W.c1_config(), W.c1_positions()
    else:
        cfg, pos = W.scaled(W.c2_config(), n_side=32, mesh=32, eps=1 / (40 * 32)), W.c2_positions(32)
    pos, tag = W.with_ghosts(pos, cfg)
    if name == "two_leaves":
        pos, tag = np.ascontiguousarray(pos[:, :20]), np.ones(20, np.int32)
    with L.Tree(pos, tag, cfg.maxleaf, cfg.box) as tree, Session(gpu, params_for(cfg, abi.FORM_SPLIT, 1.0)) as s:
        s.walk_limits(depths=depths)
        check(s, tree, cfg.cutoff_radius, 0.0)
        check(s, tree, cfg.cutoff_radius, 0.4)


def test_a_tree_whose_boxes_have_two_parents_is_refused(gpu):
    """Child codes that would make the walk by sink leaf endless or repeat boxes."""
    pos, tag = particles(12, 0)
    with L.Tree(pos, tag, 16, 1.0) as tree, Session(gpu, params_for(W.c1_config(), abi.FORM_SPLIT, 1.0)) as s:
        s.walk_limits(depths=1)
        son, first, center, width = tree.nodes()
        node = next(k for k in range(5, len(son)) if (son[k] & 1).all())
        for code in (1, 2 * node + 1, int(son[node, 0])):  # the root, itself, a sibling twice
            bad = son.copy()
            bad[node, 1] = code
            dev = DeviceWalkTree(tree, f"cuda:{gpu}")
            dev._t[0].copy_(dev._t[0].new_tensor(bad))
            s.begin(tree.pos, tree.leaf_ipart, tree.leaf_npart)
            with pytest.raises(P2PError) as e:
                s.submit_walk(dev, 0.1, 0.0)
            assert e.value.status == abi.P2P_ERR_ARG
            assert s.lib.p2p_pass_end(s.h, None) == abi.P2P_ERR_ARG
        check(s, tree, 0.1, 0.0)


def m2l_tasks(tree, cutoff, angle):
    """The M2L walk (src/fmm.c:812-957, acceptance :409-479) on the host, a front of
    pairs at a time: the tasks' number and the deepest sink box's depth."""
    son, _, nc, nw = tree.nodes()
    center, width = (np.zeros((2 * max(len(son), tree.nleaf) + 2, 3)) for _ in range(2))
    for a, leaf, node in ((center, tree.leaf_center, nc), (width, tree.leaf_width, nw)):
        a[0:2 * tree.nleaf:2], a[1:2 * len(son) + 1:2] = leaf, node
    size = (width[:, 0] + width[:, 1]) + width[:, 2]
    front, ntask = np.array([[1, 1]]), 0
    while len(front):
        A, B = front.T
        same = A == B
        d, w = center[A] - center[B], (width[A] + width[B]) * 0.5
        gap = np.abs(d) - w
        gap[gap <= 0] = 0
        near = (gap[:, 0] + gap[:, 1]) + gap[:, 2] < 1e-15
        drop = ~near & ((gap[:, 0]**2 + gap[:, 1]**2) + gap[:, 2]**2 > cutoff * cutoff)
        dist2 = (d[:, 0]**2 + d[:, 1]**2) + d[:, 2]**2
        task = ~near & ~drop & ((2 * w.max(1))**2 < angle * angle * dist2)
        leaves = (A % 2 == 0) & (B % 2 == 0)
        ntask += int((task & ~same & ~leaves).sum())
        go = (same & (A % 2 == 1)) | (~same & ~leaves & ~task & ~drop)
        A, B, same = A[go], B[go], same[go]
        open_a = ~same & (A % 2 == 1) & ((B % 2 == 0) | (size[A] > size[B]))
        out = []
        for k in range(2):
            out += [np.stack([son[A[same] >> 1, k], son[B[same] >> 1, j]], 1) for j in range(2)]
            out.append(np.stack([son[A[open_a] >> 1, k], B[open_a]], 1))
            o = ~same & ~open_a
            out.append(np.stack([A[o], son[B[o] >> 1, k]], 1))
        front = np.concatenate(out)
    depth = np.zeros(len(son), int)
    for k in range(len(son)):  # (nodes are in pre-order)
        for c in son[k]:
            if c & 1:
                depth[c >> 1] = depth[k] + 1
    return ntask, int(depth.max()) + 2


def far(gpu, pos, cutoff, angle, limits):
    import torch

    d = torch.from_numpy(np.ascontiguousarray(pos)).to(f"cuda:{gpu}")
    torch.cuda.synchronize()
    with Session(gpu) as s, DeviceTree(s, d, None, 16, 1.0) as t:
        s.walk_limits(**limits)
        p, _, ip, npt = t.device_arrays()
        out = []
        with FarField(s) as ff:
            for _ in range(2):
                acc = torch.empty((3, t.npart), dtype=torch.float64, device=d.device)
                ff.far(t.struct, p, ip, npt, t.npart, 1.0 / t.npart, cutoff / 4.5, cutoff, angle, 1e-15, acc.data_ptr())
                out.append(acc.cpu().numpy())
            st = ff.stats()
    assert np.array_equal(out[0], out[1]) and np.isfinite(out[0]).all()
    return out[0], st["n_m2l"], st["levels"]


@pytest.mark.parametrize("together", [0, 30, 300, 1100])
def test_far_field_of_a_deep_tree(gpu, together):
    """The tasks of the walk by sink leaf are the walk's; where the tree can be walked
    by depth too, the forces agree up to the order of a box's tasks: sums of some
    hundred terms of both signs, each rounded by 2^-53."""
    pos, _ = particles(14, together)
    cutoff, angle = 0.4, 0.9
    with L.Tree(pos, np.ones(pos.shape[1], np.int32), 16, 1.0) as tree:
        want = m2l_tasks(tree, cutoff, angle)
    assert want[0] > 100
    acc, *got = far(gpu, pos, cutoff, angle, {})
    assert tuple(got) == want
    for limits in (dict(depths=1), dict(depths=1, out_chunks=16), dict(depths=96)):
        other, *got = far(gpu, pos, cutoff, angle, limits)
        assert tuple(got) == want
        rms = np.sqrt((acc**2).sum(0).mean())
        assert np.abs(other - acc).max() <= 1e-11 * rms
