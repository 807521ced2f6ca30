"""Trees walked by sink leaf: chains of splits over particles at one point, whose
depth or waiting leaves outgrow the walk by depth, and ordinary trees sent that way.
The rows equal the serial walk's entry for entry."""
import numpy as np
import pytest

from photons_p2p import abi, lists as L, workloads as W
from photons_p2p.p2p import DeviceWalkTree, P2PError, Session, params_for

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
