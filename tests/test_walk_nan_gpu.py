"""The device list walk over a tree with a particle whose coordinate is not a
number: the boxes around it have NaN centres and widths, whose pairs the serial
walk opens, and the rows equal the serial walk's entry for entry."""
import numpy as np
import pytest

from photons_p2p import abi, lists as L, workloads as W
from photons_p2p.p2p import DeviceWalkTree, Session, params_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("angle", [0.0, 0.4])
def test_rows_equal_the_serial_walks(gpu, axis, angle):
    cfg = W.c1_config()
    allpos, tag = W.with_ghosts(W.c1_positions(), cfg)
    allpos = np.array(allpos)
    allpos[axis, np.flatnonzero(tag == 1)[777]] = np.nan
    with L.Tree(allpos, tag, cfg.maxleaf, cfg.box) as tree:
        _, _, center, width = tree.nodes()
        assert np.isnan(center).any() or np.isnan(width).any()
        tt, ts = tree.walk(cfg.cutoff_radius, angle)
        dev = DeviceWalkTree(tree, f"cuda:{gpu}")
        with Session(gpu, params_for(cfg, abi.FORM_SPLIT, 1.0)) as s:
            s.begin(tree.pos, tree.leaf_ipart, tree.leaf_npart)
            assert s.submit_walk(dev, cfg.cutoff_radius, angle) == len(tt)
            s.end()
            off, src = s.rows()
    assert np.array_equal(off, np.concatenate([[0], np.cumsum(np.bincount(tt, minlength=len(off) - 1))]))
    assert np.array_equal(src, ts[np.argsort(tt, kind="stable")])
