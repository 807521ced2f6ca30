"""The CSR build's stable sort at the sizes where its launches change: digit
widths by key bits, one or three launches for the offsets by tiles of 4096
entries, against a stable argsort of the list by sink."""
import numpy as np
import pytest

from photons_p2p import abi
from photons_p2p.p2p import Session, make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nleaf", [1, 254, 256, 511, 1022, 1023, 1024, 70000])
@pytest.mark.parametrize("ntask", [1, 4097, 131072, 131073])
def test_rows_are_the_list_in_order(gpu, nleaf, ntask):
    g = np.random.default_rng(nleaf + ntask)
    tt = g.integers(0, nleaf, ntask).astype(np.int32)
    ts = g.integers(0, nleaf, ntask).astype(np.int32)
    npt = np.zeros(nleaf, np.int32)  # no particles: the list alone
    npt[0] = 1
    ip = np.minimum(np.arange(nleaf), 1).astype(np.int32)
    with Session(gpu, make_params(form=abi.FORM_SPLIT, soft_mode=abi.SOFT_PLUMMER, x_cut=2.25)) as s:
        s.force_pass(np.zeros((3, 1)), ip, npt, tt, ts)
        off, src = s.rows()
    assert np.array_equal(off, np.concatenate([[0], np.cumsum(np.bincount(tt, minlength=nleaf))]))
    assert np.array_equal(src, ts[np.argsort(tt, kind="stable")])
