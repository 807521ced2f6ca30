"""PM cells of particles on the box's faces and outside it (the wrap with and
without a division) against the numpy oracle."""
import numpy as np
import pytest

from oracle import pm_oracle as O
from photons_p2p.p2p import ParticleMesh, Session

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nmesh", [4, 10, 64])
def test_cells_at_and_beyond_the_faces(gpu, nmesh):
    import torch

    g = np.random.default_rng(nmesh)
    box, h = 2.0, 2.0 / nmesh
    pos = np.concatenate([g.random((3, 500)) * box,
                          g.choice([0.0, 0.49 * h, 0.51 * h, box - 0.49 * h, box - 0.51 * h, np.nextafter(box, 0), box,
                                    box + 1.3 * h, 3.7 * box, -0.3 * h, -1.6 * box], (3, 500))], axis=1)
    with Session(gpu) as s, ParticleMesh(s, nmesh, box, 1.2 * h) as pm:
        d = torch.from_numpy(pos).to(f"cuda:{gpu}")
        acc = torch.empty_like(d)
        torch.cuda.synchronize()
        pm.forces(d, None, 1e-3, acc)
        mesh, _ = pm.download()
        torch.cuda.synchronize()
    want_mesh = O.deposit(pos, None, 1e-3, nmesh, box)
    want = O.pm_forces(pos, None, 1e-3, nmesh, box, 1.2 * h)
    # the bars of the PM's other tests: sums of up to 1000 terms, then two FFTs
    assert np.abs(mesh - want_mesh).max() <= 1e-12 * np.abs(want_mesh).max()
    assert np.abs(acc.cpu().numpy() - want).max() <= 1e-10 * np.sqrt(np.mean(want ** 2))
