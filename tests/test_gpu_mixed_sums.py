"""The mixed-precision integrator's sums take one, two or four energies per
lane by the number of energies and of parallels: an energy's flux is the same
bits whichever it is.  Cells fewer than a batch, with dark ones among them
(the second region is cut by the first), and more than are held in shared
memory; energy counts with and without a remainder."""
import copy

import numpy as np
import pytest

from xpsi_gb300 import batch as BT
from xpsi_gb300 import synthetic as SY

pytestmark = pytest.mark.gpu


def flux(torch, model, p):
    ev = BT.BatchEvaluator(model, precision="mixed")
    B = ev.upload(BT.prepare(model, p))
    ev.run(B, likelihood=False)
    torch.cuda.synchronize()
    return B["flux"].cpu().numpy()


@pytest.mark.parametrize("leaves,cells,copies", [(24, 10, 40), (101, 50, 8), (128, 300, 2),
                                                 (200, 33, 12)])
def test_energies_alike_by_lane_count(leaves, cells, copies):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    m = SY.config2_model(K=20, q=16, num_energies=64, sqrt_num_cells=cells, num_leaves=leaves,
                         num_rays=64, max_sqrt_num_cells=400, table_shape=(10, 8, 16, 60))
    p = np.array([SY.prior_vector(np.random.default_rng(leaves))])
    many = flux(torch, m, np.repeat(p, copies, axis=0))  # four per lane
    assert np.isfinite(many).all() and np.abs(many).max() > 0
    full = flux(torch, m, p)  # few parallels: two
    assert np.array_equal(full, many[:full.shape[0]])
    for n in (7, 8, 13, 32, 41):  # one, one, two, two or four, one
        part = copy.copy(m)
        part.energies = m.energies[:n].copy()
        assert np.array_equal(flux(torch, part, p), full[:, :n])
