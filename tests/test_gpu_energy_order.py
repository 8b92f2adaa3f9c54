"""The FP64 integrator keeps an energy stencil's nodes from one energy of a
column to the next: an energy's flux is the same bits whether its neighbours
lie a node or less away, many nodes away, or in descending order.  (The first
energy of a call alone sees the reference's clamped mu.)"""
import copy

import numpy as np
import pytest

from xpsi_gb300 import batch as BT
from xpsi_gb300 import synthetic as SY

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaves,nodes", [(33, 16), (128, 60), (200, 166)])
def test_energy_order(leaves, nodes):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    m = SY.config2_model(K=20, q=16, num_energies=64, sqrt_num_cells=20, num_leaves=leaves,
                         num_rays=64, max_sqrt_num_cells=128, table_shape=(10, 8, 16, nodes))
    p = np.array([SY.prior_vector(np.random.default_rng(leaves))])

    def flux(energies):
        q = copy.copy(m)
        q.energies = np.ascontiguousarray(energies)
        ev = BT.BatchEvaluator(q)
        B = ev.upload(BT.prepare(q, p))
        ev.run(B, likelihood=False)
        torch.cuda.synchronize()
        return B["flux"].cpu().numpy()

    full = flux(m.energies)
    assert np.isfinite(full).all() and np.abs(full).max() > 0
    assert np.array_equal(flux(m.energies[::9]), full[:, ::9])
    down = flux(m.energies[::-1])[:, ::-1]
    assert np.array_equal(down[:, 1:-1], full[:, 1:-1])
    mixed = np.concatenate([m.energies[:1], m.energies[60:20:-3], m.energies[21:50:2]])
    index = np.concatenate([[0], np.arange(60, 20, -3), np.arange(21, 50, 2)])
    assert np.array_equal(flux(mixed), full[:, index])
