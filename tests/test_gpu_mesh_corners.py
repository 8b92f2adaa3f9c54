"""GPU-built meshes against the host builder's, cell by cell to 1e-10 of the
mesh's largest cell: full-size two-spot vectors whose omitted region touches
cells at a corner only (their integrals are cut into dyadic pieces, integrated
side by side on the GPU and in turn on the host), in batches below and above
the size from which the area tables take a thread per entry instead of a warp."""
import numpy as np
import pytest

from xpsi_gb300 import batch as BT
from xpsi_gb300 import synthetic as SY

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [1, 4, 6])
def test_corner_cells(V):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    m = SY.config2_model(K=20, q=16, num_energies=16, num_leaves=16, num_rays=16,
                         table_shape=(10, 8, 16, 60))
    centre = SY.config2_vector(1)
    p = []
    for seed in range(3, 3 + V):
        rng = np.random.default_rng([seed, 77])
        p.append(centre * (1.0 + 0.002 * rng.uniform(-1, 1, centre.size)))
    p = np.array(p)
    ev = BT.BatchEvaluator(m)
    host = BT.prepare(m, p, meshes="host")
    B = ev.upload(BT.prepare(m, p, meshes="gpu"))
    torch.cuda.synchronize()
    area, rad = B["cellArea"].cpu().numpy(), B["radiates"].cpu().numpy()
    corner = 0
    for i in range(len(host.meshes)):
        q = host.meshes[i]
        c = slice(q.cell_off, q.cell_off + q.S0 * q.S1)
        big = host.cellArea[c].max()
        assert np.max(np.abs(area[c] - host.cellArea[c])) <= 1e-10 * big, i
        np.testing.assert_array_equal(rad[c], host.radiates[c])
        corner += np.sum((host.cellArea[c] > 0) & (host.cellArea[c] < 1e-5 * big))
    assert corner >= 2
