"""Batches built on the GPU with enough cut cells for the packed kernel (four
cells to a warp, from 5000 on): the same bits as each vector's meshes built
alone, whose cells take a CTA each, and the host builder's areas to 1e-10 of
the mesh's largest cell."""
import numpy as np
import pytest

from xpsi_gb300 import batch as BT
from xpsi_gb300 import synthetic as SY

pytestmark = pytest.mark.gpu


def built(torch, ev, model, p):
    B = ev.upload(BT.prepare(model, p, meshes="gpu"))
    torch.cuda.synchronize()
    return B["cellArea"].cpu().numpy(), B["radiates"].cpu().numpy()


@pytest.mark.parametrize("cells,vectors", [(96, 30), (33, 90)])
def test_packed_equals_alone_and_host(cells, vectors):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    m = SY.config2_model(K=20, q=16, num_energies=5, sqrt_num_cells=cells, num_leaves=10,
                         num_rays=16, max_sqrt_num_cells=200, table_shape=(10, 8, 16, 60))
    rng = np.random.default_rng(cells)
    p = np.array([SY.prior_vector(rng) for _ in range(vectors)])
    ev = BT.BatchEvaluator(m)
    A, R = built(torch, ev, m, p)
    host = BT.prepare(m, p, meshes="host")
    # cells cut by a boundary: an area between none and the mesh's whole cells'
    cut = 0
    for i in range(len(host.meshes)):
        q = host.meshes[i]
        c = slice(q.cell_off, q.cell_off + q.S0 * q.S1)
        big = host.cellArea[c].max()
        cut += np.sum((host.cellArea[c] > 0) & (host.cellArea[c] < big * (1 - 1e-9)))
        assert np.max(np.abs(A[c] - host.cellArea[c])) <= 1e-10 * big, i
        np.testing.assert_array_equal(R[c], host.radiates[c])
    # (mirrored columns are integrated once)
    assert cut > 2 * 5000
    at = 0
    for v in range(vectors):
        a, r = built(torch, ev, m, p[v:v + 1])
        np.testing.assert_array_equal(a, A[at:at + a.size])
        np.testing.assert_array_equal(r, R[at:at + r.size])
        at += a.size
    assert at == A.size
