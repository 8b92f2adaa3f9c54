"""A batch with many cut cells integrates them four to a warp, a small one a
CTA each: the same bits, for circular and crescent regions from small to
large, of few and many cells."""
import numpy as np
import pytest

from xpsi_gb300 import batch as BT
from xpsi_gb300 import synthetic as SY

pytestmark = pytest.mark.gpu


def areas(torch, model, p):
    ev = BT.BatchEvaluator(model)
    B = ev.upload(BT.prepare(model, p))
    ev.run(B, likelihood=False)
    torch.cuda.synchronize()
    return B["cellArea"].cpu().numpy(), B["radiates"].cpu().numpy()


@pytest.mark.parametrize("cells,vectors", [(100, 40), (33, 120)])
def test_packed_equals_alone(cells, vectors):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    m = SY.config2_model(K=20, q=16, num_energies=5, sqrt_num_cells=cells, num_leaves=10,
                         num_rays=64, max_sqrt_num_cells=200, table_shape=(10, 8, 16, 60))
    rng = np.random.default_rng(cells)
    p = np.array([SY.prior_vector(rng) for _ in range(vectors)])
    A, R = areas(torch, m, p)
    at = 0
    for v in range(vectors):
        a, r = areas(torch, m, p[v:v + 1])
        assert np.array_equal(a, A[at:at + a.size]) and np.array_equal(r, R[at:at + r.size])
        at += a.size
    assert at == A.size
