"""The FP64 integrator where its shared memory is nearly full: leaf counts
with the power sums over runs of cells, and beyond them the per-cell form.
Against the mixed-precision form, whose shared memory is laid out otherwise,
to 1e-4 of each energy row's largest value (FP32 sums and splines: a misplaced
or overlapping array is wrong in the first digit)."""
import numpy as np
import pytest

from conftest import row_rel
from xpsi_gb300 import batch as BT
from xpsi_gb300 import synthetic as SY

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaves", [440, 545])
def test_many_leaves(leaves):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    m = SY.config2_model(K=20, q=16, num_energies=9, sqrt_num_cells=14, num_leaves=leaves,
                         num_rays=64, max_sqrt_num_cells=128, table_shape=(10, 8, 4, 4))
    p = np.array([SY.prior_vector(np.random.default_rng(3))])
    flux = []
    for precision in ("plain", "mixed"):
        ev = BT.BatchEvaluator(m, precision=precision)
        B = ev.upload(BT.prepare(m, p))
        ev.run(B, likelihood=False)
        torch.cuda.synchronize()
        flux.append(B["flux"].cpu().numpy())
    assert np.abs(flux[0]).max() > 0
    for i in range(flux[0].shape[0]):
        assert row_rel(flux[1][i], flux[0][i]) <= 1e-4
