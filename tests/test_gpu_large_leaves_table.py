"""The FP64 integrator's leaf counts at the full-size table (67 mu, 166
energies), where its shared memory is tightest, with 1024 rays: below, at and
above the last count of the form with runs, and the largest.  Against the
mixed-precision form, whose shared memory is laid out otherwise, to 1e-4 of each
energy row's largest value (FP32 sums and splines: a misplaced or overlapping
array is wrong in the first digit), and the form with runs against the per-cell
form to 1e-12."""
import numpy as np
import pytest

from conftest import row_rel
from integrate_call import integrate_scratch
from xpsi_gb300 import batch as BT
from xpsi_gb300 import synthetic as SY

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaves,runs", [(400, 1), (469, 1), (472, 0), (490, 0), (514, 0)])
def test_many_leaves(leaves, runs):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    m = SY.config2_model(K=20, q=16, num_energies=9, sqrt_num_cells=14, num_leaves=leaves,
                         num_rays=1024, max_sqrt_num_cells=128, table_shape=(6, 5, 67, 166))
    p = np.array([SY.prior_vector(np.random.default_rng(4))])
    flux = {}
    for precision in ("plain", "mixed"):
        ev = BT.BatchEvaluator(m, precision=precision)
        B = ev.upload(BT.prepare(m, p))
        ev.run(B, likelihood=False)
        torch.cuda.synchronize()
        flux[precision], st, s, _ = integrate_scratch(ev, B)
        assert (st == 0).all() and s.run_sums == (runs if precision == "plain" else 0)
        if precision == "plain":
            cells = integrate_scratch(ev, B, limit_bytes=1)[0]
    assert np.abs(flux["plain"]).max() > 0
    for i in range(len(cells)):
        assert row_rel(flux["plain"][i], cells[i]) <= 1e-12
        assert row_rel(flux["mixed"][i], flux["plain"][i]) <= 1e-4
