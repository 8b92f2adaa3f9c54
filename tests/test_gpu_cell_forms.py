"""The two forms of the FP64 integrator's cell x phase sums, chosen per call by
the room left for the run records: the power sums over runs of cells (the form
that runs) and the cell by cell form give the same fluxes to 1e-12 of each
energy row's largest value on the small Num4D and blackbody batches, the latter
with an omitted crescent and polar caps among the members, and on one with a
blackbody elsewhere (every value is added)."""
import numpy as np
import pytest

import batch_cases
from conftest import row_rel
from integrate_call import integrate_scratch
from xpsi_gb300 import batch as BT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("builder", ["small_num4d", "small_blackbody", "small_elsewhere"])
def test_power_sums_equal_cell_sums(builder):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    m, params = getattr(batch_cases, builder)()
    ev = BT.BatchEvaluator(m)
    B = ev.upload(BT.prepare(m, params))
    ev.run(B, likelihood=False)
    torch.cuda.synchronize()
    runs, st_r, s, _ = integrate_scratch(ev, B)
    cells, st_c, q, _ = integrate_scratch(ev, B, limit_bytes=1)
    assert (s.run_sums, q.run_sums) == (1, 0)
    np.testing.assert_array_equal(st_r, st_c)
    assert np.abs(cells).max() > 0
    # two orders of summation: not the same program twice
    assert not np.array_equal(runs, cells)
    for i in range(len(runs)):
        assert row_rel(runs[i], cells[i]) <= 1e-12, i
