"""A parallel whose ray table failed (no largest deflection, or one below zero)
in a batch: it has no images, so its member's flux is that of the mesh without
the parallel (1e-12 of each energy row's largest value: the order of the sums
may differ), and every other member keeps its bits."""
import numpy as np
import pytest

from conftest import row_rel
from integrate_call import integrate
from xpsi_gb300 import batch as BT
from xpsi_gb300 import synthetic as SY

pytestmark = pytest.mark.gpu


def integrated(torch, precision):
    """A batch of six vectors of two Num4D regions after its integration, and
    the lit parallel of most images of the third vector's first region."""
    m = SY.config2_model(K=20, q=16, num_energies=20, sqrt_num_cells=14, num_leaves=24,
                         num_rays=64, max_sqrt_num_cells=24, table_shape=(10, 8, 16, 60))
    rng = np.random.default_rng(5)
    p = np.array([SY.prior_vector(rng) for _ in range(6)])
    ev = BT.BatchEvaluator(m, precision=precision)
    P = BT.prepare(m, p)
    B = ev.upload(P)
    ev.run(B, likelihood=False)
    torch.cuda.synchronize()
    member = 4
    M = P.meshes[member]
    lit = B["radiates"].cpu().numpy()[M.cell_off:M.cell_off + M.S0 * M.S1].reshape(M.S0, M.S1)
    return ev, P, B, member, int(np.argmax(lit.sum(axis=1)))


@pytest.mark.parametrize("precision", ["plain", "mixed"])
@pytest.mark.parametrize("largest", [float("nan"), -7.0, -1e300])
def test_row_without_images(precision, largest):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ev, P, B, member, row = integrated(torch, precision)
    whole, st_whole = integrate(ev, B)
    B["maxDefl"][P.meshes[member].row_off + row] = largest
    failed, st_failed = integrate(ev, B)
    M = P.meshes[member]
    c0 = M.cell_off + row * M.S1
    B["radiates"][c0:c0 + M.S1] = 0
    dark, st_dark = integrate(ev, B)
    np.testing.assert_array_equal(st_failed, st_whole)
    np.testing.assert_array_equal(st_dark, st_whole)
    assert st_whole[member] == 0
    assert row_rel(failed[member], dark[member]) <= 1e-12
    assert row_rel(failed[member], whole[member]) > 1e-6
    others = [i for i in range(len(whole)) if i != member]
    np.testing.assert_array_equal(failed[others], whole[others])


@pytest.mark.parametrize("precision", ["plain", "mixed"])
def test_row_of_infinite_deflection(precision):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ev, P, B, member, row = integrated(torch, precision)
    whole, st_whole = integrate(ev, B)
    B["maxDefl"][P.meshes[member].row_off + row] = float("inf")
    failed, st_failed = integrate(ev, B)
    others = [i for i in range(len(whole)) if i != member]
    np.testing.assert_array_equal(failed[others], whole[others])
    np.testing.assert_array_equal(st_failed[others], st_whole[others])
