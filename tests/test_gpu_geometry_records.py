"""The integrator's geometry records: a batch whose parallels carry more images
than the records' room (stars just outside the photon sphere, about eight
images each), where the integrator's CTAs form the images that found none
themselves, gives the fluxes of the same vectors integrated one by one, which
all find room, to 1e-12 of each energy row's largest value."""
import numpy as np
import pytest

from conftest import row_rel
from xpsi_gb300 import batch as BT
from xpsi_gb300 import synthetic as SY

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blackbody", [False, True])
def test_images_beyond_the_records(blackbody):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    V = 40
    m = SY.config2_model(K=20, q=16, num_energies=20, sqrt_num_cells=20, num_leaves=33,
                         num_rays=64, max_sqrt_num_cells=24, table_shape=(10, 8, 16, 60))
    if blackbody:
        for r in m.regions:
            r.atm_ext = 1
        m.atmosphere = None
    rng = np.random.default_rng(3)
    p = np.array([SY.prior_vector(rng) for _ in range(V)])
    p[:, 1] = (3.0 + 1e-4 * rng.uniform(1, 10, V)) * p[:, 0] * 0.5 * 2.95325024
    ev = BT.BatchEvaluator(m)
    P = BT.prepare(m, p)
    B = ev.upload(P)
    ev.run(B, likelihood=False)
    torch.cuda.synchronize()
    images = torch.ceil(B["maxDefl"] / np.pi).sum().item()
    assert images > 2 * P.n_rows + 1024
    flux, status = B["flux"].cpu().numpy(), B["mesh_status"].cpu().numpy()
    assert (status == 0).sum() > V
    for v in range(V):
        B1 = ev.upload(BT.prepare(m, p[v:v + 1]))
        ev.run(B1, likelihood=False)
        torch.cuda.synchronize()
        f1, s1 = B1["flux"].cpu().numpy(), B1["mesh_status"].cpu().numpy()
        np.testing.assert_array_equal(status[2 * v:2 * v + 2], s1)
        for h in range(2):
            if s1[h] == 0:
                assert row_rel(flux[2 * v + h], f1[h]) <= 1e-12, (v, h)
