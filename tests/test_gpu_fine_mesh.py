"""A mesh of more parallels than 48 KB of shared memory hold the edges of: the
GPU builder's cells against the host builder's, areas to 1e-10 of the largest."""
import numpy as np
import pytest

from xpsi_gb300 import batch as BT
from xpsi_gb300 import synthetic as SY

pytestmark = pytest.mark.gpu


def spot():
    w = SY.config1_workload(n_channels=20, n_inputs=8, n_energies=8)
    region = BT.HotRegionSpec(atm_ext=1, sqrt_num_cells=2300, min_sqrt_num_cells=10,
                              max_sqrt_num_cells=6000, num_leaves=8, num_rays=16)
    m = BT.Model(regions=[region], instrument=BT.Instrument(w["matrix"], w["input_edges"]),
                 data=BT.Data(counts=np.zeros((20, 32), np.int32), phase_edges=w["phase_edges"],
                              exposure=1.0), num_energies=8)
    return m, np.array([[1.4, 12.0, 300.0, 0.5, 1.0, 1.2, 0.3, 6.0, 0.1]])


def test_fine_mesh_matches_the_host():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    m, p = spot()
    host = BT.prepare(m, p, meshes="host")
    assert 2571 < host.n_rows < 5144
    B = BT.BatchEvaluator(m).upload(BT.prepare(m, p, meshes="gpu"))
    torch.cuda.synchronize()
    area = B["cellArea"].cpu().numpy()
    assert np.max(np.abs(area - host.cellArea)) <= 1e-10 * host.cellArea.max()
    np.testing.assert_array_equal(B["radiates"].cpu().numpy(), host.radiates)
