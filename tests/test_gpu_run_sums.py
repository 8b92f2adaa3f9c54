"""The FP64 integrator's power sums over runs of cells (the form that runs)
against the per-cell form (XGPU_CELL_SUMS=cells), to 1e-12 of each energy
row's largest value: leaf counts that give energy chunks of 8, 16 and 32,
odd ones among them, energy counts that leave a remainder or less than one
chunk, cells far coarser and finer than the leaves, the elsewhere correction
(negative values are added), and a star near the photon sphere (several
images per parallel)."""
import os
import subprocess
import sys

import numpy as np
import pytest

from batch_cases import small_elsewhere
from conftest import ROOT, row_rel
from xpsi_gb300 import batch as BT
from xpsi_gb300 import synthetic as SY

pytestmark = pytest.mark.gpu

# (leaves, energies, cells)
SIZES = [(7, 5, 10), (24, 33, 12), (63, 32, 40), (64, 41, 16), (65, 16, 64), (101, 17, 24),
         (128, 50, 90), (200, 9, 14)]


def run_sizes():
    """Fluxes of a Num4D model of two regions at every size, and of a
    corrected blackbody one."""
    import torch
    out = []
    for n, (leaves, energies, cells) in enumerate(SIZES):
        m = SY.config2_model(K=20, q=16, num_energies=energies, sqrt_num_cells=cells,
                             num_leaves=leaves, num_rays=64, max_sqrt_num_cells=128,
                             table_shape=(10, 8, 16, 60))
        rng = np.random.default_rng(n)
        p = np.array([SY.prior_vector(rng) for _ in range(2)])
        p[0, 1] = 3.06 * p[0, 0] * 0.5 * 2.95325024
        ev = BT.BatchEvaluator(m)
        B = ev.upload(BT.prepare(m, p))
        ev.run(B, likelihood=False)
        torch.cuda.synchronize()
        out.append(B["flux"].cpu().numpy())
    m, p = small_elsewhere()
    ev = BT.BatchEvaluator(m)
    B = ev.upload(BT.prepare(m, p))
    ev.run(B, likelihood=False)
    torch.cuda.synchronize()
    out.append(B["flux"].cpu().numpy())
    return out


def test_run_sums_equal_cell_sums(tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    assert os.environ.get("XGPU_CELL_SUMS", "runs") == "runs"
    out = str(tmp_path / "cells.npz")
    code = ("import sys; sys.path[:0] = [%r, %r]\nimport numpy as np, test_gpu_run_sums as T\n"
            "np.savez(%r, *T.run_sizes())\n" % (ROOT, os.path.join(ROOT, "tests"), out))
    subprocess.run([sys.executable, "-c", code], check=True, timeout=900,
                   env=dict(os.environ, XGPU_CELL_SUMS="cells"))
    got = run_sizes()
    ref = np.load(out)
    for n, f in enumerate(got):
        r = ref["arr_%d" % n]
        assert np.abs(r).max() > 0
        for i in range(f.shape[0]):
            assert row_rel(f[i], r[i]) <= 1e-12, (n, i)
