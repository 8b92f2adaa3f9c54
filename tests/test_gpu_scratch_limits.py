"""The integrator where its scratch is bounded: without geometry records (every
image formed again inside the integrator) and without the run records too (the
per-cell form), for one vector, whose parallels' energies are shared by several
CTAs, and for a batch; the fluxes to 1e-12 of each energy row's largest value
(the mixed form's, whose geometry is FP64 as well, likewise), the statuses
equal.  A failed parallel takes no records from the others.  The scratch is what
the library and the serving loop's estimate say."""
import numpy as np
import pytest

from conftest import row_rel
from integrate_call import integrate_scratch
from xpsi_gb300 import batch as BT
from xpsi_gb300 import synthetic as SY
from xpsi_gb300._native import lib
from xpsi_gb300.serving import estimate_bytes

pytestmark = pytest.mark.gpu


def uploaded(torch, V, precision="plain", meshes="host"):
    m = SY.config2_model(K=20, q=16, num_energies=41, sqrt_num_cells=24, num_leaves=33,
                         num_rays=64, max_sqrt_num_cells=48, table_shape=(10, 8, 16, 60))
    rng = np.random.default_rng(V)
    p = np.array([SY.prior_vector(rng) for _ in range(V)])
    ev = BT.BatchEvaluator(m, precision=precision)
    P = BT.prepare(m, p, meshes=meshes)
    B = ev.upload(P)
    ev.run(B)
    torch.cuda.synchronize()
    return ev, P, B


@pytest.fixture(scope="module")
def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def total(ev, P):
    cells = max(q.S1 for q in P.meshes)
    return lib().xgpu_integrate_scratch_bytes(
        P.V * P.H, P.n_rows, cells, len(ev.model.energies), ev.N_L, ev.N_L, ev.atmos.nmu,
        ev.atmos.nE, int(ev.precision == "mixed"), 0, ev.sms)


@pytest.mark.parametrize("precision", ["plain", "mixed"])
@pytest.mark.parametrize("V", [1, 40])
def test_bounded_scratch(cuda, V, precision):
    ev, P, B = uploaded(cuda, V, precision)
    runs = int(precision == "plain")
    flux, st, s, again = integrate_scratch(ev, B)
    assert s.used_bytes == total(ev, P) and s.record_room == 2 * P.n_rows + 1024
    assert s.run_sums == runs and again == 0
    assert (st == 0).any() and np.abs(flux).max() > 0
    last = s.used_bytes
    for limit, r in ((s.used_bytes - 1, runs), (1, 0)):
        f, t, q, again = integrate_scratch(ev, B, limit)
        assert q.record_room == 0 and q.run_sums == r and q.used_bytes <= last
        assert (q.used_bytes < last) == (limit > 1 or runs == 1)
        last = q.used_bytes
        # every parallel with an image
        lit = B["radiates"].cpu().numpy()
        rows = sum(int((lit[M.cell_off:M.cell_off + M.S0 * M.S1].reshape(M.S0, M.S1) == 1)
                       .any(axis=1).sum()) for M in P.meshes)
        assert 0 < again <= rows
        np.testing.assert_array_equal(t, st)
        for i in np.nonzero(st == 0)[0]:
            assert row_rel(f[i], flux[i]) <= 1e-12, (limit, i)


@pytest.mark.parametrize("largest", [float("nan"), float("inf"), -7.0])
def test_failed_row_leaves_the_records(cuda, largest):
    ev, P, B = uploaded(cuda, 6)
    M = P.meshes[0]
    lit = B["radiates"].cpu().numpy()[M.cell_off:M.cell_off + M.S0 * M.S1].reshape(M.S0, M.S1)
    B["maxDefl"][M.row_off + int(np.argmax(lit.sum(axis=1)))] = largest
    again = integrate_scratch(ev, B)[3]
    # (the parallel of infinite deflection forms its own images again)
    assert again <= (1 if largest == float("inf") else 0)


@pytest.mark.parametrize("precision", ["plain", "mixed"])
def test_estimate_covers_the_launch(cuda, precision):
    ev, P, B = uploaded(cuda, 12, precision, meshes="gpu")
    s = integrate_scratch(ev, B)[2]
    tensors = [t for t in list(B.values()) + list(B["row"].values()) if hasattr(t, "data_ptr")]
    held = sum({t.data_ptr(): t.nbytes for t in tensors}.values())  # (one is held twice)
    assert held + s.used_bytes <= estimate_bytes(ev, P) <= 1.1 * (held + s.used_bytes) + 2 ** 20
