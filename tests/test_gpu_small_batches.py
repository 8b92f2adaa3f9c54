"""The energy integration and the response fold choose their column and tile
sizes by the number of signals: a signal alone gives the bits that it gives in
a batch large enough for the largest sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MANY = 320  # with 64 x 64 tiles and 16 columns at every size below


def ptr(t):
    return t.data_ptr()


# energies: the fewest, an odd number, and one whose columns shared memory
# limits; phases: one, a remainder of every column count, two blocks and more
@pytest.mark.parametrize("n_e", [5, 33, 700])
@pytest.mark.parametrize("n_p", [1, 17, 35])
def test_energy_alone_equals_batch(n_e, n_p):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from xpsi_gb300._native import check, lib
    rng = np.random.default_rng(n_e + n_p)
    dev = torch.device("cuda", 0)
    logE = np.sort(rng.uniform(-1.0, 1.2, n_e))
    # intervals inside a piece, over several, equal edges, and past the last energy
    edges = np.sort(np.concatenate([rng.uniform(logE[0], logE[-1], 40), [logE[0], logE[-1] + 0.1],
                                    [0.5 * (logE[0] + logE[-1])] * 2]))
    n_out = edges.size - 1
    sig = rng.uniform(0.5, 2.0, (MANY, n_e, n_p))
    d_sq = rng.uniform(1.0, 3.0, MANY)
    out = {}
    for n in (1, MANY):
        t = [torch.tensor(x, device=dev) for x in
             (sig[:n], np.arange(n, dtype=np.int64) * n_e * n_p, logE, edges, d_sq[:n],
              np.arange(n, dtype=np.int64) * n_out * n_p)]
        res = torch.full((n, n_out, n_p), np.nan, dtype=torch.float64, device=dev)
        check(lib().xgpu_energy_batch(n, n_e, n_p, edges.size, ptr(t[0]), ptr(t[1]), ptr(t[2]),
                                      ptr(t[3]), ptr(t[4]), ptr(res), ptr(t[5]), 0,
                                      torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        out[n] = res.cpu().numpy()
    assert np.isfinite(out[MANY]).all() and out[MANY].max() > 0
    assert np.array_equal(out[1][0], out[MANY][0])


@pytest.mark.parametrize("K,q,N", [(65, 16, 64), (33, 7, 31), (1, 1, 1), (200, 50, 70)])
def test_fold_alone_equals_batch(K, q, N):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from xpsi_gb300._native import check, lib
    rng = np.random.default_rng(K)
    dev = torch.device("cuda", 0)
    M = torch.tensor(rng.uniform(-1, 1, (K, q)), device=dev)
    X = torch.tensor(rng.uniform(0, 1, (MANY, q, N)), device=dev)
    out = {}
    for n in (1, MANY):
        res = torch.full((n, K, N), np.nan, dtype=torch.float64, device=dev)
        check(lib().xgpu_fold_batch(n, K, q, N, ptr(M), q, ptr(X), ptr(res),
                                    torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        out[n] = res.cpu().numpy()
    assert np.array_equal(out[1][0], out[MANY][0])
    ref = M.cpu().numpy() @ X[0].cpu().numpy()
    assert np.abs(out[1][0] - ref).max() <= 1e-12 * q
