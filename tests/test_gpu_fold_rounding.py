"""The last bit of a double joined from a float pair: an identity response
returns inputs just below and above a power of two, which a float pair holds
exactly (2^k (1 -+ n 2^-53), 2^-52), bit for bit, in the small and the large
output tiles and for either sign."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 400])
def test_identity_returns_the_inputs(batch):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from xpsi_gb300._native import check, lib
    q, N = 33, 40
    n = np.arange(1, q + 1, dtype=np.float64)[:, None]
    k = np.linspace(-50, 50, N).astype(int)[None, :]
    below = np.ldexp(1.0 - n * 2.0 ** -53, k)
    above = np.ldexp(1.0 + n * 2.0 ** -52, k)
    X = np.empty((batch, q, N))
    for b in range(batch):
        X[b] = (below, above, -below, -above)[b % 4]
    if batch == 1:
        X[0, :, 1::2] = -X[0, :, 1::2]
    dev = torch.device("cuda", 0)
    dM, dX = torch.eye(q, dtype=torch.float64, device=dev), torch.tensor(X, device=dev)
    out = torch.full((batch, q, N), np.nan, dtype=torch.float64, device=dev)
    check(lib().xgpu_fold_batch(batch, q, q, N, dM.data_ptr(), q, dX.data_ptr(), out.data_ptr(),
                                torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), X)
