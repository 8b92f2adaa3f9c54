"""The ray integrals from a first panel of 31 points and of 61: either rule
holds every integral to 1e-12 of itself by its own error estimate, so that a
deflection, twice the integral of the whole range less that of a part of it,
agrees to 6e-12 of itself and a lag to 6e-12 of its row's largest terms (three
integrals of either rule), from weak fields to stars near the photon sphere,
where about half the rays go on to the 61 points.  Other panels are refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

R_S = 4000.0


def tables(torch, u, N_R, points):
    from xpsi_gb300._native import lib
    dev = torch.device("cuda", 0)
    n = u.size
    t = lambda a: torch.tensor(np.asarray(a, np.float64), device=dev)
    out = {k: torch.full((n, N_R), np.nan, dtype=torch.float64, device=dev)
           for k in ("defl", "ca", "lag")}
    # the largest angle of a surface that is not tilted, pi / 2, and one beyond
    ma = t(np.where(np.arange(n) % 2 == 0, np.pi / 2, np.pi / 2 + 0.3))
    du, rs, md = t(u), t(np.full(n, R_S)), t(np.zeros(n))
    st = torch.zeros(n, dtype=torch.int32, device=dev)
    p = lambda x: x.data_ptr()
    rc = lib().xgpu_rays_batch_rule(n, N_R, p(du), p(rs), p(ma), p(out["defl"]), p(out["ca"]),
                                    p(out["lag"]), p(md), p(st), None, None, points,
                                    torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return rc, {k: v.cpu().numpy() for k, v in out.items()}, st.cpu().numpy()


@pytest.fixture(scope="module")
def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("N_R", [3, 127, 128, 129, 1024])
def test_panels_agree(cuda, N_R):
    u = np.concatenate([np.linspace(0.02, 0.6, 12), np.linspace(0.61, 0.6666, 12)])
    rc31, a, st31 = tables(cuda, u, N_R, 31)
    rc61, b, st61 = tables(cuda, u, N_R, 61)
    assert rc31 == rc61 == 0
    np.testing.assert_array_equal(st31, st61)
    np.testing.assert_array_equal(a["ca"], b["ca"])
    ok = st61 == 0
    assert ok.sum() >= 20
    d = np.abs(a["defl"] - b["defl"])[ok]
    assert np.all(d <= 6e-12 * b["defl"][ok])
    scale = np.max(np.abs(b["lag"]), axis=1, keepdims=True)[ok]
    # the logarithm that follows the integrals is of the order of 10 r_s / c
    scale = np.maximum(scale, 10 * R_S / 2.99792458e8)
    e = np.abs(a["lag"] - b["lag"])[ok] / scale
    assert np.all(e <= 6e-12)
    with np.errstate(divide="ignore", invalid="ignore"):
        print("largest differences: deflection %.1e of itself, lag %.1e of its row's scale"
              % (np.nanmax(d / b["defl"][ok]), e.max()))


@pytest.mark.parametrize("points", [0, 15, 21, 30, 62, -31])
def test_other_panels_are_refused(cuda, points):
    assert tables(cuda, np.array([0.3]), 8, points)[0] != 0
