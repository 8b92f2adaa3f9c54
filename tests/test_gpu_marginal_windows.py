"""Marginal integrals whose window has no width of its own: where the star
vanishes in some bin and Newton's background ends at zero, the window is ten
times 1e90 wide.  With one count in a bin of star count rate s,

    int_0^inf (s + B) / s exp(-T B) dB = 1 / T + 1 / (s T^2)

exactly, so the channel's term is its logarithm plus log(S s) - sum_j S s_j."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# bins: fewer than a warp, its lanes, more; channels: one, more than a CTA has
@pytest.mark.parametrize("bins", [20, 32, 64])
@pytest.mark.parametrize("channels", [1, 7])
def test_one_count_and_dark_bins(bins, channels):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from xpsi_gb300.likelihoods import default_background_marginalisation as DBM
    T, n_p = 1.0e6, 129
    x = np.linspace(0.0, 1.0, n_p)
    edges = np.linspace(0.0, 1.0, bins + 1)
    # lit over an eighth of a turn in the middle; the mean of the star below
    # the one count's rate, its rate in the bin of the count above 1 / T
    lit = np.where(np.abs(x - 0.5) < 1.0 / 16.0, 1.0, 0.0)
    rate = np.linspace(3.0e-6, 5.0e-6, channels)
    comp = np.ascontiguousarray(rate[:, None] * lit[None, :])
    counts = np.zeros((channels, bins))
    counts[:, bins // 2] = 1.0
    support = np.tile([0.0, -1.0], (channels, 1))
    ll, star, background, _ = DBM.eval_marginal_likelihood(
        T, edges, counts, [comp], [x], np.zeros(1), np.zeros(channels), support, 1000, 0.0, 1e-8,
        1e-3, 10.0, -1e90)
    assert (background == 0.0).all() and (star == 0.0).any(axis=1).all()
    S = T / bins
    s = star[:, bins // 2] / S
    assert (s > 1.0 / T).all()
    terms = (np.log(1.0 / T + 1.0 / (s * T * T)) + np.log(S * s) - star.sum(axis=1))
    # quadrature to 1e-13, a double-float integrand (1e-14), sums of up to 64 bins
    assert abs(ll - math.fsum(terms)) <= 1.0e-12 * np.abs(terms).sum()
