"""NaN in a caller's ray tables, decided as the reference decides it: a NaN
phase knot does not end a parallel (its order check is a <= that a NaN passes),
a NaN deflection ends the scan for the first ray beyond pi/2, whatever the
NaN's sign."""
import numpy as np
import pytest

from conftest import row_rel
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def integrate():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from xpsi_gb300.cellmesh import integrator_for_azimuthal_invariance as integ
    return integ.integrate


def arguments(f, deflection, lag, inclination):
    return (1, float(f["R"]), float(f["Omega"]), float(f["r_s"]), inclination, f["cellArea"],
            f["radius"], f["u"], f["theta"], f["phi"], f["params"], f["radiates"], None,
            int(f["N_R"]), deflection, f["cos_alpha"], lag, f["maxDeflection"], f["cos_gamma"],
            f["energies"], f["leaves"], f["phases"], (), None, 1, None, 0,
            int(f["image_order_limit"]) or None)


@pytest.mark.parametrize("nan", [np.nan, -np.nan])
def test_nan_knot_ends_nothing(golden, integrate, nan):
    f = golden("config1")
    i = float(f["inclination"])
    clean = O.integrate(*arguments(f, f["deflection"], f["lag"], i))[1]
    lag = f["lag"].copy()
    lag[37, 250] = nan  # a table entry that the parallel's leaves see
    args = arguments(f, f["deflection"], lag, i)
    st_o, ref = O.integrate(*args)
    assert st_o == 0 and np.isfinite(ref).all() and row_rel(ref, clean) > 1e-4
    st, flux = integrate(*args)
    assert st == 0 and np.isfinite(flux).all()
    # one of 38 parallels loses some of its image
    assert row_rel(flux, clean) < 0.05


def test_nan_deflection_of_either_sign(golden, integrate):
    f = golden("config1")
    clean = integrate(*arguments(f, f["deflection"], f["lag"], 0.3))[1]
    out = []
    for nan in (np.nan, -np.nan):
        D = f["deflection"].copy()
        D[:, 3] = nan  # below every leaf's deflection
        st, flux = integrate(*arguments(f, D, f["lag"], 0.3))
        assert st == 0
        out.append(flux)
    np.testing.assert_array_equal(out[0], out[1])
    # every value from the main table, none from the table on the cosines
    assert 0.0 < row_rel(out[0], clean) < 1e-3
