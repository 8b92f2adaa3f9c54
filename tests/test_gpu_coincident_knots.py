"""Phase knots that nearly coincide: a knot interval of 1e-20, whose pieces'
coefficients leave the float range (1 / h^2 = 1e40) although no cell falls into
it, leaves the flux what the oracle gives, within the parity tolerance (1e-9 of
each energy row's largest value), at energy counts that leave the lanes of one
to four groups to a warp."""
import numpy as np
import pytest

from conftest import row_rel
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def arguments(f, num_energies):
    """config1's spot with the lag left out, so that the knots are the leaves,
    the second 1e-20 after the first; phases at which the cells of a parallel
    fall into an odd number of knot intervals, by halves."""
    leaves = f["leaves"].copy()
    leaves[1] = 1e-20
    return (1, float(f["R"]), float(f["Omega"]), float(f["r_s"]), float(f["inclination"]),
            f["cellArea"], f["radius"], f["u"], f["theta"], f["phi"], f["params"], f["radiates"],
            None, int(f["N_R"]), f["deflection"], f["cos_alpha"], np.zeros_like(f["lag"]),
            f["maxDeflection"], f["cos_gamma"], f["energies"][:num_energies], leaves,
            f["phases"] + 0.012, (), None, 1, None, 0, int(f["image_order_limit"]) or None)


@pytest.mark.parametrize("num_energies", [5, 13, 40])
def test_interval_beyond_the_float_range(golden, num_energies):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from xpsi_gb300.cellmesh import integrator_for_azimuthal_invariance as integ
    args = arguments(golden("config1"), num_energies)
    st_o, ref = O.integrate(*args)
    st, flux = integ.integrate(*args)
    assert st == st_o == 0 and np.abs(ref).max() > 0
    assert row_rel(flux, ref) <= 1e-9
