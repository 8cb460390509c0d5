"""The local Thomas-Fermi density has unit mass also where the three-body term is a small
correction, beta3 << beta2^2, and the roots carry the rounding of a cancelling square root:
the mass that normalises the density is the sum of the same roots, rounded the same way.

Tolerance: sums of up to 1.5e5 positive values in two orders, each within a few tens of eps:
1e-13. A mass of roots rounded otherwise is off by 4e-11 and 5e-10 in the first two cases."""
import pytest

from becgpp_b200 import default_cfg, make_grid
from becgpp_b200.thomasfermi import _device_density

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,b2,b3", [(128, 100.0, 1e-4), (128, 1e4, 1e-2), (384, 100.0, 1e-4), (64, 300.0, 1e-3)])
def test_unit_mass(N, b2, b3):
    cfg = default_cfg(mode="single", dimension="2D", Ngrid=N, L=12.0, beta2=b2, beta3=b3)
    G = make_grid(cfg)
    n = _device_density(cfg, G, False, 1, 0.3)["n"]
    assert abs(float(n.sum()) * G["dx"] ** 2 - 1.0) < 1e-13
