"""Two steps of the device's Thomas-Fermi fixed point against a numpy restatement
(becgpp/thomasfermi.py:33-62, 83-115), over the sizes where the team that takes a step
changes: one point per thread in a few CTAs, full clusters, the last size of each rule
(with and without the square root of b3 > 0) and grid-wide launches; b2 < 0 too.

The potential is the device's own convolution. Differences come from the order of sums of
up to 1.5e5 positive terms (a few 1e-14 relative), amplified by the second step's
convolution and normalisations by less than 10: tolerance 1e-12 of the largest density."""
import numpy as np
import pytest
import torch

from becgpp_b200 import default_cfg, make_grid
from becgpp_b200.interactions import long_range_phi
from becgpp_b200.thomasfermi import _device_density

pytestmark = pytest.mark.gpu


def _rho(mu, base, b2, b3):
    rhs = mu - base
    if b3 > 1e-30:
        disc = b2 * b2 + 4.0 * b3 * rhs
        return np.where(disc > 0.0, np.maximum((np.sqrt(np.maximum(disc, 0.0)) - b2) / (2.0 * b3), 0.0), 0.0)
    return np.maximum(rhs / b2, 0.0)


def _step(n, base, b2, b3, dv, relax):
    lo, hi = base.min(), base.max() + abs(b2) + abs(b3) + 1.0
    while _rho(hi, base, b2, b3).sum() * dv < 1.0:
        hi = lo + 2.0 * (hi - lo) + 1e-9
    for _ in range(90):
        mid = 0.5 * (lo + hi)
        if _rho(mid, base, b2, b3).sum() * dv < 1.0:
            lo = mid
        else:
            hi = mid
    mu = 0.5 * (lo + hi)
    new = _rho(mu, base, b2, b3)
    new = new / (new.sum() * dv)
    out = (1.0 - relax) * n + relax * new
    return out / (out.sum() * dv), mu


CASES = [("2D", N, 40.0, b3) for N in (16, 24, 48, 128, 192, 256, 384) for b3 in (0.0, 20.0)] + [
    ("3D", 16, 40.0, 0.0), ("3D", 32, 40.0, 20.0), ("3D", 48, 40.0, 0.0), ("2D", 64, -30.0, 60.0), ("2D", 192, -30.0, 60.0)]


@pytest.mark.parametrize("dim,N,b2,b3", CASES)
def test_two_steps(dim, N, b2, b3):
    kern = "newton" if dim == "3D" else "log"
    cfg = default_cfg(mode="single", dimension=dim, kernel=kern, Ngrid=N, L=9.0, beta2=b2, beta3=b3, G_C=3.0, Omega=0.3)
    G = make_grid(cfg)
    relax, dv = 0.4, G["dx"] ** G["ndim"]
    x = (np.arange(N) - N // 2) * G["dx"]
    c = np.meshgrid(*([x] * G["ndim"]), indexing="ij")
    r2 = sum(a * a for a in c)
    veff = 0.5 * r2 - 0.5 * 0.3 ** 2 * (c[0] ** 2 + c[1] ** 2)
    n = np.exp(-r2 / (2.0 * (0.15 * 9.0) ** 2))
    n = n / (n.sum() * dv)
    for _ in range(2):
        phi = long_range_phi(torch.as_tensor(n).cuda(), G, 3.0).cpu().numpy()
        n, mu = _step(n, veff + phi, b2, b3, dv, relax)
    got = _device_density(cfg, G, True, 2, relax)
    err = np.max(np.abs(got["n"].cpu().numpy() - n)) / n.max()
    assert err <= 1e-12, err
    assert abs(got["mu"] - mu) <= 1e-12 * max(1.0, abs(mu), np.abs(veff + phi).max())
