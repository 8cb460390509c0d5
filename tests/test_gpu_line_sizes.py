"""H psi through the stream passes at every compiled grid size, with each tile width and
factorization of its line transforms, against the oracle: 2D grids up to 512 (with the
logarithmic kernel up to 384, whose padded lines are 768), 3D grids with the Newton
kernel. Tolerance 1e-12 relative (max-norm), the single-apply bar."""
import numpy as np
import pytest
import torch

from becgpp_b200 import HamiltonianBatch, default_cfg, make_grid
from oracle import gpp as O

pytestmark = pytest.mark.gpu

CASES = [("2D", n) for n in (16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512)] + [("3D", n) for n in (16, 24, 32, 48)]


@pytest.mark.parametrize("dim,N", CASES)
def test_every_tile_width_and_factorization(dim, N):
    kern = "newton" if dim == "3D" else ("log" if N <= 384 else "none")
    c = default_cfg(mode="single", dimension=dim, kernel=kern, Ngrid=N, L=7.0, Omega=0.4, beta2=30.0, beta3=5.0,
                    G_C=(0.0 if kern == "none" else 6.0))
    G = make_grid(c)
    shape = (N,) * (3 if dim == "3D" else 2)
    rng = np.random.default_rng(N)
    R2 = G["R2"].cpu().numpy()
    psi = np.exp(-0.1 * R2) * (1.0 + 0.3 * rng.standard_normal(shape) + 0.3j * rng.standard_normal(shape))
    want = O.apply_H(psi, O.make_grid(c), c)
    dev = torch.as_tensor(psi).cuda()
    hb = HamiltonianBatch([c], [G])
    for v in (0, 1):
        for ln in (2, 4, 8):
            cv = 3 if v and 2 * N % 32 == 0 else 0
            hb.set_schedule(N, ln, v, ln, cv, conv_strided_lines=max(ln, 4))
            got = hb.apply([dev])[0].cpu().numpy()
            err = np.max(np.abs(got - want)) / np.max(np.abs(want))
            assert err < 1e-12, (dim, N, ln, v, err)
    hb.close()
