"""H psi through the stream passes at every compiled grid size, with each tile width and
factorization of its line transforms, against the oracle: 2D grids up to 512 (with the
logarithmic kernel up to 384, whose padded lines are 768), 3D grids with the Newton
kernel. Tolerance 1e-12 relative (max-norm), the single-apply bar."""
import numpy as np
import pytest
import torch

from becgpp_b200 import HamiltonianBatch, _lib, default_cfg, make_grid
from becgpp_b200.grid import plan_for
from becgpp_b200.interactions import kernel_convolution
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


@pytest.mark.parametrize("dim,N", [("2D", 16), ("2D", 96), ("3D", 24)])
def test_convolution_of_fields_on_8_byte_boundaries(dim, N):
    """Densities and outputs that start on 8 but not 16 bytes (contiguous slices of larger
    arrays): the same bits as aligned ones."""
    kern = "newton" if dim == "3D" else "log"
    G = make_grid(default_cfg(mode="single", dimension=dim, kernel=kern, Ngrid=N, L=7.0, G_C=6.0))
    shape = (N,) * (3 if dim == "3D" else 2)
    n = N ** len(shape)
    rho = torch.rand(n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(N))
    want = kernel_convolution(rho.view(shape), G)
    big = torch.zeros(n + 1, dtype=torch.float64, device="cuda")
    big[1:] = rho
    odd = big[1:].view(shape)
    assert odd.data_ptr() % 16 == 8
    assert torch.equal(kernel_convolution(odd, G), want)
    plan = plan_for(G, dict(beta2=0.0, beta3=0.0, Omega=0.0, G_C=1.0))
    out = torch.zeros(n + 2, dtype=torch.float64, device="cuda")
    _lib.check(_lib.lib().bgp_convolve(plan.handle, 0, _lib.ptr(odd), _lib.ptr(out[1:]), 0, _lib.stream_ptr()),
               "bgp_convolve")
    assert torch.equal(out[1:-1].view(shape), want)
    assert out[0] == 0.0 and out[-1] == 0.0


def test_batched_outputs_are_tensors_of_their_own():
    """Writing one output of a batched apply in place leaves the others' autograd state alone."""
    cfgs = [default_cfg(mode="single", dimension="2D", kernel="none", Ngrid=16, L=7.0, beta2=b) for b in (1.0, 2.0, 3.0)]
    grids = [make_grid(c) for c in cfgs]
    psi = torch.randn(16, 16, dtype=torch.complex128, device="cuda")
    hb = HamiltonianBatch(cfgs, grids)
    outs = hb.apply([psi] * 3)
    before = [o.clone() for o in outs]
    w = torch.full((), 2.0, dtype=torch.float64, device="cuda", requires_grad=True)
    outs[0].mul_(w)
    assert outs[0].requires_grad and not outs[1].requires_grad and outs[1]._version == 0
    assert torch.equal(outs[0], 2.0 * before[0])
    assert torch.equal(outs[1], before[1]) and torch.equal(outs[2], before[2])
    hb.close()
