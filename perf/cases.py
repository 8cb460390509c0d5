"""Performance cases: the calls a user of this package makes, over the grid sizes it compiles.

Families (the key ``what`` of a case):

* ``hpsi``      one Hamiltonian apply of a state, ``apply_H`` (2D, 3D, with and without the
                long-range potential, rotating or not): the call of a time stepper, an
                eigensolver or a residual check of the caller's own.
* ``batch``     the apply of a whole sweep of instances, ``HamiltonianBatch.apply``.
* ``phi``       the free-space potential of a density, ``long_range_phi``.
* ``evaluate``  ``energy_components`` and ``compute_residual`` of a state, the pair a run
                reports for any state it is handed.
* ``grad``      the differentiable energy, forward and backward to the state and to the
                parameters (``autodiff.energy``).
* ``tf``        the Thomas-Fermi reference density, ``extract_tf``, a fixed number of steps.
* ``solve``     ``ground_state`` from a seed, the first ``maxit`` iterations of the solver
                (FP64), with the observables of the state it returns.
* ``sweep``     ``BatchSolver.solve`` of a sweep of droplets on two grid sizes in one batch.

The solves stop after a few tens of iterations, while two correct FP64 runs still agree to
many digits: near its stop the algorithm's accept/reject decisions are decided by the last bits.
"""
import math

import numpy as np
import torch

import becgpp_b200 as B
from becgpp_b200 import autodiff

SIZES = (16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512)


# ------------------------------------------------------------------------------ the cases
def _case(what, N, dim="2D", kernel="none", name=None, **more):
    c = dict(what=what, dim=dim, N=N, kernel=kernel, L=12.0, s=2.0, l_z=0.0, beta2=100.0, beta3=0.0, Omega=0.0,
             G_C=(0.0 if kernel == "none" else 10.0), instances=1, maxit=0)
    if kernel == "q2d":
        c["l_z"] = 0.5
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: one apply on a small plane grid, where launches and the call itself count
        _case("hpsi", 64, L=10.0, name="hpsi_2d_64"),
        # a rotating condensate on an odd-radix grid (384 = 2^7 3)
        _case("hpsi", 384, Omega=0.9, beta2=200.0, name="hpsi_2d_rotating_384"),
        # the droplet sweep in one call: 64 instances, half on 128^2 and half on 256^2
        _case("batch", 128, L=20.0, beta2=-400.0, beta3=1e3, instances=64, name="hpsi_sweep_64"),
        # a self-gravitating condensate: the apply with its zero-padded potential (256^3)
        _case("hpsi", 128, "3D", "newton", L=16.0, beta2=10.0, G_C=20.0, name="hpsi_3d_newton_128"),
        # the largest grid of an apply: 16.8 M points, rotating
        _case("hpsi", 256, "3D", L=10.0, Omega=0.3, name="hpsi_3d_256"),
        # the potential alone on the largest padded box here (384^3)
        _case("phi", 192, "3D", "newton", L=12.0, G_C=20.0, name="phi_3d_newton_192"),
        # energy terms and residual of a plane state with the logarithmic kernel
        _case("evaluate", 192, kernel="log", G_C=5.0, name="evaluate_2d_log_192"),
        # forward and backward of the energy of a quasi-2D pancake, rotating
        _case("grad", 256, "quasi2D", "q2d", L=16.0, beta2=50.0, Omega=0.3, name="grad_q2d_256"),
        # the Thomas-Fermi reference of the same pancake
        _case("tf", 256, "quasi2D", "q2d", L=16.0, beta2=50.0, Omega=0.3, maxit=25, name="tf_q2d_256"),
        # the pancake's ground state, one instance in the solver
        _case("solve", 256, "quasi2D", "q2d", L=16.0, beta2=50.0, Omega=0.3, maxit=40, name="solve_q2d_256"),
        # a sweep of droplets in one batched solve
        _case("sweep", 128, L=20.0, beta2=-400.0, beta3=1e3, instances=16, maxit=30, name="solve_sweep_16"),
        # the self-gravitating condensate in the solver
        _case("solve", 128, "3D", "newton", L=16.0, beta2=10.0, G_C=20.0, maxit=12, name="solve_3d_newton_128"),
    ]


def draw(rng):
    def size(lo, hi):
        # evenly over the logarithm of the compiled sizes
        x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        return min((n for n in SIZES if lo <= n <= hi), key=lambda n: abs(math.log(n / x)))

    what = rng.choice(("hpsi", "hpsi", "hpsi", "batch", "phi", "evaluate", "evaluate", "grad", "tf", "solve", "solve",
                       "sweep"))
    c = dict(L=round(rng.uniform(8.0, 16.0), 2), beta2=round(rng.uniform(10.0, 300.0), 1),
             Omega=rng.choice((0.0, 0.0, round(rng.uniform(0.1, 0.8), 2))))
    if what in ("batch", "sweep"):
        top = rng.choice((1, 2, 4, 8, 16, 32)) if what == "batch" else rng.choice((2, 4, 8, 12))
        return _case(what, size(32, 192 if what == "batch" else 128), L=20.0, beta2=-400.0, beta3=1e3, instances=top,
                     maxit=(rng.randrange(10, 31) if what == "sweep" else 0))
    if what == "tf":
        k, dim = rng.choice((("q2d", "quasi2D"), ("log", "2D"), ("newton", "3D")))
        return _case(what, size(32, 256) if dim != "3D" else size(16, 64), dim, k, beta2=c["beta2"], Omega=0.0,
                     L=c["L"], maxit=rng.randrange(8, 26))
    dim, k = rng.choice((("2D", "none"), ("2D", "none"), ("2D", "log"), ("quasi2D", "q2d"), ("quasi2D", "newton"),
                         ("3D", "none"), ("3D", "newton")))
    if what == "phi" and k == "none":
        dim, k = rng.choice((("2D", "log"), ("quasi2D", "q2d"), ("3D", "newton")))
    if what == "grad" and k in ("log", "newton"):
        dim, k = ("quasi2D", "q2d") if dim != "3D" else (dim, k)
    if dim != "3D":
        N = size(24, 512 if k == "none" else 384)
    elif what == "solve":
        N = size(16, 96)
    else:
        N = size(16, 192 if k == "none" else 128)
    if what == "hpsi" and rng.random() < 0.25:
        c["s"] = 4.0          # quartic trap
    if rng.random() < 0.2:
        c["beta3"] = round(rng.uniform(1.0, 50.0), 1)
    if what == "solve":
        c["maxit"] = rng.randrange(6, 13) if dim == "3D" else rng.randrange(15, 41)
    return _case(what, N, dim, k, **c)


# ----------------------------------------------------------------------- inputs and the pass
def _cfg(case, **over):
    c = dict(mode="single", dimension=case["dim"], kernel=case["kernel"], Ngrid=case["N"], L=case["L"], s=case["s"],
             l_z=case["l_z"], beta2=case["beta2"], beta3=case["beta3"], Omega=case["Omega"], G_C=case["G_C"],
             res_tol=1e-8)
    if case["maxit"]:
        c["maxit"] = case["maxit"]
    c.update(over)
    return B.default_cfg(**c)


def _ndim(case):
    return 3 if case["dim"] == "3D" else 2


def _state(ndim, N, L, seed):
    """A trapped cloud with 1 % amplitude noise and 5 % phase noise, unit mass, from the seed alone."""
    g = torch.Generator(device=B.DEV).manual_seed(seed)
    dx = 2.0 * L / N
    x = (torch.arange(N, dtype=torch.float64, device=B.DEV) - N // 2) * dx
    w = (0.2 * L) ** 2
    env = torch.exp(-0.5 * x * x / w)
    env = env[:, None] * env[None, :] if ndim == 2 else env[:, None, None] * env[None, :, None] * env[None, None, :]
    amp = env * (1.0 + 1e-2 * torch.randn(env.shape, generator=g, dtype=torch.float64, device=B.DEV))
    ph = 5e-2 * torch.randn(env.shape, generator=g, dtype=torch.float64, device=B.DEV)
    psi = torch.polar(amp.abs(), ph)
    return psi / torch.sqrt((psi.abs() ** 2).sum() * dx ** ndim)


def _sweep(case, seed):
    """The instances of a droplet sweep: beta2 from its first value to -50, grids N and 2N in turn."""
    k = case["instances"]
    out = []
    for b, b2 in enumerate(np.linspace(case["beta2"], -50.0, k) if k > 1 else [case["beta2"]]):
        out.append(_cfg(case, beta2=float(b2), Ngrid=case["N"] * (1 + b % 2), seed="gaussian", rng=seed * 64 + b))
    return out


def prepare(case, seed):
    what = case["what"]
    if what in ("batch", "sweep"):
        cfgs = _sweep(case, seed)
        grids = [B.make_grid(c) for c in cfgs]
        if what == "batch":
            psis = [_state(2, c["Ngrid"], c["L"], seed * 64 + i) for i, c in enumerate(cfgs)]
            return dict(what=what, hb=B.HamiltonianBatch(cfgs, grids), psis=psis)
        return dict(what=what, bs=B.BatchSolver(cfgs, grids), psis=[B.make_seed(G, c) for G, c in zip(grids, cfgs)])
    if what == "tf":
        # the density follows from the parameters alone: another seed is another coupling
        cfg = _cfg(case, beta2=case["beta2"] * (1.0 + 0.01 * (seed % 97)), tf_cache=False)
        return dict(what=what, cfg=cfg, G=B.make_grid(cfg), iters=case["maxit"])
    cfg = _cfg(case, seed="gaussian", rng=seed)
    G = B.make_grid(cfg)
    s = dict(what=what, cfg=cfg, G=G)
    if what == "solve":
        s["psi"] = B.make_seed(G, cfg)
        return s
    psi = _state(_ndim(case), case["N"], case["L"], seed)
    if what == "phi":
        s["rho"] = (psi.real ** 2 + psi.imag ** 2).contiguous()
    else:
        s["psi"] = psi
    if what == "grad":
        s["psi"].requires_grad_(True)
        s["params"] = [torch.tensor(float(cfg[k]), dtype=torch.float64, requires_grad=True)
                       for k in ("beta2", "beta3", "G_C", "Omega")]
    return s


def run(state):
    what = state["what"]
    if what == "hpsi":
        return B.apply_H(state["psi"], state["G"], state["cfg"])
    if what == "batch":
        return state["hb"].apply(state["psis"])
    if what == "phi":
        return B.long_range_phi(state["rho"], state["G"], float(state["cfg"]["G_C"]))
    if what == "evaluate":
        c, G = state["cfg"], state["G"]
        terms = B.energy_components(state["psi"], G, c["beta2"], c["beta3"], c["Omega"], c["G_C"])
        r, mu, rel = B.compute_residual(state["psi"], G, c)
        return dict(terms, resid=r, mu=mu, resid_rel=rel)
    if what == "grad":
        psi, params = state["psi"], state["params"]
        E = autodiff.energy(psi, state["G"], *params)
        g = torch.autograd.grad(E, [psi] + params)
        return dict(E=E.detach(), psi=g[0], params=list(g[1:]))
    if what == "tf":
        tf = B.extract_tf(state["cfg"], state["G"], iters=state["iters"])
        return dict(n=tf["n"], mu=tf["mu"], R90=tf["R90"], R99=tf["R99"])
    if what == "solve":
        psi, _, obs = B.ground_state(state["cfg"], G=state["G"], psi0=state["psi"], verbose=False)
        return dict(psi=psi, E=obs["E"], mu=obs["mu"], Lz=obs["Lz"], iters=int(obs["iters"]))
    got = state["bs"].solve(state["psis"])
    return dict(psi=[g[0] for g in got], E=[g[2]["E"] for g in got], iters=[int(g[2]["iters"]) for g in got])


# ---------------------------------------------------------------------------- what a pass needs
def _fft(n):
    return 5.0 * n * math.log2(n)


def _conv_flops(ndim, N):
    """Zero-padded real convolution, only the lines that are not known to be zero (or unused)."""
    M, Mh = 2 * N, N + 1
    one = _fft(M)
    if ndim == 2:
        return 2 * N * 0.5 * one + 2 * Mh * one
    return 2 * N * N * 0.5 * one + 2 * N * Mh * one + 2 * M * Mh * one


def work(case):
    what, ndim, N = case["what"], _ndim(case), case["N"]
    n = float(N) ** ndim
    kern = case["kernel"] != "none"
    table = 8.0 * (N + 1) ** ndim if kern else 0.0
    conv = _conv_flops(ndim, N) if kern else 0.0
    h = 2 * _fft(n) + 20 * n
    if what in ("batch", "sweep"):
        tot = dict(bytes=0.0, flops=0.0)
        for b in range(case["instances"]):
            m = n * (1 if b % 2 == 0 else 4)
            it = 1 if what == "batch" else case["maxit"]
            tot["bytes"] += 32 * m
            tot["flops"] += (2 * _fft(m) + 20 * m) if what == "batch" else it * (5 * _fft(m) + 80 * m)
        return tot
    if what == "hpsi":
        return dict(bytes=32 * n + table, flops=h + conv)
    if what == "phi":
        return dict(bytes=16 * n + table, flops=conv)
    if what == "evaluate":
        # the state in and the potential out once; two potentials, one energy and one H psi
        return dict(bytes=2 * 16 * n + 8 * n + table, flops=2 * conv + _fft(n) + h + 30 * n)
    if what == "grad":
        # two tables and two convolutions (potential, and the width's derivative) for q2d
        k = 2 if case["kernel"] == "q2d" else 1
        return dict(bytes=32 * n + k * table, flops=k * conv + _fft(n) + h + 20 * n)
    if what == "tf":
        return dict(bytes=8 * n + table, flops=case["maxit"] * (conv + 90 * 6 * n))
    # a solve: per iteration one gradient, one preconditioner, one energy; with a kernel one potential
    return dict(bytes=32 * n + table, flops=case["maxit"] * (5 * _fft(n) + 80 * n + conv))


# ------------------------------------------------------------------- the same in plain torch, 64 bits
_GL = ((-0.8611363115940526, 0.3478548451374538), (-0.3399810435848563, 0.6521451548625461),
       (0.3399810435848563, 0.6521451548625461), (0.8611363115940526, 0.3478548451374538))


def _point(kind, lz, u2):
    if kind == "newton":
        return torch.rsqrt(u2)
    if kind == "log":
        return -0.5 * torch.log(u2)
    x = u2 / (4.0 * lz * lz)
    k0 = torch.special.scaled_modified_bessel_k0(x)
    if kind == "q2d":
        return k0 / (math.sqrt(2.0 * math.pi) * lz)
    return 2.0 * x * (k0 - torch.special.scaled_modified_bessel_k1(x)) / (math.sqrt(2.0 * math.pi) * lz)


def _self_cell(kind, lz, ndim, dx):
    """Mean of the kernel over the cell at the origin."""
    if ndim == 3:
        return 2.3800773640 / dx
    if kind == "newton":
        return 4.0 * math.asinh(1.0) / dx
    if kind == "log":
        return -math.log(dx) + 1.5 + 0.5 * math.log(2.0) - 0.25 * math.pi
    t, w = np.polynomial.legendre.leggauss(48)
    t, w = torch.as_tensor(t), torch.as_tensor(w)
    th, wth = math.pi / 8.0 * (t + 1.0), math.pi / 8.0 * w
    tt, wtt = 0.5 * (t + 1.0), 0.5 * w
    R = 0.5 * dx / torch.cos(th)[:, None]
    f = _point(kind, lz, (R * tt ** 2) ** 2) * 2.0 * R * R * tt ** 3 * wtt
    return 8.0 * float((wth * f.sum(1)).sum()) / (dx * dx)


def _kernel_hat(kind, lz, ndim, N, dx, dev):
    M = 2 * N
    j = torch.arange(M, dtype=torch.float64, device=dev)
    d = torch.where(j <= M // 2, j, j - M) * dx
    ker = torch.zeros((M,) * ndim, dtype=torch.float64, device=dev)
    for u, wu in _GL:
        a = (d + 0.5 * dx * u) ** 2
        for v, wv in _GL:
            b = (d + 0.5 * dx * v) ** 2
            if ndim == 2:
                ker += 0.25 * wu * wv * _point(kind, lz, a[:, None] + b[None, :])
                continue
            ab = a[:, None, None] + b[None, :, None]
            for w, ww in _GL:
                ker += (wu * wv * ww / 8.0) * _point(kind, lz, ab + ((d + 0.5 * dx * w) ** 2)[None, None, :])
    ker.view(-1)[0] = _self_cell(kind, lz, ndim, dx)
    return torch.fft.fftn(ker.to(torch.complex128))


def _convolve(rho, khat, ndim, N, dx):
    M, i0 = 2 * N, N // 2
    box = torch.zeros((M,) * ndim, dtype=torch.complex128, device=rho.device)
    sl = (slice(i0, i0 + N),) * ndim
    box[sl] = rho.to(torch.complex128)
    return torch.fft.ifftn(torch.fft.fftn(box) * khat).real[sl].contiguous() * dx ** ndim


def _operators(case, psi, N, beta2):
    """H psi, energy terms and potential of a state."""
    ndim, L = _ndim(case), case["L"]
    dx = 2.0 * L / N
    dv = dx ** ndim
    dev = psi.device
    x = (torch.arange(N, dtype=torch.float64, device=dev) - N // 2) * dx
    k = 2.0 * math.pi * torch.fft.fftfreq(N, d=dx, dtype=torch.float64).to(dev)
    axis = lambda v, a: v.reshape([-1 if b == a else 1 for b in range(ndim)])
    K2 = sum(axis(k, a) ** 2 for a in range(ndim))
    R2 = sum(axis(x, a) ** 2 for a in range(ndim))
    V = 0.5 * R2 ** (case["s"] / 2.0)
    rho = psi.real ** 2 + psi.imag ** 2
    fp = torch.fft.fftn(psi)
    kin = torch.fft.ifftn(0.5 * K2 * fp)
    lz = -1j * (axis(x, 0) * torch.fft.ifftn(1j * axis(k, 1) * fp) - axis(x, 1) * torch.fft.ifftn(1j * axis(k, 0) * fp))
    phi = torch.zeros_like(rho)
    if case["kernel"] != "none":
        phi = -case["G_C"] * _convolve(rho, _kernel_hat(case["kernel"], case["l_z"], ndim, N, dx, dev), ndim, N, dx)
    H = kin + (V + beta2 * rho + case["beta3"] * rho ** 2 + phi) * psi - case["Omega"] * lz
    s = lambda f: float(f.sum()) * dv
    t = dict(Ekin=0.5 * float((K2 * (fp.real ** 2 + fp.imag ** 2)).sum()) * dv / psi.numel(), Etrap=s(V * rho),
             Econtact=0.5 * beta2 * s(rho ** 2), Ethree=case["beta3"] / 3.0 * s(rho ** 3),
             Lz=s((psi.conj() * lz).real), Egrav=0.5 * s(phi * rho))
    t["Erot"] = -case["Omega"] * t["Lz"]
    t["E"] = t["Ekin"] + t["Etrap"] + t["Econtact"] + t["Ethree"] + t["Erot"] + t["Egrav"]
    return H, t, phi, rho, dx


def exact(case, seed):
    what, ndim = case["what"], _ndim(case)
    if what in ("tf", "solve", "sweep"):
        return None           # iterations: no closed value
    if what == "batch":
        out = []
        for i, c in enumerate(_sweep(case, seed)):
            out.append(_operators(case, _state(2, c["Ngrid"], c["L"], seed * 64 + i), c["Ngrid"], c["beta2"])[0])
        return out
    psi = _state(ndim, case["N"], case["L"], seed)
    if what == "phi":
        dx = 2.0 * case["L"] / case["N"]
        khat = _kernel_hat(case["kernel"], case["l_z"], ndim, case["N"], dx, psi.device)
        return -case["G_C"] * _convolve(psi.real ** 2 + psi.imag ** 2, khat, ndim, case["N"], dx)
    H, t, phi, rho, dx = _operators(case, psi, case["N"], case["beta2"])
    dv = dx ** ndim
    if what == "hpsi":
        return H
    if what == "evaluate":
        mu = float((psi.conj() * H).real.sum()) * dv
        r = math.sqrt(float(((H - mu * psi).abs() ** 2).sum()) * dv)
        return dict(t, phi=phi, resid=r, mu=mu, resid_rel=r / max(1.0, abs(mu)))
    f = lambda v: torch.tensor(v, dtype=torch.float64)
    gc = f(t["Egrav"] / case["G_C"] if case["kernel"] != "none" else 0.0)
    return dict(E=f(t["E"]), psi=2.0 * H * dv, params=[f(0.5 * float((rho ** 2).sum()) * dv),
                                                       f(float((rho ** 3).sum()) * dv / 3.0), gc, f(-t["Lz"])])
