"""The mixed-precision solver's passes at every compiled grid size and in each of its
configurations (tile widths and factorizations follow from the points of a group of
instances), against the FP64 solver: ground states of a trapped repulsive cloud with and
without a long-range kernel, alone and in batches that fill the GPU or mix sizes.

Tolerance on the energy: 1e-10 max(1, |E|), the solver's bar. Both runs stop at a residual
r <= 1e-6, and the energy is second order in it (r^2 ~ 1e-12 at most)."""
import pytest
import torch

from becgpp_b200 import BatchSolver, default_cfg, ground_state, make_grid, make_seed

pytestmark = pytest.mark.gpu

CASES = [("2D", n, k) for n in (16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512) for k in ("none", "log")
         if k == "none" or n in (16, 48, 96, 192, 384)] + [("3D", n, k) for n in (16, 24, 48, 64) for k in ("none", "newton")]


def _cfg(dim, N, kern, **kw):
    return default_cfg(mode="single", dimension=dim, kernel=kern, Ngrid=N, L=(5.0 if N < 32 else 7.0), beta2=20.0,
                       G_C=(0.0 if kern == "none" else 2.0), seed="gaussian", seed_noise=1e-2, rng=N, res_tol=1e-7,
                       maxit=600, **kw)


def _check(om, o6):
    assert om["resid_rel"] <= 1e-6 and o6["resid_rel"] <= 1e-6, (om["resid_rel"], o6["resid_rel"])
    assert abs(om["E"] - o6["E"]) <= 1e-10 * max(1.0, abs(o6["E"])), (om["E"], o6["E"])
    assert om["fp64_from"] > 0


@pytest.mark.parametrize("dim,N,kern", CASES)
def test_energy_equals_fp64(dim, N, kern):
    c = _cfg(dim, N, kern)
    G = make_grid(c)
    psi0 = make_seed(G, c)
    _, _, o6 = ground_state(c, G=G, psi0=psi0, verbose=False)
    _, _, om = ground_state(dict(c, precision="mixed"), G=G, psi0=psi0, verbose=False)
    _check(om, o6)


@pytest.mark.parametrize("sizes", [(256,) * 4, (64, 64, 96, 96, 128), (256,) * 9, (32,) * 70])
def test_batches_equal_fp64(sizes):
    cfgs = [_cfg("2D", n, "none", precision="mixed") for n in sizes]
    for i, c in enumerate(cfgs):
        c["beta2"] += i
    grids = [make_grid(c) for c in cfgs]
    psi0 = [make_seed(G, c) for G, c in zip(grids, cfgs)]
    bs = BatchSolver(cfgs, grids)
    res = bs.solve(psi0)
    bs.close()
    for i in sorted({0, 1, len(sizes) // 2, len(sizes) - 1}):
        _, _, o6 = ground_state(dict(cfgs[i], precision="fp64"), G=grids[i], psi0=psi0[i], verbose=False)
        _check(res[i][2], o6)


def test_iteration_limit_before_the_hand_over():
    # the state returned is still an FP32 iterate, evaluated in FP64
    c = _cfg("2D", 96, "none", precision="mixed")
    c["maxit"] = 4
    _, _, o = ground_state(c, verbose=False)
    assert o["iters"] == 4 and o["fp64_from"] == -1 and o["stop_reason"] == "maxit"
    c6 = dict(c, precision="fp64")
    _, _, o6 = ground_state(c6, verbose=False)
    # four steps of FP32 transforms: a few ulps of FP32 each
    assert abs(o["E"] - o6["E"]) <= 1e-5 * abs(o6["E"]), (o["E"], o6["E"])
