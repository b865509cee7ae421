"""FP32 Sinkhorn on resident row slabs: sizes at the edges of its tiles (8 rows, 4 or 8
pairs, 128 / 1024 columns per warp / warp set, the largest slab), against float64."""

import pytest
import torch

from torchmorph_gb300 import _C

pytestmark = pytest.mark.gpu


def _problem(n, d, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    a, b = (torch.rand((n, d), generator=g, device="cuda") + 1e-2 for _ in range(2))
    p = torch.rand((d, 3), generator=g, device="cuda")
    cost = ((p[:, None] - 0.9 * p[None]) ** 2).sum(-1)  # not symmetric
    return a / a.sum(1, keepdim=True), b / b.sum(1, keepdim=True), (cost / cost.max()).contiguous()


def _solve64(a, b, cost, eps, its, log_space):
    a, b, cost = a.double(), b.double(), cost.double()
    kern = torch.exp(-cost / eps)
    tiny = 0.0 if log_space else 1e-12
    u, v = torch.ones_like(a), torch.ones_like(b)
    for _ in range(its):
        u = a / (v @ kern.T + tiny)
        v = b / (u @ kern + tiny)
    plan_cost = (u * (v @ (kern * cost).T)).sum(1)
    residual = (a - u * (v @ kern.T)).abs().sum(1)
    return u.log(), v.log(), plan_cost, residual


@pytest.mark.parametrize("log_space", [False, True])
@pytest.mark.parametrize("n,d", [(1, 1), (3, 7), (9, 8), (8, 128), (17, 129), (33, 257), (5, 1021), (9, 1024),
                                 (6, 1025), (4, 1216), (13, 1217), (2, 1700)])
def test_slab_solve_against_float64(cuda, log_space, n, d):
    """20 iterations: a half-step's sum of d positive terms is good to ~1e-6 (a tree of fp32
    sums; the log form adds |z| 2^-24 with |z| <= 1.5 / eps), and the maps do not expand, so
    the log-potentials stay within 40 of those."""
    eps, its = 0.1, 20
    a, b, cost = _problem(n, d, 100 * n + d)
    log_u, log_v, got_cost, row_err, iterations = _C.sinkhorn_f32_solve(a, b, cost, eps, its, 0.0, log_space)
    u64, v64, c64, r64 = _solve64(a, b, cost, eps, its, log_space)
    tol = 40 * (2.5e-6 if log_space else 1e-6)
    # the scalings are defined up to one factor per pair, which u = 1 at the start fixes
    assert (log_u - u64).abs().max().item() <= tol
    assert (log_v - v64).abs().max().item() <= tol
    assert ((got_cost - c64).abs() / c64.clamp(min=1e-6)).max().item() <= 2 * tol
    assert (row_err - r64).abs().max().item() <= 2 * tol
    assert int(iterations) == its


@pytest.mark.parametrize("log_space", [False, True])
@pytest.mark.parametrize("n,d", [(20, 100), (11, 1100)])
def test_slab_stopping_test_matches_the_float64_iteration(cuda, log_space, n, d):
    """The first multiple of 5 whose residual is below the threshold in float64 is the one
    the device stops at (the threshold lies between the checks at 5 and 10, a factor away
    from both and far above the residual that float32 potentials keep, about 3e-7)."""
    eps = 0.1
    a, b, cost = _problem(n, d, 7)
    errs = [_solve64(a, b, cost, eps, k - 1, log_space) for k in (5, 10)]

    def row_residual(sol, its):  # residual of the plan that iteration `its` starts from
        return (a.double() - sol[0].exp() * (sol[1].exp() @ torch.exp(-cost.double() / eps).T)).abs().sum(1).max()

    e5, e10 = (float(row_residual(s, k)) for s, k in zip(errs, (5, 10)))
    assert e10 < 0.1 * e5
    threshold = (e5 * e10) ** 0.5
    out = _C.sinkhorn_f32_solve(a, b, cost, eps, 100, threshold, log_space, check_every=5)
    fixed = _C.sinkhorn_f32_solve(a, b, cost, eps, 10, 0.0, log_space)
    assert int(out[4]) == 10
    assert (out[0] - fixed[0]).abs().max().item() <= 1e-4
