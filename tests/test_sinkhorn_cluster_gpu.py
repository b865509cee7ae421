"""Scaling-form Sinkhorn with the matrix kept by a cluster: pair counts around the clusters a
device holds (1, 2 and 4 pairs each), sizes at the edges of its rows, columns and splits,
with and without a stopping test, against float64."""

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


def _solve64(a, b, cost, eps, its):
    a, b, kern = a.double(), b.double(), torch.exp(-cost.double() / eps)
    u, v = torch.ones_like(a), torch.ones_like(b)
    for _ in range(its):
        u = a / (v @ kern.T + 1e-12)
        v = b / (u @ kern + 1e-12)
    return u.log(), v.log()


@pytest.mark.parametrize("n,d", [(1, 2), (152, 5), (153, 33), (305, 17), (601, 64), (2, 127), (77, 130), (40, 240),
                                 (30, 511), (15, 513), (9, 640), (14, 783), (16, 784), (28, 785), (7, 829)])
def test_cluster_solve_against_float64(cuda, n, d):
    """20 iterations: a sum of d positive terms in fp32 chains of at most 50 and trees is good to
    ~2e-6, and the maps do not expand, so the log-potentials stay within 40 of those.  A
    threshold below every residual changes nothing, bit for bit."""
    eps, its = 0.1, 20
    a, b, cost = _problem(n, d, 100 * n + d)
    log_u, log_v, _, _, iterations = _C.sinkhorn_f32_solve(a, b, cost, eps, its, 0.0, False)
    u64, v64 = _solve64(a, b, cost, eps, its)
    assert int(iterations) == its
    assert (log_u - u64).abs().max().item() <= 40 * 2e-6
    assert (log_v - v64).abs().max().item() <= 40 * 2e-6
    checked = _C.sinkhorn_f32_solve(a, b, cost, eps, its, 1e-30, False, check_every=7)
    assert torch.equal(checked[0], log_u) and torch.equal(checked[1], log_v) and int(checked[4]) == its


@pytest.mark.parametrize("n,d", [(20, 100), (160, 40), (10, 700)])
def test_cluster_stopping_test(cuda, n, d):
    """Stops at the multiple of 5 whose float64 residual first lies below the threshold (set
    between the checks at 5 and 10, a factor away from both)."""
    eps = 0.1
    a, b, cost = _problem(n, d, 7)
    kern = torch.exp(-cost.double() / eps)

    def residual(its):  # of the plan that iteration `its` starts from
        u, v = _solve64(a, b, cost, eps, its - 1)
        return float((a.double() - u.exp() * (v.exp() @ kern.T)).abs().sum(1).max())

    e5, e10 = residual(5), residual(10)
    assert e10 < 0.1 * e5
    out = _C.sinkhorn_f32_solve(a, b, cost, eps, 100, (e5 * e10) ** 0.5, False, check_every=5)
    fixed = _C.sinkhorn_f32_solve(a, b, cost, eps, 10, 0.0, False)
    assert int(out[4]) == 10 and torch.equal(out[0], fixed[0]) and torch.equal(out[1], fixed[1])
