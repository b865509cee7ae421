"""FP32 Sinkhorn beyond the matrices that clusters and row slabs keep (more than 2048 points): the
tiled contractions in both forms, 16- and 64-pair tiles, one and several pair blocks, float4 and
scalar staging, the stopping test and its grid barrier, the caller's own matrices, the line
cost, and the transport-cost kernel of large batches, against float64."""

import pytest
import torch

from torchmorph_gb300 import _C, _lib, autotune

pytestmark = pytest.mark.gpu

EPS, ITS = 0.1, 20


def _problem(n, d, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    a, b = (torch.rand((n, d), generator=g, device="cuda") + 1e-2 for _ in range(2))
    p = torch.rand((d, 3), generator=g, device="cuda")
    cost = ((p[:, None] - 0.9 * p[None]) ** 2).sum(-1)  # not symmetric
    return a / a.sum(1, keepdim=True), b / b.sum(1, keepdim=True), (cost / cost.max()).contiguous()


def _solve64(a, b, cost, eps, its, log_space, kern=None, kern_t=None):
    a, b, cost = a.double(), b.double(), cost.double()
    kern = torch.exp(-cost / eps) if kern is None else kern.double()
    kern_t = kern.T if kern_t is None else kern_t.double()
    tiny = 0.0 if log_space else 1e-12
    u, v = torch.ones_like(a), torch.ones_like(b)
    for _ in range(its):
        u = a / (v @ kern.T + tiny)
        v = b / (u @ kern_t.T + tiny)
    plan_cost = (u * (v @ (kern * cost).T)).sum(1)
    residual = (a - u * (v @ kern.T)).abs().sum(1)
    return u.log(), v.log(), plan_cost, residual


def _tol(d):
    """40 half-steps; each sums d positive terms in one fp32 chain, whose rounding errors of at most
    2^-24 of the sum add up like a random walk: 4 sqrt(d) 2^-24 with room.  The maps do not expand."""
    return 40 * 4 * d ** 0.5 * 2.0 ** -24


# n = 5 takes the 16-pair tiles, 70 and 150 the 64-pair ones (one, two and three blocks of pairs);
# 150 pairs are enough for the cost kernel of 128-row blocks, the others take the 4-row one
@pytest.mark.parametrize("log_space", [False, True])
@pytest.mark.parametrize("n,d", [(5, 2100), (70, 2100), (30, 2051), (150, 2101)])
def test_tiles_against_float64(cuda, log_space, n, d):
    a, b, cost = _problem(n, d, n + d)
    log_u, log_v, got, row_err, iterations = _C.sinkhorn_f32_solve(a, b, cost, EPS, ITS, 0.0, log_space)
    u64, v64, c64, r64 = _solve64(a, b, cost, EPS, ITS, log_space)
    assert int(iterations) == ITS
    assert (log_u - u64).abs().max().item() <= _tol(d)
    assert (log_v - v64).abs().max().item() <= _tol(d)
    assert ((got - c64).abs() / c64).max().item() <= 2 * _tol(d)
    assert (row_err - r64).abs().max().item() <= 2 * _tol(d)


@pytest.mark.parametrize("log_space", [False, True])
@pytest.mark.parametrize("n,d", [(5, 2101), (70, 2100)])
def test_tiles_stopping_test(cuda, log_space, n, d):
    """Stops at the multiple of 5 whose float64 residual first lies below the threshold (set
    between the checks at 5 and 10, a factor away from both)."""
    a, b, cost = _problem(n, d, 7)

    def residual(its):  # of the plan that iteration `its` starts from
        return float(_solve64(a, b, cost, EPS, its - 1, log_space)[3].max())

    e5, e10 = residual(5), residual(10)
    assert e10 < 0.1 * e5
    out = _C.sinkhorn_f32_solve(a, b, cost, EPS, 100, (e5 * e10) ** 0.5, log_space, check_every=5)
    fixed = _C.sinkhorn_f32_solve(a, b, cost, EPS, 10, 0.0, log_space)
    assert int(out[4]) == 10 and torch.equal(out[0], fixed[0]) and torch.equal(out[1], fixed[1])


@pytest.mark.parametrize("log_space", [False, True])
def test_tiles_line_cost(cuda, log_space):
    n, d = 6, 2100
    a, b, _ = _problem(n, d, 11)
    at = torch.arange(d, device="cuda", dtype=torch.float32)
    cost = (at[:, None] - at[None]).abs()
    got = _C.sinkhorn_f32_solve(a, b, None, EPS * d, ITS, 0.0, log_space)
    u64, v64, c64, _ = _solve64(a, b, cost, EPS * d, ITS, log_space)
    assert (got[0] - u64).abs().max().item() <= _tol(d)
    assert (got[1] - v64).abs().max().item() <= _tol(d)
    assert ((got[2] - c64).abs() / c64).max().item() <= 2 * _tol(d)


@pytest.mark.parametrize("log_space", [False, True])
def test_tiles_on_the_callers_matrices(cuda, log_space):
    """The second matrix is used as it is, transpose of the first or not."""
    n, d = 20, 2052
    a, b, cost = _problem(n, d, 13)
    other = _problem(n, d, 14)[2]
    u, v = torch.ones_like(a), torch.ones_like(b)
    if log_space:
        u, v = torch.zeros_like(a), torch.zeros_like(b)
        _C.sinkhorn_logiter(a.log(), b.log(), cost, other, u, v, ITS, EPS)
    else:
        _C.sinkhorn_fastiter(a, b, torch.exp(-cost / EPS), torch.exp(-other / EPS), u, v, ITS)
        u, v = u.log(), v.log()
    u64, v64, _, _ = _solve64(a, b, cost, EPS, ITS, log_space, kern_t=torch.exp(-other.double() / EPS))
    # (the fp32 matrices: |cost| / eps 2^-24 relative)
    assert (u - u64).abs().max().item() <= _tol(d) + 40 * 2 * 2.0 ** -24 / EPS
    assert (v - v64).abs().max().item() <= _tol(d) + 40 * 2 * 2.0 ** -24 / EPS


@pytest.mark.parametrize("log_space", [False, True])
@pytest.mark.parametrize("n", [9, 70])
def test_tile_variants_agree_bit_for_bit(cuda, n, log_space):
    d = 2100
    a, b, cost = _problem(n, d, 17)
    cls = autotune.work_class("sinkhorn_f32", n, d)
    ref = _C.sinkhorn_f32_solve(a, b, cost, EPS, 5, 0.0, log_space)
    try:
        for variant in range(autotune.variants("sinkhorn_f32")):
            autotune.set_variant("sinkhorn_f32", cls, variant)
            got = _C.sinkhorn_f32_solve(a, b, cost, EPS, 5, 0.0, log_space)
            assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])
    finally:
        autotune.set_variant("sinkhorn_f32", cls, -1)


# the tiles, the slabs (log form) and the clusters, whose stopping test is their one common wait
@pytest.mark.parametrize("n,d,log_space", [(70, 2100, False), (20, 700, True), (60, 300, False)])
def test_wait_budget_of_the_stopping_test(cuda, n, d, log_space):
    lib = _lib.load()
    a, b, cost = _problem(n, d, 19)
    args = (a, b, cost, EPS, 12, 1e-30, log_space)
    ref = _C.sinkhorn_f32_solve(*args, check_every=3)
    torch.cuda.synchronize()
    assert lib.tm_device_error(1) == 0
    lib.tm_set_grid_wait_budget(0)
    try:
        _C.sinkhorn_f32_solve(*args, check_every=3)
        torch.cuda.synchronize()
        assert lib.tm_device_error(1) == 1
    finally:
        lib.tm_set_grid_wait_budget(-1)
    again = _C.sinkhorn_f32_solve(*args, check_every=3)
    torch.cuda.synchronize()
    assert lib.tm_device_error(1) == 0
    assert torch.equal(again[0], ref[0]) and torch.equal(again[1], ref[1])
