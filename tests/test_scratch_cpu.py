"""Scratch sizes (no GPU): what a solver asks for grows with the problem, not with kernels that
the problem does not reach."""

import pytest

from torchmorph_gb300 import _lib


def _up(nbytes):
    return (nbytes + 255) & ~255


@pytest.mark.parametrize("log_space", [0, 1])
@pytest.mark.parametrize("check", [0, 10])
@pytest.mark.parametrize("n,d", [(10 ** 6, 64), (10 ** 6, 200), (20000, 1024)])
def test_sinkhorn_f32_scratch_of_many_pairs(n, d, check, log_space):
    # matrices, scalings, and per pair and 128 rows one residual and two cost partials
    blocks = -(-d // 128)
    limit = 2 * _up(4 * d * d) + 2 * _up(4 * n * d) + 3 * _up(8 * blocks * n) + _up(8 * n) + 4096
    assert _lib.load().tm_sinkhorn_f32_workspace_size(n, d, log_space, 100, check, 0) <= limit


def test_sinkhorn_f32_scratch_holds_the_residuals_of_every_kernel():
    size = _lib.load().tm_sinkhorn_f32_workspace_size
    for n, d in [(1, 1), (16, 64), (16, 784), (300, 2048), (16384, 64), (3, 5000)]:
        rows = max(-(-d // 128), min(160, max(32, -(-d // 8))))
        assert size(n, d, 0, 100, 10, 0) - size(n, d, 0, 100, 0, 0) >= 8 * n * rows
        rows = max(-(-d // 128), min(160, -(-d // 8)))  # (the log form has no clusters)
        assert size(n, d, 1, 100, 10, 0) - size(n, d, 1, 100, 0, 0) >= 8 * n * rows
