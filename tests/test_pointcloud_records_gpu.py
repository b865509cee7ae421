"""Records of the point-cloud solver: clouds whose last step ends anywhere between packed
neighbours, against float64."""

import math

import pytest
import torch

import torchmorph_gb300 as tm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [1, 15, 16, 17, 33, 48, 49, 63, 64, 65, 112, 127, 129])
def test_last_steps_between_neighbours(cuda, first):
    """Three iterations (the first with running maxima, the others shifted) of clouds around
    multiples of 16 and 64 partners; one neighbour holds NaN and infinity, which stay its own."""
    eps, its = 0.1, 3
    nx, ny = [first, 40, 16, first + 3], [first + 1, 7, first, 80]
    gen = torch.Generator(device="cuda").manual_seed(first)
    x, y = (torch.rand((sum(k), 3), generator=gen, device="cuda") for k in (nx, ny))
    x[nx[0]:nx[0] + 2, 1] = torch.tensor([math.nan, math.inf], device="cuda")
    res = tm.PointCloudSinkhorn(epsilon=eps, max_iter=its, threshold=0.0).solve(x, y, nx, ny)
    ox = oy = 0
    for p, (n, m) in enumerate(zip(nx, ny)):
        xp, yp = x[ox:ox + n].double(), y[oy:oy + m].double()
        if p != 1:
            k = -((xp[:, None] - yp[None]) ** 2).sum(-1) / eps
            la, lb = -math.log(n), -math.log(m)
            g = torch.full((m,), -lb, dtype=torch.float64, device="cuda")
            for _ in range(its):
                f = -torch.logsumexp(k + (g + lb), 1)
                g = -torch.logsumexp(k + (f + la)[:, None], 0)
            # |C| / eps <= 30 and sums of 2^-24 each, over 6 half-steps
            tol = 6 * eps * (30 * 2.0 ** -22)
            assert (res["f"][ox:ox + n].double() - eps * f).abs().max().item() <= tol
            assert (res["g"][oy:oy + m].double() - eps * g).abs().max().item() <= tol
        ox, oy = ox + n, oy + m
