"""Point-cloud Sinkhorn at the edges of its work split (16 own points to a warp, 64 partners to
a step, more items than warps) and where the shifted sums leave their range, vs float64."""

import numpy as np
import pytest
import torch

import oracle
from torchmorph_gb300 import PointCloudSinkhorn, _lib, pack_clouds

pytestmark = pytest.mark.gpu

EDGES = [(15, 63), (16, 64), (17, 65), (1, 129), (33, 128), (31, 1), (64, 16), (130, 320)]


@pytest.mark.parametrize("sizes,eps,iters", [
    (EDGES, 0.1, 12),
    (EDGES, 0.003, 12),  # exponents move by thousands from one iteration to the next
    ([(17 + p % 30, 3 + p % 70) for p in range(1500)], 0.2, 4),
], ids=["edges", "tiny_eps", "many"])
def test_items_vs_fp64_oracle(cuda, sizes, eps, iters):
    r = np.random.default_rng(5)
    xs = [r.uniform(-1, 1, (n, 3)).astype(np.float32) for n, _ in sizes]
    ys = [r.uniform(-1, 1, (m, 3)).astype(np.float32) for _, m in sizes]
    x, nx = pack_clouds([torch.from_numpy(v).cuda() for v in xs])
    y, ny = pack_clouds([torch.from_numpy(v).cuda() for v in ys])
    res = PointCloudSinkhorn(epsilon=eps, max_iter=iters, threshold=0.0).solve(x, y, nx, ny)
    torch.cuda.synchronize()
    assert _lib.load().tm_device_error(1) == 0
    f, g = res["f"].cpu().numpy(), res["g"].cpu().numpy()
    ox, oy = np.cumsum([0] + nx), np.cumsum([0] + ny)
    # A half-iteration's own error, in potential units: 4 roundings (2^-24) of terms up to
    # 2 |x^| |y^| <= 2 * 12 (centred points of the cube) -> 6e-6; the log-sum-exp passes earlier
    # errors on without growth, so 2 * iters of them add at most.
    tol = 2 * iters * 6e-6
    for p in range(len(sizes)):
        fo, go, _, cost = oracle.pointcloud_sinkhorn(xs[p].astype(np.float64), ys[p].astype(np.float64), eps, iters,
                                                     threshold=0.0)
        df, dg = f[ox[p]:ox[p + 1]] - fo, g[oy[p]:oy[p + 1]] - go
        assert max(np.abs(df).max(), np.abs(dg).max()) < tol, (sizes[p], np.abs(df).max(), np.abs(dg).max())
        assert abs(res["cost"][p].item() - cost) < 2 * tol
