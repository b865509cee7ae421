"""EDT line passes (windows, then halving) at the edges of their tiles and ranges, bit for
bit against the oracle: objects with distances inside the first window, the second, and far
beyond both; lines around 8, 32, 128 voxels and the longest; unaligned rows; spacings that
run on integers."""

import numpy as np
import pytest
import torch

import oracle
import torchmorph_gb300 as tm

pytestmark = pytest.mark.gpu


def _masks(shape, kind, seed):
    r = np.random.default_rng(seed)
    if kind == "noise":
        return r.random(shape) < 0.8
    if kind == "sparse":
        return r.random(shape) < 1.0 - 3.0 / np.prod(shape[2:])
    if kind == "seed":  # one background voxel per item
        x = np.ones(shape, bool)
        for b in range(shape[0]):
            x[(b, 0) + tuple(int(r.integers(0, s)) for s in shape[2:])] = False
        return x
    if kind == "stripes":  # equal distances on both sides: ties everywhere
        x = np.ones(shape, bool)
        x[..., ::7] = False
        x[:, :, ::5] = False
        return x
    # blocks of foreground and background about 30 voxels wide
    cells = r.random(shape[:2] + tuple(-(-s // 30) + 1 for s in shape[2:])) < 0.6
    for axis, s in enumerate(shape[2:], start=2):
        cells = np.repeat(cells, 30, axis=axis).take(np.arange(s) + 7, axis=axis)
    return cells


def _check(x, sampling=None, dtype=torch.bool):
    t = torch.as_tensor(x, device="cuda").to(dtype)
    d, idx = tm.euclidean_distance_transform(t, sampling=sampling, return_indices=True)
    sq, od, oi = oracle.edt(x, sampling)
    np.testing.assert_array_equal(d.cpu().numpy(), od.astype(np.float32))
    np.testing.assert_array_equal(idx.cpu().numpy(), oi)
    alone = tm.euclidean_distance_transform(t, sampling=sampling)
    assert torch.equal(alone, d)
    if sampling is None:
        s = tm.euclidean_distance_transform_squared(t)
        np.testing.assert_array_equal(s.cpu().numpy(), sq.astype(np.int32))


SHAPES_2D = [(2, 1, 1, 1), (1, 1, 7, 8), (3, 1, 33, 31), (2, 1, 9, 129), (1, 1, 128, 128), (2, 1, 257, 65),
             (1, 1, 500, 333), (1, 1, 40, 2100), (1, 1, 2100, 20), (1, 1, 3, 4096)]


@pytest.mark.parametrize("kind", ["noise", "sparse", "seed", "stripes", "blocks"])
@pytest.mark.parametrize("shape", SHAPES_2D)
def test_lines_2d(cuda, shape, kind):
    _check(_masks(shape, kind, sum(shape)))


SHAPES_3D = [(1, 1, 3, 5, 2), (2, 1, 9, 8, 16), (1, 1, 5, 33, 17), (2, 1, 31, 40, 100), (1, 1, 64, 70, 128),
             (1, 1, 40, 90, 129), (1, 1, 70, 257, 33), (1, 1, 3, 1024, 9), (1, 1, 260, 6, 40), (1, 1, 6, 5, 700)]


@pytest.mark.parametrize("kind", ["noise", "sparse", "seed", "stripes", "blocks"])
@pytest.mark.parametrize("shape", SHAPES_3D)
def test_lines_3d(cuda, shape, kind):
    _check(_masks(shape, kind, sum(shape)))


@pytest.mark.parametrize("kind", ["noise", "sparse", "blocks"])
@pytest.mark.parametrize("shape,sampling", [((2, 1, 30, 44, 52), (2.5, 1.0, 1.0)), ((1, 1, 33, 40, 129), (1.0, 1.0, 2.5)),
                                            ((1, 1, 25, 60, 40), (3.0, 0.75, 0.75)), ((2, 1, 90, 133), (0.5, 2.0)),
                                            ((1, 1, 64, 200), (1.25, 0.875)), ((1, 1, 20, 30, 40), (255.0, 1.0, 2.0))])
def test_lines_with_integer_spacing(cuda, shape, sampling, kind):
    _check(_masks(shape, kind, sum(shape)), sampling)


@pytest.mark.parametrize("shape", [(3, 1, 61, 47), (3, 1, 20, 24, 40)])
def test_lines_mixed_items_float_and_unaligned_outputs(cuda, shape):
    """Items without background or foreground between ordinary ones, float input, and
    outputs that start off a 16-byte boundary."""
    x = _masks(shape, "blocks", 3)
    x[0] = True
    x[2] = False
    _check(x, dtype=torch.float32)
    _check(x)
    n = int(np.prod(shape))
    buf = torch.empty(n + 1, dtype=torch.float32, device="cuda")
    out = buf[1:].view(shape)
    tm.euclidean_distance_transform(torch.as_tensor(x, device="cuda"), distances=out)
    np.testing.assert_array_equal(out.cpu().numpy(), oracle.edt(x)[1].astype(np.float32))
