"""Items of more rows of tiles than a grid has blocks along y."""

import pytest
import torch

import torchmorph_gb300 as tm

pytestmark = pytest.mark.gpu

ROWS = 65535 * 32 + 3000


@pytest.mark.parametrize("width", [8, 5])  # 16-byte aligned rows, others
def test_tall_flat_windows(cuda, width):
    x = torch.rand((1, 1, ROWS, width), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    box = torch.ones((13, 7), dtype=torch.bool)  # (beyond the bit tiles)
    for op, v in ((lambda t: tm.grey_dilation(t, size=7), x), (lambda t: tm.grey_dilation(t, size=(1, 3)), x),
                  (lambda t: tm.grey_erosion(t, size=(9, 1)), x),
                  (lambda t: tm.binary_erosion(t, structure=box), x > 0.1)):
        whole = op(v)
        # rows on both sides of the last block's, and the end: as in a part of the item
        for lo, hi in ((0, 2000), (65535 * 32 - 1000, 65535 * 32 + 1000), (ROWS - 2000, ROWS)):
            part = op(v[:, :, lo:hi].contiguous())
            a, b = (0 if lo == 0 else 10), (None if hi == ROWS else -10)
            assert torch.equal(whole[:, :, lo:hi][:, :, a:b], part[:, :, a:b])


def test_tall_staged_tiles(cuda):
    """The persistent kernel of compile-time windows (aligned rows of more than a tile)."""
    x = torch.rand((1, 1, ROWS, 144), generator=torch.Generator(device="cuda").manual_seed(2), device="cuda")
    whole = tm.grey_dilation(x, size=3, origin=1)
    for lo, hi in ((0, 500), (65535 * 32 - 300, 65535 * 32 + 300), (ROWS - 500, ROWS)):
        part = tm.grey_dilation(x[:, :, lo:hi].contiguous(), size=3, origin=1)
        a, b = (0 if lo == 0 else 10), (None if hi == ROWS else -10)
        assert torch.equal(whole[:, :, lo:hi][:, :, a:b], part[:, :, a:b])
