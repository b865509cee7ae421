"""One-pass opening / closing tiles: window sizes around the runs of 4 and 8 outputs, on
items around the 32 x 128 tile, bit for bit against the oracle's two operators."""

import numpy as np
import pytest
import torch

import oracle
import torchmorph_gb300 as tm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 33), (33, 1), (2, 3), (3, 4), (4, 5), (5, 7), (7, 8), (8, 9), (9, 2), (16, 33),
                                  (33, 33)])
@pytest.mark.parametrize("shape,mode", [((2, 1, 31, 127), "reflect"), ((1, 1, 33, 129), "nearest"),
                                        ((1, 1, 65, 260), "mirror"), ((1, 1, 40, 131), "constant"),
                                        ((1, 1, 64, 128), "wrap"), ((2, 1, 5, 3), "reflect")])
def test_open_close_tophat_windows(cuda, shape, mode, size):
    r = np.random.default_rng(size[0] * 40 + size[1])
    x = r.random(shape, dtype=np.float32)
    st = np.zeros(size, np.float32)
    ero = lambda v, d: oracle.grey(v, st, mode=mode, cval=0.25, dilation=d)  # noqa: E731
    opened, closed = ero(ero(x, False), True), ero(ero(x, True), False)
    t = torch.from_numpy(x).cuda()
    kw = dict(size=size, mode=mode, cval=0.25)
    np.testing.assert_array_equal(tm.grey_opening(t, **kw).cpu().numpy(), opened)
    np.testing.assert_array_equal(tm.grey_closing(t, **kw).cpu().numpy(), closed)
    np.testing.assert_array_equal(tm.white_tophat(t, **kw).cpu().numpy(), x - opened)
    np.testing.assert_array_equal(tm.black_tophat(t, **kw).cpu().numpy(), closed - x)
