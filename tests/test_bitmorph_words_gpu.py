"""Bit tiles of 1-D / 2-D items: row starts at every byte alignment, rows that end in every part
of a word, and the fused operators where their reaches add up to one word, just fit and do
not: bit-exact against the oracle."""

import numpy as np
import pytest
import torch

import oracle
import torchmorph_gb300 as tm
from tests.helpers import rng

pytestmark = pytest.mark.gpu


def _line(n):
    return np.ones((1, n), bool)


@pytest.mark.parametrize("width", [1, 15, 31, 33, 127, 129, 161, 259])
@pytest.mark.parametrize("name,st,origin", [
    ("reach32", _line(33), (0, 0)),    # 16 + 16 columns
    ("reach34", _line(35), (0, 0)),
    ("left", _line(9), (0, 4)),        # all taps on one side
    ("column", np.ones((5, 1), bool), (0, 0)),
    ("ring", np.array([[1, 1, 1], [1, 0, 1], [1, 1, 0]], bool), (0, 0)),
])
@pytest.mark.parametrize("border", [False, True])
def test_words_and_alignment(cuda, width, name, st, origin, border):
    r = rng(width + len(name))
    for offset in (0, 3, 13):  # first byte of the items in their 16-byte piece
        x = r.random((2, 1, 37, width)) < (0.9 if border else 0.6)
        buf = torch.ones(x.size + offset + 64, dtype=torch.bool, device="cuda")
        v = buf[offset:offset + x.size].view(x.shape)
        v.copy_(torch.from_numpy(x))
        ero = oracle.binary(x, st, origin, border, dilation=False)
        want = {"erosion": ero, "opening": oracle.binary(ero, st, origin, border, dilation=True)}
        for kind, fn in (("erosion", tm.binary_erosion), ("opening", tm.binary_opening)):
            got = fn(v, structure=torch.from_numpy(st), border_value=border, origin=list(origin))
            np.testing.assert_array_equal(got.cpu().numpy(), want[kind], err_msg="%s offset %d" % (kind, offset))
