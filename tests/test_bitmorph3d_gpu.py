"""Bit-packed 3-D binary morphology at the edges of its tiles (8 planes, 8 / 16 / 32 rows,
words of 32 voxels) and of its reach, bit for bit against the oracle."""

import numpy as np
import pytest
import torch

import oracle
import torchmorph_gb300 as tm

pytestmark = pytest.mark.gpu

_OPS = {"erosion": tm.binary_erosion, "dilation": tm.binary_dilation, "opening": tm.binary_opening,
        "closing": tm.binary_closing}


def _expected(kind, x, st, origin, border):
    if kind in ("erosion", "dilation"):
        return oracle.binary(x, st, origin, border, dilation=kind == "dilation")
    first = oracle.binary(x, st, origin, border, dilation=kind == "closing")
    return oracle.binary(first, st, origin, border, dilation=kind == "opening")


def _element(name, r):
    if name == "cross":
        return None, tm.generate_binary_structure(3, 1).numpy(), 0
    if name == "box":
        return np.ones((3, 3, 3), bool), np.ones((3, 3, 3), bool), 0
    if name == "box5":
        return np.ones((5, 5, 5), bool), np.ones((5, 5, 5), bool), 0
    if name == "wide":  # the reach's edge: 5 x 5 x 33 with a few voxels, shifted
        st = np.zeros((5, 5, 33), bool)
        st[r.integers(0, 5, 40), r.integers(0, 5, 40), r.integers(0, 33, 40)] = True
        st[0, 4, 0] = st[4, 0, 32] = True
        return st, st, 0
    if name == "even":
        st = r.random((2, 4, 6)) < 0.7
        st[0, 0, 0] = True
        return st, st, (0, -1, 2)
    st = np.ones((7, 3, 3), bool)  # beyond the reach: the byte tiles
    return st, st, 0


@pytest.mark.parametrize("kind", list(_OPS))
@pytest.mark.parametrize("element", ["cross", "box", "box5", "wide", "even", "beyond"])
@pytest.mark.parametrize("shape", [(1, 1, 1, 1, 1), (2, 1, 3, 5, 7), (1, 2, 8, 8, 31), (1, 1, 9, 33, 32),
                                   (2, 1, 17, 15, 33), (1, 1, 8, 16, 64), (1, 1, 10, 9, 65), (1, 1, 5, 17, 129),
                                   (1, 1, 16, 8, 200)])
def test_bit_tiles_3d(cuda, shape, element, kind):
    r = np.random.default_rng(sum(shape) + len(element))
    x = r.random(shape) < (0.8 if kind in ("erosion", "opening") else 0.2)
    given, st, origin = _element(element, r)
    structure = None if given is None else torch.from_numpy(given)
    for border in (False, True):
        got = _OPS[kind](torch.from_numpy(x).cuda(), structure=structure, border_value=border, origin=origin)
        o = [origin] * 3 if isinstance(origin, int) else list(origin)
        np.testing.assert_array_equal(got.cpu().numpy(), _expected(kind, x, st, o, border).astype(bool))


def test_bit_tiles_3d_off_alignment_and_iterations(cuda):
    """Inputs that start off a 4-byte boundary, and the paths that keep composing operators."""
    r = np.random.default_rng(3)
    shape = (2, 1, 11, 13, 45)
    x = r.random(shape) < 0.6
    buf = torch.zeros(x.size + 3, dtype=torch.bool, device="cuda")
    view = buf[3:].view(shape)
    view.copy_(torch.from_numpy(x))
    st = tm.generate_binary_structure(3, 1).numpy()
    got = tm.binary_opening(view)
    np.testing.assert_array_equal(got.cpu().numpy(), _expected("opening", x, st, [0, 0, 0], False).astype(bool))
    twice = tm.binary_opening(view, iterations=2)
    e = oracle.binary(oracle.binary(x, st, [0] * 3, False), st, [0] * 3, False)
    d = oracle.binary(oracle.binary(e, st, [0] * 3, False, dilation=True), st, [0] * 3, False, dilation=True)
    np.testing.assert_array_equal(twice.cpu().numpy(), d.astype(bool))


def test_bit_tiles_3d_ignore_the_bytes_behind_the_input(cuda):
    """The last words of the input are loaded whole; what lies behind its end does not count."""
    r = np.random.default_rng(4)
    shape = (1, 1, 2, 3, 7)
    x = r.random(shape) < 0.5
    buf = torch.full((x.size + 64,), 255, dtype=torch.uint8, device="cuda")
    for start in range(4):
        view = buf[start:start + x.size].view(torch.bool).view(shape)
        view.copy_(torch.from_numpy(x))
        got = tm.binary_dilation(view)
        exp = oracle.binary(x, tm.generate_binary_structure(3, 1).numpy(), [0, 0, 0], False, dilation=True)
        np.testing.assert_array_equal(got.cpu().numpy(), exp.astype(bool))
