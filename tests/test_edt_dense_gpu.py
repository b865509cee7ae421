"""EDT line passes over dense backgrounds, bit for bit against the oracle: tiles that end with the
first window and tiles that do not, rows staged flat and in units (around 73, 128, 146 and 256
voxels), tiles of 8, 16 and 32 lines, lines without background, spacings with and without the
table of small distances."""

import numpy as np
import pytest
import torch

import oracle
import torchmorph_gb300 as tm

pytestmark = pytest.mark.gpu


def _check(x, sampling=None):
    t = torch.as_tensor(x, device="cuda")
    d, idx = tm.euclidean_distance_transform(t, sampling=sampling, return_indices=True)
    _, od, oi = oracle.edt(x, sampling)
    np.testing.assert_array_equal(d.cpu().numpy(), od.astype(np.float32))
    np.testing.assert_array_equal(idx.cpu().numpy(), oi)
    assert torch.equal(tm.euclidean_distance_transform(t, sampling=sampling), d)


def _noise(shape, fill):
    x = np.random.default_rng(sum(shape)).random(shape) < fill
    if shape[0] > 1:
        x[1] = True  # an item without background
    return x


# (few rows: tiles of 8 or 16 lines; 640 x 32 rows: tiles of 32, in 3-D 16 at 129 .. 256)
@pytest.mark.parametrize("fill", [0.5, 0.95])
@pytest.mark.parametrize("width", [5, 73, 74, 128, 129, 146, 147, 256, 257])
def test_dense_rows(cuda, width, fill):
    _check(_noise((3, 1, 37, width), fill))
    _check(_noise((2, 1, 7, 11, width), fill))


@pytest.mark.parametrize("shape", [(640, 1, 32, 61), (640, 1, 32, 127), (24, 1, 20, 21, 131), (24, 1, 20, 21, 202)])
def test_dense_rows_of_many_tiles(cuda, shape):
    _check(_noise(shape, 0.5))


@pytest.mark.parametrize("sampling", [(1.0, 0.5), (0.25, 0.25), (1.0, 1.5), (2.0, 2.0)])
def test_dense_rows_with_spacing(cuda, sampling):
    _check(_noise((2, 1, 40, 77), 0.5), sampling)
    _check(_noise((2, 1, 6, 21, 140), 0.5), (1.0, *sampling))
