"""Calls inside and after a CUDA default device: the elements stay on the host."""

import pytest
import torch

import torchmorph_gb300 as tm
from torchmorph_gb300 import ragged

pytestmark = pytest.mark.gpu


def _grey_calls(x, batch):
    fp = torch.tensor([[True, True, False], [True, True, True], [False, True, True]])
    ops = [tm.grey_erosion, tm.grey_dilation, tm.grey_opening, tm.grey_closing, tm.morphological_gradient,
           tm.morphological_laplace, tm.white_tophat, tm.black_tophat]
    out = [op(x, size=size) for op in ops for size in (3, 9)]
    out += [op(x, footprint=fp) for op in ops]
    out += [op(batch, size=5).data for op in (ragged.grey_erosion, ragged.grey_dilation, ragged.grey_opening)]
    leaf = x.clone().requires_grad_()
    res = tm.grey_dilation(leaf, size=5, differentiable=True)
    return out + [res.detach(), torch.autograd.grad(res.sum(), leaf)[0]]


def test_grey_under_a_cuda_default_device(cuda):
    x = torch.rand((2, 1, 40, 52), device="cuda")
    batch = ragged.RaggedBatch.from_images([x[0, 0], x[1, 0, :17, :23]])
    with torch.device("cuda"):
        inside = _grey_calls(x, batch)
    tm.grey_erosion(x, size=3)
    after = _grey_calls(x, batch)
    assert all(torch.equal(a, b) for a, b in zip(inside, after))


def _binary_calls(x, batch):
    ops = [tm.binary_erosion, tm.binary_dilation, tm.binary_opening, tm.binary_closing, tm.binary_hit_or_miss,
           tm.binary_fill_holes]
    box = torch.ones((3, 3), dtype=torch.bool)
    out = [op(x) for op in ops] + [op(x, structure=box) for op in ops[:4]]
    return out + [op(batch).data for op in (ragged.binary_erosion, ragged.binary_dilation, ragged.binary_opening)]


def test_binary_under_a_cuda_default_device(cuda):
    x = torch.rand((2, 1, 40, 52), device="cuda") > 0.4
    batch = ragged.RaggedBatch.from_images([x[0, 0], x[1, 0, :17, :23]])
    with torch.device("cuda"):
        inside = _binary_calls(x, batch)
    tm.binary_erosion(x)
    after = _binary_calls(x, batch)
    assert all(torch.equal(a, b) for a, b in zip(inside, after))
