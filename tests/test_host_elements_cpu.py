"""Structuring elements are read on the host: they stay CPU tensors with memory of their own under
any default device, and under a mode whose tensors have none nothing is kept for later calls."""

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from torchmorph_gb300 import _lib
from torchmorph_gb300.morphology import binary, generate_binary_structure, grey


def _is_plain(t):
    return type(t) is torch.Tensor and t.device.type == "cpu" and t.data_ptr() != 0


@pytest.mark.parametrize("size", [3, (4, 11), (70, 70)])  # (cached, and beyond the cache)
def test_grey_box_under_a_default_device(size):
    with torch.device("meta"):
        inside, _ = grey._resolve_element(2, size, None, None)
    after, _ = grey._resolve_element(2, size, None, None)
    assert _is_plain(inside) and _is_plain(after)


def test_grey_footprint_under_a_default_device():
    fp = torch.tensor([[True, False], [True, True]])
    with torch.device("meta"):
        struct, mask = grey._resolve_element(2, None, fp, None)
    assert _is_plain(struct) and _is_plain(mask)


def test_grey_box_made_under_a_mode_is_not_kept():
    with FakeTensorMode():
        grey._resolve_element(2, (6, 13), None, None)
    assert _is_plain(grey._resolve_element(2, (6, 13), None, None)[0])

    def traced(x):
        grey._resolve_element(2, (6, 17), None, None)
        return x + 1

    torch.func.functionalize(traced)(torch.zeros(3))
    assert _is_plain(grey._resolve_element(2, (6, 17), None, None)[0])


def test_no_host_address_of_a_device_tensor():
    with pytest.raises(RuntimeError, match="CPU tensor"):
        _lib.ctypes_f32(torch.zeros(3, device="meta"))
    with pytest.raises(RuntimeError, match="CPU tensor"):
        _lib.ctypes_u8(torch.zeros(3, dtype=torch.bool, device="meta"))


@pytest.mark.parametrize("nd", [1, 2, 3, 4])
def test_default_cross_under_a_default_device(nd):
    with torch.device("meta"):
        inside, empty = binary._normalize_structure(None, nd)
    after, _ = binary._normalize_structure(None, nd)
    assert not empty and _is_plain(inside) and _is_plain(after)
    assert torch.equal(after, generate_binary_structure(nd, 1))


def test_default_cross_made_under_a_mode_is_not_kept():
    with FakeTensorMode():
        binary._normalize_structure(None, 5)
    assert _is_plain(binary._normalize_structure(None, 5)[0])
