"""The autotuner decides by calls that the variants apply to: others leave a class as it was."""

import pytest
import torch

import torchmorph_gb300 as tm
from torchmorph_gb300 import autotune

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _restore_table():
    yield
    for op in autotune.OPS:
        for cls in range(64):
            autotune.set_variant(op, cls, -1)


def _sinkhorn(n, d):
    gen = torch.Generator(device="cuda").manual_seed(d)
    a, b = (torch.rand((n, d), generator=gen, device="cuda") + 0.1 for _ in range(2))
    return a / a.sum(1, keepdim=True), b / b.sum(1, keepdim=True), torch.rand((d, d), generator=gen, device="cuda")


def _entry(path, op, res):
    name = torch.cuda.get_device_name(torch.cuda.current_device())
    return autotune.load_cache(path)["devices"][name][op][str(res["class"])]


@pytest.mark.parametrize("log_space", [False, True])
def test_a_problem_of_other_kernels_decides_nothing(cuda, tmp_path, log_space):
    path = str(tmp_path / "t.json")
    a, b, cost = _sinkhorn(40, 300)  # clusters, slabs
    res = autotune.tune_sinkhorn(a, b, cost, 0.1, max_iter=5, log_space=log_space, path=path)
    assert res["best"] == -1 and len(res["times_ms"]) == autotune.variants("sinkhorn_f32")
    assert autotune.get_variant("sinkhorn_f32", res["class"]) == -1 == _entry(path, "sinkhorn_f32", res)
    assert autotune.apply_cache(path=path) == 0
    # a class that has a choice keeps it, and the cache its entry
    autotune.set_variant("sinkhorn_f32", res["class"], 2)
    data = autotune.load_cache(path)
    next(iter(data["devices"].values()))["sinkhorn_f32"][str(res["class"])] = 2
    autotune.save_cache(data, path)
    again = autotune.tune_sinkhorn(a, b, cost, 0.1, max_iter=5, log_space=log_space, path=path)
    assert again["best"] == 2 == autotune.get_variant("sinkhorn_f32", res["class"]) == _entry(path, "sinkhorn_f32", res)


def test_a_problem_of_the_tiles_decides(cuda, tmp_path):
    path = str(tmp_path / "t.json")
    a, b, cost = _sinkhorn(40, 2100)
    res = autotune.tune_sinkhorn(a, b, cost, 0.1, max_iter=3, path=path)
    assert 0 <= res["best"] < 4 and _entry(path, "sinkhorn_f32", res) == res["best"]


def test_boxes(cuda, tmp_path):
    path = str(tmp_path / "t.json")
    x = torch.rand((8, 1, 1024, 1024), device="cuda")
    assert autotune.tune_grey_dilation(x, size=3, path=path)["best"] == -1  # the register walkers
    res = autotune.tune("grey_flat2d", lambda: tm.grey_dilation(x, size=3, origin=1), x.numel(), path=path)
    assert 0 <= res["best"] < 4 and _entry(path, "grey_flat2d", res) == res["best"]


def test_distance_transforms(cuda, tmp_path):
    path = str(tmp_path / "t.json")
    odd = torch.rand((1, 1, 40, 40, 41), device="cuda") < 0.9  # no shell search for either
    assert autotune.tune_edt(odd, path=path)["best"] == -1
    assert autotune.tune_cdt(odd, path=path)["best"] == -1
    even = torch.rand((1, 1, 40, 40, 128), device="cuda") < 0.9
    assert autotune.tune_edt(even, path=path)["best"] in (0, 1)
    assert autotune.tune_cdt(even, path=path)["best"] in (0, 1, 2)
