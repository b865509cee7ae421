"""Two threads, two problem sizes, one kernel: the kernels' shared-memory limit belongs to the
process, so neither thread's launches may depend on what the other has just set."""

import threading

import pytest
import torch

import torchmorph_gb300 as tm
from torchmorph_gb300 import _C

pytestmark = pytest.mark.gpu


def _sinkhorn(n, d, log_space):
    gen = torch.Generator(device="cuda").manual_seed(d)
    a, b = (torch.rand((n, d), generator=gen, device="cuda") + 0.1 for _ in range(2))
    a, b = a / a.sum(1, keepdim=True), b / b.sum(1, keepdim=True)
    cost = torch.rand((d, d), generator=gen, device="cuda")
    return lambda: _C.sinkhorn_f32_solve(a, b, cost, 0.1, 2, 0.0, log_space)[:2]


def _image(op, shape, **kw):
    x = torch.rand(shape, generator=torch.Generator(device="cuda").manual_seed(shape[-1]), device="cuda")
    return lambda: (op(x, **kw),)


def _edt(shape, sampling=None):
    x = torch.rand(shape, generator=torch.Generator(device="cuda").manual_seed(shape[-1]), device="cuda") < 0.9
    return lambda: (tm.euclidean_distance_transform(x, sampling=sampling),)


CALLS = {  # (smaller, larger) problems of one kernel, both beyond 48 KB of shared memory
    "sinkhorn_clusters": lambda: (_sinkhorn(1, 600, False), _sinkhorn(1, 784, False)),
    "sinkhorn_slabs": lambda: (_sinkhorn(3, 600, True), _sinkhorn(3, 1000, True)),
    "edt_lines": lambda: (_edt((1, 1, 8, 1400)), _edt((1, 1, 8, 2000))),
    "edt_sampled": lambda: (_edt((1, 1, 8, 300), [1.0, 0.7]), _edt((1, 1, 8, 700), [1.0, 0.7])),
    "flat_box": lambda: (_image(tm.grey_dilation, (1, 1, 40, 200), size=17),
                         _image(tm.grey_dilation, (1, 1, 40, 200), size=63)),
    "opening": lambda: (_image(tm.grey_opening, (1, 1, 40, 200), size=9),
                        _image(tm.grey_opening, (1, 1, 40, 200), size=33)),
}


@pytest.mark.parametrize("name", sorted(CALLS))
def test_two_threads_two_sizes(cuda, name):
    calls = CALLS[name]()
    expected = [call() for call in calls]
    torch.cuda.synchronize()
    errors, last = [], [None, None]
    start = threading.Barrier(2)

    def work(k):
        try:
            start.wait()
            for _ in range(400):
                last[k] = calls[k]()
        except Exception as e:  # noqa: BLE001
            errors.append(f"{k}: {e}")

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for got, exp in zip(last, expected):
        assert all(torch.equal(x, y) for x, y in zip(got, exp))
