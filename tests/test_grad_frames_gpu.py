"""Frames of the 3 x 3 / 5 x 5 walkers in the differentiable grey operators: every border mode at
the smallest items the walkers take and around, values and arguments bit-exact and the
gradient against the float64 scatter."""

import numpy as np
import pytest
import torch

import oracle
from tests.helpers import rng
from torchmorph_gb300 import _C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["reflect", "constant", "nearest", "mirror", "wrap"])
@pytest.mark.parametrize("k", [3, 5])
@pytest.mark.parametrize("hw", [(1, 128), (2, 132), (3, 128), (5, 128), (6, 256), (11, 132), (40, 256)])
def test_frames(cuda, mode, k, hw):
    r = rng(hw[0] + k)
    x = r.random((2, 1) + hw).astype(np.float32)
    st, none = torch.zeros(k, k), torch.empty(0, dtype=torch.bool)
    for dilation, fn in ((True, _C.grey_dilation_arg), (False, _C.grey_erosion_arg)):
        out, arg = fn(torch.from_numpy(x).cuda(), st, none, [0, 0], oracle._MODES[mode], 0.4)
        exp_out, exp_arg = oracle.grey_arg(x, st.numpy(), None, (0, 0), mode, 0.4, dilation)
        np.testing.assert_array_equal(out.cpu().numpy(), exp_out)
        np.testing.assert_array_equal(arg.cpu().numpy(), exp_arg)
        g = r.standard_normal(x.shape).astype(np.float32)
        gin = _C.grey_morphology_backward(torch.from_numpy(g).cuda(), arg, [k, k], none, [0, 0], oracle._MODES[mode],
                                          dilation)
        exp = oracle.grey_backward(g, exp_arg, (k, k), None, (0, 0), mode, dilation)
        # an fp32 sum of n gradients of size <= 5: n^2 2^-24 5; n < 30 but where a short mirrored
        # or clamped axis gathers a whole footprint
        np.testing.assert_allclose(gin.cpu().numpy(), exp, rtol=2e-5, atol=3e-4)
