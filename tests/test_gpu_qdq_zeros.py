"""NVFP4 fake quantisation of values that are zeros for a good part (gw_weight_qdq_apply), bit for bit."""
import numpy as np
import pytest
import torch

from oracle import nvfp4 as onv
from tests.gpu_helpers import bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [0.02, 1e-38, 3e38])
@pytest.mark.parametrize("n", [16, 4096 + 16])
def test_zeros_of_both_signs(scale, n):
    import gewell_b200 as gw
    x = torch.randn(n, generator=torch.Generator().manual_seed(n)).mul_(scale / 4).clamp_(-scale, scale).bfloat16()
    x[::3] = 0.0
    x[1::5] = -0.0
    expected = bits(x)
    x = x.cuda()
    for _ in range(2):                       # the second pass sees values that are on the grid already
        gw.weight_qdq_apply(2, x)
        torch.cuda.synchronize()
        expected = onv.qdq(expected)
        assert np.array_equal(bits(x), expected)
