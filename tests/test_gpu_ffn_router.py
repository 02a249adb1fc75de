"""Router logits of the feed-forward block around the last row count of their own kernel (128), element by element."""
import pytest
import torch

from tests.gpu_helpers import bf16_normal
from tests.test_gpu_ffn_block import H, block_layer
from tests.test_gpu_moe import experts, experts_shared, gw  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 7, 9, 127, 128, 129])
def test_router_logits(gw, experts_shared, rows):
    """Half a BF16 unit of the exact logit, and what 2816 FP32 additions of the magnitudes' sum can lose."""
    from gewell_b200 import _lib
    layer = block_layer(gw, experts_shared[0], "bf16", 11)
    block = gw.FfnBlock([layer], max(rows, 64), _lib.POLICY_ALWAYS)
    block.prepare(rows, _lib.PHASE_DECODE)
    block.run(0, bf16_normal((rows, H), 90 + rows, 2.0).cuda())
    torch.cuda.synchronize()
    assert gw.kernel_error() == 0
    x, w = block.buffer("router_input").double(), layer["router_proj"].double()
    exact, magnitudes = x @ w.T, x.abs() @ w.abs().T
    error = (block.buffer("router_logits").double() - exact).abs()
    assert torch.all(error <= exact.abs() * 2.0 ** -8 + magnitudes * (H * 2.0 ** -24))
