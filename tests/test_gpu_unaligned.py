"""NVFP4 projections into an output that is only 2-byte aligned: beyond 128 rows the swap form, with several token tiles."""
import pytest
import torch

from tests.gpu_helpers import assert_gemm_close, bf16_normal, bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,k,n", [(128, 640, 128), (129, 640, 256), (256, 256, 384), (300, 2816, 2816), (513, 192, 128)])
def test_unaligned_output(rows, k, n):
    """Against the same plan's aligned result (compared with the oracle in test_gpu_linear.py); nothing beside the output is written."""
    import gewell_b200 as gw
    weight = gw.nvfp4_pack_weights((bf16_normal((n, k), 1) * 0.02).cuda(), 6 / 2688)
    x = bf16_normal((rows, k), 2).cuda()
    plan = gw.Nvfp4Plan(rows, k, n)
    scratch = torch.empty(plan.scratch_bytes(), dtype=torch.uint8, device="cuda")
    y = torch.empty(rows * n + 16, dtype=torch.bfloat16, device="cuda")
    results = []
    for offset in (0, 1, 0, 7):
        y.fill_(-7.0)
        plan.run(x, weight, y[offset:offset + rows * n], scratch)
        torch.cuda.synchronize()
        assert gw.kernel_error() == 0
        assert torch.all(y[:offset] == -7.0) and torch.all(y[offset + rows * n:] == -7.0)
        results.append(bits(y[offset:offset + rows * n].reshape(rows, n)))
    for got in results[1:]:
        assert_gemm_close(got, results[0], f"{rows}x{k}x{n}")
