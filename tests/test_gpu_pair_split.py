"""NVFP4 projections of more than 128 rows whose K loop several CTA pairs share (gemm_pair.cu), against the single-CTA kernel
(GW_DENSE_NO_PAIR), which test_gpu_linear.py compares with the oracle."""
import pytest
import torch

from tests.gpu_helpers import assert_gemm_close, bf16_normal, bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,k,n", [(129, 16448, 128), (255, 8256, 384), (257, 12352, 2560), (256, 21504, 5376), (512, 16384, 4096),
                                      (513, 8256, 2816), (65, 8192, 128), (128, 16448, 4608), (100, 8256, 2816)])
def test_shared_k(monkeypatch, rows, k, n):
    """K over two to four pairs (of 148 SMs); tokens and channels that end within a tile, K that ends within a stage."""
    import gewell_b200 as gw
    weight = gw.nvfp4_pack_weights((bf16_normal((n, k), 1) * 0.02).cuda(), 6 / 2688)
    x = bf16_normal((rows, k), 2).cuda()
    results = []
    for apart in (False, True):
        if apart:
            monkeypatch.setenv("GW_DENSE_NO_PAIR", "1")
        else:
            monkeypatch.delenv("GW_DENSE_NO_PAIR", raising=False)
        plan = gw.Nvfp4Plan(rows, k, n)
        scratch = torch.empty(plan.scratch_bytes(), dtype=torch.uint8, device="cuda")
        y = torch.full((rows * n + 64,), -7.0, dtype=torch.bfloat16, device="cuda")
        y[:-64] = float("nan")
        plan.run(x, weight, y, scratch)
        torch.cuda.synchronize()
        assert gw.kernel_error() == 0 and torch.all(y[-64:] == -7.0)
        results.append(bits(y[:-64]))
    assert_gemm_close(results[0], results[1], f"{rows}x{k}x{n}")
