"""NVFP4 projections of more than 128 rows whose K loop several CTA pairs share (gemm_pair.cu), against the single-CTA kernel
(GW_DENSE_NO_PAIR), which test_gpu_linear.py compares with the oracle."""
import pytest
import torch

from tests.gpu_helpers import assert_gemm_close, assert_reference_tolerance, bf16_normal, bits

pytestmark = pytest.mark.gpu

# test_dense_routes.py asserts that all of them share K
SHARED = [(129, 16448, 128), (255, 8256, 384), (257, 12352, 2560), (256, 21504, 5376), (512, 16384, 4096),
          (513, 8256, 2816), (33, 8192, 128), (64, 12288, 2816), (65, 8192, 128), (128, 16448, 4608), (100, 8256, 2816)]


@pytest.mark.parametrize("rows,k,n", SHARED)
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
    assert_reference_tolerance(results[0], results[1], f"{rows}x{k}x{n}")       # a last bit of a value


def test_one_plan_on_both_routes():
    """65 to 128 rows: an output that is not 16-byte aligned keeps the call on the other kernel, whose tensor maps have other boxes."""
    import gewell_b200 as gw
    rows, k, n = 100, 8192, 256
    weight = gw.nvfp4_pack_weights((bf16_normal((n, k), 1) * 0.02).cuda(), 6 / 2688)
    x = bf16_normal((rows, k), 2).cuda()
    plan = gw.Nvfp4Plan(rows, k, n)
    scratch = torch.empty(plan.scratch_bytes(), dtype=torch.uint8, device="cuda")
    y = torch.zeros(rows * n + 8, dtype=torch.bfloat16, device="cuda")
    results = []
    for offset in (0, 1, 0, 1):
        y.fill_(float("nan"))
        plan.run(x, weight, y[offset:offset + rows * n], scratch)
        torch.cuda.synchronize()
        assert gw.kernel_error() == 0
        results.append(bits(y[offset:offset + rows * n]))
    for got in results[1:]:
        assert_gemm_close(got, results[0])


def test_one_chain_with_dequantised_and_bound_weights():
    """40 rows: BF16 weights take the CTA pairs, weights just dequantised of more than L2 holds the swap form, through the same plan."""
    import gewell_b200 as gw
    from gewell_b200 import _lib
    rows, hidden, mlp = 40, 5376, 12544
    weights = [(bf16_normal(s, 3 + i) * 0.02).cuda() for i, s in enumerate([(mlp, hidden), (mlp, hidden), (hidden, mlp)])]
    shapes = [(hidden, mlp), (hidden, mlp), (mlp, hidden)]
    packed = [gw.nvfp4_pack_weights(w, 6 / 2688) for w in weights]
    bound = {storage: [gw.make_projection(w, *s) for w, s in zip(of, shapes)] for storage, of in (("bf16", weights), ("nvfp4", packed))}
    x = bf16_normal((rows, hidden), 9).cuda()

    def run(chain, storage):
        y = chain.run(*bound[storage], x, _lib.PHASE_DECODE)
        torch.cuda.synchronize()
        assert gw.kernel_error() == 0
        return bits(y)

    def fresh():
        chain = gw.MlpChain(hidden, mlp, rows, _lib.POLICY_PREFILL)
        chain.prepare(rows)
        return chain

    both = fresh()
    for storage in ("bf16", "nvfp4", "bf16", "nvfp4"):
        assert_gemm_close(run(both, storage), run(fresh(), storage), storage)
