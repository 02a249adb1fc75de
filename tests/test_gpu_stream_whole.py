"""The weight-streaming kernel where some SMs have one row block more than others, and where a row block does not feed
a block's warps, against the tcgen05 swap form."""
import pytest
import torch

from tests.gpu_helpers import assert_gemm_close, assert_reference_tolerance, bf16_normal, bits

pytestmark = pytest.mark.gpu

# test_dense_routes.py asserts that all of them stream
SHAPES = [(1, 64, 4736), (1, 64, 4864), (5, 576, 19072), (8, 256, 128), (1, 5376, 23552)]
STREAMED = {"nvfp4": SHAPES + [(2, 1024, 9472), (2, 2816, 4864)], "fp8": SHAPES + [(2, 1024, 9600), (8, 2816, 4864)],
            "bf16": SHAPES + [(2, 1024, 9600), (8, 2816, 4864)]}


@pytest.mark.parametrize("storage,rows,k,n", [(storage, *shape) for storage, shapes in STREAMED.items() for shape in shapes])
def test_uneven_row_blocks(monkeypatch, storage, rows, k, n):
    import gewell_b200 as gw
    x, w = bf16_normal((rows, k), rows + k).cuda(), (bf16_normal((n, k), n) * 0.02).cuda()
    if storage == "nvfp4":
        weight, make = gw.nvfp4_pack_weights(w, 6 / 2688), gw.Nvfp4Plan
    elif storage == "fp8":
        scale = float(w.float().abs().max() / 448)
        weight, make = gw.Fp8Weight(gw.fp8_pack_weights(w, scale), 6 / 448, scale), gw.Fp8Plan
    else:
        weight, make = w, gw.Bf16Plan
    results = []
    for form in (None, "s"):
        monkeypatch.delenv("GW_DENSE_FORM", raising=False)
        if form:
            monkeypatch.setenv("GW_DENSE_FORM", form)
        plan = make(rows, k, n)
        y = torch.full((rows * n + 64,), -3.0, dtype=torch.bfloat16, device="cuda")
        for _ in range(2):
            plan.run(x, weight, y, torch.empty(max(256, plan.scratch_bytes()), dtype=torch.uint8, device="cuda"))
        torch.cuda.synchronize()
        assert gw.kernel_error() == 0
        assert torch.all(y[rows * n:] == -3.0)
        results.append(bits(y[:rows * n].reshape(rows, n)))
    assert_gemm_close(results[0], results[1], f"{storage} {rows}x{k}x{n}")
    assert_reference_tolerance(results[0], results[1], f"{storage} {rows}x{k}x{n}")       # a last bit of a value
