"""The grouped GEMMs with an expert's tokens on the columns (gemm_moe_narrow.cu) where a tile, a scale atom or an MMA
width ends, against the group-descriptor plan (compared with the oracle in test_gpu_moe.py) and against the oracle."""
import numpy as np
import pytest
import torch

from oracle import codecs as C
from oracle import moe as omoe
from tests.gpu_helpers import assert_gemm_close, bf16_normal, bits, to_f32
from tests.test_gpu_moe import E, H, I, experts, experts_shared, gw, make_scores  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [64, 128])
@pytest.mark.parametrize("counts", [
    [1], [15, 16, 17], [31, 32, 33, 47, 48, 49], [63, 64, 65], [127, 128, 129], [0, 0, 191, 0, 192, 193], [255, 256, 257, 1],
    [3] * 128, [0] * 127 + [5], [640] + [1] * 60])
def test_tile_edges(gw, experts_shared, monkeypatch, tile, counts):
    """Same quantised operands and the same K order of the sums: the BF16 results agree to the GEMM gate, the captured
    intermediates too, whichever plan wrote them."""
    table, _ = experts_shared
    counts = counts + [0] * (E - len(counts))
    rows = sum(counts)
    offsets = torch.tensor([0] + list(np.cumsum(counts)), dtype=torch.int32, device="cuda")
    x = bf16_normal((rows, H), 300 + rows).cuda()
    results = {}
    for form in ("narrow", "swap"):
        monkeypatch.setenv("GW_MOE_FORM", form)
        monkeypatch.setenv("GW_MOE_BLOCK_N", str(tile) if form == "narrow" else "32")
        ws = gw.MoeWorkspace(max(64, (rows + 7) // 8))
        y = torch.full((rows * H + 64,), -3.0, dtype=torch.bfloat16, device="cuda")
        ws.run_sorted(x, offsets, 0, E, rows, table, y)
        torch.cuda.synchronize()
        assert gw.kernel_error() == 0
        assert torch.all(y[rows * H:] == -3.0)
        results[form] = [bits(y[:rows * H].reshape(rows, H))] + [bits(ws._alias(pointer, (rows, width), torch.bfloat16)) for pointer, width in (
            (ws._lib.gw_moe_gate_up_capture(ws._ws), 2 * I), (ws._lib.gw_moe_activated_capture(ws._ws), I))]
    for got, expected, what in zip(results["narrow"], results["swap"], ("down", "gate_up", "activated")):
        assert_gemm_close(got, expected, f"{what} tile={tile} counts={counts[:6]}")


@pytest.mark.parametrize("rows,mode,tile", [(1, "hot", 64), (40, "normal", 64), (200, "hot", 64), (200, "hot", 128), (129, "uneven", 128)])
def test_layer_vs_oracle(gw, experts_shared, monkeypatch, rows, mode, tile):
    table, host = experts_shared
    monkeypatch.setenv("GW_MOE_FORM", "narrow")
    monkeypatch.setenv("GW_MOE_BLOCK_N", str(tile))
    x = bf16_normal((rows, H), 200 + rows)
    scores = make_scores(rows, mode, rows)
    ws = gw.MoeWorkspace(max(rows, 64))
    y = torch.empty((rows, H), dtype=torch.bfloat16, device="cuda")
    ws.run(x.cuda(), scores.cuda(), torch.ones(E, dtype=torch.bfloat16, device="cuda"), table, y, rows)
    torch.cuda.synchronize()
    assert gw.kernel_error() == 0
    capture = {}
    expected = omoe.forward(to_f32(x), to_f32(scores), np.ones(E, dtype=np.float32), host, capture=capture, rcp_fn=gw.rcp_approx,
                            gelu_fn=gw.geglu_bf16)
    assert_gemm_close(bits(ws.gate_up_capture()), C.bf16_bits(capture["gate_up"]), "gate/up capture")
    assert_gemm_close(bits(ws.activated_capture()), C.bf16_bits(capture["activated"]), "activated capture")
    assert_gemm_close(bits(ws.down_capture()), C.bf16_bits(capture["down"]), "down capture")
    assert_gemm_close(bits(y), expected, f"MoE rows={rows} {mode} tile={tile}")
