"""The grouped GEMMs with an expert's tokens on the columns (gemm_moe_narrow.cu, gemm_moe_plain.cu) where a tile, a scale atom or an MMA
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


@pytest.fixture(scope="module", params=["fp8", "fp8 channel", "bf16", "w4a16"])
def plain_table(gw, request):
    """Tables of one kind (FP8 with one input scale for gate and up), as gemm_moe_plain.cu takes them."""
    kind = request.param
    g = torch.Generator(device="cuda").manual_seed(21)
    triples = []
    for e in range(E):
        row = []
        for n, k in ((I, H), (I, H), (H, I)):
            w = (torch.randn((n, k), generator=g, device="cuda") * 0.02).bfloat16()
            scale = (0.004 if k == H else 0.001) * (1 + (e % 4) / 16)
            if kind == "bf16":
                row.append(w)
            elif kind == "w4a16":
                padded = torch.zeros(((n + 127) // 128 * 128, k), dtype=torch.bfloat16, device="cuda")
                padded[:n] = w
                row.append(gw.nvfp4_pack_weights(padded, scale))
            elif kind == "fp8":
                amax = float(w.float().abs().max() / 448)
                row.append(gw.Fp8Weight(gw.fp8_pack_weights(w, amax), 5 * scale, amax))
            else:
                rows = (w.float().abs().amax(dim=1) / 448).contiguous()
                row.append(gw.Fp8Weight(gw.fp8_pack_weights(w, 0.0, rows), 5 * scale, 1.0, (rows * (5 * scale)).contiguous()))
        triples.append(tuple(row))
    table = gw.ExpertTable(triples)
    if kind == "w4a16":
        table.enable_w4a16()
    return kind, table


@pytest.mark.parametrize("tile", [64, 128])
@pytest.mark.parametrize("rows,mode", [(1, "hot"), (15, "hot"), (17, "distributed"), (64, "hot"), (65, "hot"), (128, "hot"), (129, "uneven"), (300, "normal")])
def test_plain_kinds(gw, plain_table, monkeypatch, tile, rows, mode):
    """Against the group-descriptor plan: same operands and K order, so the captures agree to the GEMM gate; after the
    second quantisation (FP8) a last-bit difference may become a step, which the gate covers too."""
    kind, table = plain_table
    x, scores = bf16_normal((rows, H), 400 + rows).cuda(), make_scores(rows, mode, rows).cuda()
    one = torch.ones(E, dtype=torch.bfloat16, device="cuda")
    flags = {"has_fp8": kind.startswith("fp8"), "has_bf16": kind == "bf16", "has_nvfp4": kind == "w4a16", "fp4": False}
    results = {}
    for form in ("narrow", "swap"):
        monkeypatch.setenv("GW_MOE_FORM", form)
        monkeypatch.setenv("GW_MOE_BLOCK_N", str(tile) if form == "narrow" else "32")
        ws = gw.MoeWorkspace(max(64, rows), fp8_experts=kind.startswith("fp8"))
        y = torch.empty((rows, H), dtype=torch.bfloat16, device="cuda")
        ws.run(x, scores, one, table, y, rows, **flags)
        torch.cuda.synchronize()
        assert gw.kernel_error() == 0
        results[form] = [bits(t) for t in (ws.gate_up_capture(), ws.activated_capture(), ws.down_capture(), y)]
    for got, expected, what in zip(results["narrow"], results["swap"], ("gate_up", "activated", "down", "layer")):
        assert_gemm_close(got, expected, f"{kind} {what} rows={rows} {mode} tile={tile}")
