"""FP8 and BF16 projections of more than 128 rows (gemm_pair_wide.cu) at the edges of their tiles: rows around the
token tile, a last tile of one token, channels that fill part of a pair, K of less than one slab and of a ragged one."""
import numpy as np
import pytest
import torch

from oracle import codecs as C
from oracle import fp8 as ofp8
from tests.gpu_helpers import assert_gemm_close, bf16_normal, bits, to_f32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["fp8", "fp8 per channel", "bf16"])
@pytest.mark.parametrize("rows,k,n", [(129, 16, 16), (161, 144, 272), (256, 2832, 512), (257, 128, 20000), (1025, 656, 2064), (2400, 80, 784)])
def test_pair(kind, rows, k, n):
    import gewell_b200 as gw
    values, x = bf16_normal((n, k), 5, 0.02), bf16_normal((rows, k), 6)
    if kind == "bf16":
        plan, weight = gw.Bf16Plan(rows, k, n), values.cuda()
        want = C.bf16_bits(to_f32(x) @ to_f32(values).T)
    else:
        w = (ofp8.pack_weights_per_channel if "channel" in kind else ofp8.pack_weights)(to_f32(values), 0.01)
        scales = torch.from_numpy(w.channel_scales.copy()).cuda() if "channel" in kind else None
        plan = gw.Fp8Plan(rows, k, n, "channel" in kind)
        weight = gw.Fp8Weight(torch.from_numpy(w.data.copy()).cuda(), w.input_scale, w.weight_scale, scales)
        want = ofp8.linear_w8a8(to_f32(x), w)
    y = torch.full((rows * n + 64,), -7.0, dtype=torch.bfloat16, device="cuda")
    y[:-64] = float("nan")
    scratch = torch.empty(max(plan.scratch_bytes(), 256), dtype=torch.uint8, device="cuda")
    plan.run(x.cuda(), weight, y, scratch)
    torch.cuda.synchronize()
    assert gw.kernel_error() == 0 and torch.all(y[-64:] == -7.0)
    assert_gemm_close(bits(y[:-64]).reshape(rows, n), want, f"{kind} rows={rows} K={k} N={n}")


@pytest.mark.parametrize("kind", ["fp8", "bf16"])
@pytest.mark.parametrize("rows,n", [(250, 19456), (200, 28160), (256, 43008), (300, 19216)])
def test_last_wave_in_pieces(kind, rows, n):
    """Tiles behind the last whole wave (of 148 SMs), cut into eight, two, three and five pieces; the last pieces are cut short or empty."""
    test_pair(kind, rows, 80, n)


@pytest.mark.parametrize("kind,rows,k,n", [("fp8", 131, 8208, 272), ("bf16", 257, 4104, 768), ("fp8 per channel", 218, 8208, 5136),
                                           ("bf16", 300, 4104, 2576), ("fp8", 700, 8208, 272), ("bf16", 140, 4104, 8080)])
def test_shared_k(kind, rows, k, n):
    """K over four, four, three, three, three and two pairs (of 148 SMs); channels and tokens that end within a tile."""
    test_pair(kind, rows, k, n)


# test_dense_routes.py asserts that all of them run on the CTA pairs
FEW_ROWS = [("fp8", 33, 4112, 272), ("fp8", 65, 80, 784), ("fp8 per channel", 128, 8208, 5376), ("bf16", 33, 16, 16),
            ("bf16", 64, 2056, 6128), ("bf16", 97, 72, 9360), ("bf16", 128, 4104, 2816)]


@pytest.mark.parametrize("kind,rows,k,n", FEW_ROWS)
def test_few_rows(kind, rows, k, n):
    """One wave of tiles for at most 128 rows: one slab of K (one accumulator) and many, one pair to a tile and several."""
    test_pair(kind, rows, k, n)
