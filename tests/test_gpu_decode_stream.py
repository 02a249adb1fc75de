"""The weight-streaming projections of small row counts (decode_stream.cu) at the edges of their division of the work:
K of one partial chunk, a chunk, whole and ragged slabs; row blocks shared by warps and by SMs; one and two token
groups; two matrices with GeGLU; W4A16 over several launches."""
import numpy as np
import pytest
import torch

from oracle import codecs as C
from oracle import fp8 as ofp8
from oracle import nvfp4 as onv
from tests.gpu_helpers import assert_gemm_close, bf16_normal, bits, device_weight_to_oracle, oracle_weight_to_device, to_f32

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gw():
    import gewell_b200
    return gewell_b200


def run(gw, plan, x, weight, n):
    need = plan.scratch_bytes()
    scratch = torch.full((need + 256,), 0xCD, dtype=torch.uint8, device="cuda")
    y = torch.full((x.shape[0] * n + 64,), -7.0, dtype=torch.bfloat16, device="cuda")
    results = []
    for _ in range(2):                       # the counters must come back to zero, the bits must repeat
        y[:-64] = float("nan")
        plan.run(x.cuda(), weight, y, scratch[:need])
        torch.cuda.synchronize()
        assert gw.kernel_error() == 0
        results.append(bits(y[:-64]).reshape(x.shape[0], n).copy())
    assert np.array_equal(*results) and torch.all(y[-64:] == -7.0) and torch.all(scratch[need:] == 0xCD)
    return results[0]


@pytest.mark.parametrize("rows", [1, 8, 9, 16])
@pytest.mark.parametrize("k,n", [(64, 128), (320, 384), (2816, 2816), (3392, 640), (21504, 256)])
def test_nvfp4(gw, rows, k, n):
    w = onv.pack_weights(to_f32(bf16_normal((n, k), 3, 0.02)), 0.01)
    x = bf16_normal((rows, k), 4 + rows)
    y = run(gw, gw.Nvfp4Plan(rows, k, n), x, oracle_weight_to_device(w), n)
    assert_gemm_close(y, onv.linear_w4a4(to_f32(x), w, rcp_fn=gw.rcp_approx), f"NVFP4 rows={rows} K={k} N={n}")


@pytest.mark.parametrize("rows", [1, 8, 9, 16])
@pytest.mark.parametrize("k,n,channel", [(16, 32, False), (144, 96, True), (2832, 1056, False), (5376, 4096, True), (16384, 128, False)])
def test_fp8(gw, rows, k, n, channel):
    values = to_f32(bf16_normal((n, k), 5, 0.02))
    w = ofp8.pack_weights_per_channel(values, 0.01) if channel else ofp8.pack_weights(values, 0.01)
    scales = torch.from_numpy(w.channel_scales.copy()).cuda() if channel else None
    dev = gw.Fp8Weight(torch.from_numpy(w.data.copy()).cuda(), w.input_scale, w.weight_scale, scales)
    x = bf16_normal((rows, k), 6 + rows)
    y = run(gw, gw.Fp8Plan(rows, k, n, channel), x, dev, n)
    assert_gemm_close(y, ofp8.linear_w8a8(to_f32(x), w), f"FP8 rows={rows} K={k} N={n}")


@pytest.mark.parametrize("rows", [1, 8, 13])
@pytest.mark.parametrize("k,n", [(16, 32), (80, 160), (2816, 704), (8192, 384)])
def test_bf16(gw, rows, k, n):
    w, x = bf16_normal((n, k), 7, 0.02), bf16_normal((rows, k), 8 + rows)
    y = run(gw, gw.Bf16Plan(rows, k, n), x, w.cuda(), n)
    assert_gemm_close(y, C.bf16_bits(to_f32(x) @ to_f32(w).T), f"BF16 rows={rows} K={k} N={n}")


@pytest.mark.parametrize("rows", [1, 8, 16, 17, 48, 49])
@pytest.mark.parametrize("hidden,mlp", [(128, 128), (640, 1408)])
@pytest.mark.parametrize("policy", ["always", "prefill"])
def test_nvfp4_pair_and_w4a16(gw, rows, hidden, mlp, policy):
    """Gate and up with scales of their own (one launch with GeGLU up to 16 rows), W4A16 up to 48 rows and beyond."""
    from gewell_b200 import _lib
    gate, up = (gw.nvfp4_pack_weights(bf16_normal((mlp, hidden), s, 0.05).cuda(), 0.002) for s in (1, 2))
    down = gw.nvfp4_pack_weights(bf16_normal((hidden, mlp), 3, 0.05).cuda(), 0.004)
    x = bf16_normal((rows, hidden), 4)
    chain = gw.MlpChain(hidden, mlp, 64, getattr(_lib, "POLICY_" + policy.upper()))
    chain.prepare(rows)
    bound = [gw.make_projection(w, i, o) for w, i, o in ((gate, hidden, mlp), (up, hidden, mlp), (down, mlp, hidden))]
    y = bits(chain.run(*bound, x.cuda(), _lib.PHASE_DECODE))
    assert np.array_equal(y, bits(chain.run(*bound, x.cuda(), _lib.PHASE_DECODE))) and gw.kernel_error() == 0
    hg, hu, hd = (device_weight_to_oracle(w, n, k) for w, n, k in ((gate, mlp, hidden), (up, mlp, hidden), (down, hidden, mlp)))
    if policy == "always":
        g, u = (C.bf16_to_f32(onv.linear_w4a4(to_f32(x), h, rcp_fn=gw.rcp_approx)) for h in (hg, hu))
        expected = onv.linear_w4a4(gw.geglu_bf16(g, u), hd, rcp_fn=gw.rcp_approx)
    else:
        g, u = (C.bf16_to_f32(onv.linear_w4a16(to_f32(x), h)) for h in (hg, hu))
        expected = onv.linear_w4a16(C.gelu_tanh_multiply_bf16(g, u), hd)
    assert_gemm_close(y, expected, f"chain rows={rows} {hidden}/{mlp} {policy}")
