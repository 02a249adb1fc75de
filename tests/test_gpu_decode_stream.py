"""The weight-streaming projections of small row counts (decode_stream.cu) at the edges of their division of the work:
K of one partial chunk, a chunk, whole and ragged slabs; row blocks shared by warps and by SMs; one group of eight tokens, and
two for W4A16; two matrices with GeGLU; W4A16 over several launches.  Row counts above the kernel's (8; W4A16: 32) and shapes
where it does not pay run on the kernels beside it."""
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
    """Gate and up with scales of their own: one launch with GeGLU for up to eight rows (W4A16: sixteen a launch, up to 32
    rows), projections one by one beyond."""
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


@pytest.mark.parametrize("rows", [32, 33])
def test_w4a16_last_streamed_rows(gw, rows):
    """Two launches of the packed weights, and the first row count that dequantises them."""
    test_nvfp4_pair_and_w4a16(gw, rows, 640, 1408, "prefill")


@pytest.mark.parametrize("rows,k,n", [(1, 8192, 2048), (1, 8448, 2048), (4, 3072, 2816), (4, 3136, 2816), (8, 1088, 256)])
@pytest.mark.parametrize("storage", ["nvfp4", "fp8"])
def test_geglu_inputs_around_their_limit(gw, storage, rows, k, n):
    """A plan that streams plain inputs hands GeGLU inputs above a size to the quantiser and the tensor-core kernel; the two
    take turns on one plan and its scratch, whose counters have to come back to zero."""
    x, gate_up = bf16_normal((rows, k), 61), bf16_normal((rows, 2 * k), 62)
    values = to_f32(bf16_normal((n, k), 63, 0.02))
    if storage == "nvfp4":
        w = onv.pack_weights(values, 0.01)
        dev, plan, linear = oracle_weight_to_device(w), gw.Nvfp4Plan(rows, k, n), lambda a: onv.linear_w4a4(a, w, rcp_fn=gw.rcp_approx)
    else:
        w = ofp8.pack_weights(values, 0.01)
        dev = gw.Fp8Weight(torch.from_numpy(w.data.copy()).cuda(), w.input_scale, w.weight_scale)
        plan, linear = gw.Fp8Plan(rows, k, n), lambda a: ofp8.linear_w8a8(a, w)
    scratch = torch.full((plan.scratch_bytes(),), 0xCD, dtype=torch.uint8, device="cuda")
    product = gw.geglu_bf16(to_f32(gate_up[:, :k]), to_f32(gate_up[:, k:]))
    for _ in range(2):
        for source, transform, expected in ((x, gw.TRANSFORM_IDENTITY, linear(to_f32(x))),
                                            (gate_up, gw.TRANSFORM_GELU_TANH_MULTIPLY, linear(product))):
            y = torch.full((rows, n), float("nan"), dtype=torch.bfloat16, device="cuda")
            plan.run(source.cuda(), dev, y, scratch, transform=transform)
            torch.cuda.synchronize()
            assert gw.kernel_error() == 0
            assert_gemm_close(bits(y), expected, f"{storage} rows={rows} K={k} N={n} transform={transform}")


@pytest.mark.parametrize("rows", [1, 16, 32, 33, 64])
def test_w4a16_arithmetic(gw, rows):
    """Up to 32 rows the products of exact weights, beyond of weights rounded to BF16; each against the FP64 sum over its own
    operands: one BF16 rounding (2^-8 relative) and FP32 sums of K terms ((K + 4) 2^-24 of the magnitudes' sum).  Sums that
    cancel tell the two apart."""
    from gewell_b200 import _lib
    k, n = 1408, 640
    w = onv.pack_weights(to_f32(bf16_normal((n, k), 71, 0.02)))
    x = bf16_normal((rows, k), 72)
    dev = oracle_weight_to_device(w)
    p = gw.make_projection(dev, k, n)
    ws = gw.ProjectionWorkspace([p], 64, _lib.POLICY_PREFILL)
    ws.prepare(rows, _lib.PHASE_DECODE)
    y = torch.empty((rows, n), dtype=torch.bfloat16, device="cuda")
    ws.run(p, x.cuda(), y)
    torch.cuda.synchronize()
    assert gw.kernel_error() == 0
    values, scales = onv.decoded_weight_values(w)
    unrounded = (values.reshape(n, -1, 16).astype(np.float64) * scales.astype(np.float64)[:, :, None]).reshape(n, k) * float(w.weight_scale)
    rounded = C.bf16_to_f32(onv.dequantize(w)).astype(np.float64)
    a, got = to_f32(x).astype(np.float64), to_f32(y).astype(np.float64)

    def outside(weights):
        reference = a @ weights.T
        bound = 2.0 ** -8 * np.abs(reference) + (k + 4) * 2.0 ** -24 * (np.abs(a) @ np.abs(weights).T)
        return int((np.abs(got - reference) > bound).sum())
    own, other = (unrounded, rounded) if rows <= 32 else (rounded, unrounded)
    assert outside(own) == 0
    assert outside(other) > 0
