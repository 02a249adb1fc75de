"""How long the FP32 sums of a K loop are.  A row of K begins with a product of +L and ends with one of -L; every product between them
is so small that what one tensor instruction adds to L is lost to rounding, and what a few dozen add up to on their own is not.
So the result tells which share of K was summed apart from its two ends: all of it exactly, none in one accumulator."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gw():
    import gewell_b200
    return gewell_b200


def ends(rows, k, end, between, sign):
    """[rows, k]: `between`, with `end` in front and `sign` * `end` at the back."""
    m = torch.full((rows, k), between, dtype=torch.bfloat16, device="cuda")
    m[:, 0], m[:, -1] = end, sign * end
    return m


def operands(gw, kind, rows, k, n):
    """x, weight and the sum of the small products.  L is 2^25, 448^2 or 2688^2."""
    if kind == "bf16":
        return ends(rows, k, 2.0 ** 12, 2.0 ** -4, 1), ends(n, k, 2.0 ** 13, 1.0, -1), (k - 2) * 2.0 ** -4
    if kind == "fp8":
        data = gw.fp8_pack_weights(ends(n, k, 448.0, 2.0 ** -7, -1), 1.0)
        return ends(rows, k, 448.0, 2.0 ** -6, 1), gw.Fp8Weight(data, 1.0, 1.0), (k - 2) * 2.0 ** -13
    small = 6 * 2.0 ** -7                              # blocks of sixteen equal values are exact; those of the ends hold one value

    def fp4(rows, end, sign):
        m = ends(rows, k, end, small, sign)
        m[:, 1:16] = m[:, -16:-1] = 0
        return m
    weight = gw.nvfp4_pack_weights(fp4(n, 2688.0, -1), 1.0, 1.0)
    return fp4(rows, 2688.0, 1), weight, (k - 32) * small * small


def projected(gw, kind, x, weight, k, n):
    rows = x.shape[0]
    y = torch.empty((rows, n), dtype=torch.bfloat16, device="cuda")
    plan = {"bf16": gw.Bf16Plan, "fp8": gw.Fp8Plan, "w4a4": gw.Nvfp4Plan}[kind](rows, k, n)
    plan.run(x, weight, y, torch.empty(max(256, plan.scratch_bytes()), dtype=torch.uint8, device="cuda"))
    torch.cuda.synchronize()
    assert gw.kernel_error() == 0
    return y.float()


@pytest.mark.parametrize("kind,piece", [("bf16", 64), ("fp8", 128)])
@pytest.mark.parametrize("rows", [1, 8])
def test_streaming_sums_pieces(gw, kind, piece, rows):
    """Weight-streaming kernel, fewer row blocks than half of the SMs: all pieces of 128 bytes of K but the first and the last are
    kept.  A piece is a whole number of units in the last place of L."""
    k, n = 5376, 1024
    x, weight, whole = operands(gw, kind, rows, k, n)
    kept = projected(gw, kind, x, weight, k, n) / whole
    assert kept.min() >= 1 - 2 * piece / k - 2.0 ** -8 and kept.max() <= 1 + 2.0 ** -8, (kept.min(), kept.max())


@pytest.mark.parametrize("rows", [12, 64, 100])
def test_swap_form_split_sums_sixths(gw, rows):
    """42 tiles of NVFP4 channels: three CTAs a tile, and two accumulators in each of them; the four parts between the ends are kept."""
    k, n = 21504, 5376
    x, weight, whole = operands(gw, "w4a4", rows, k, n)
    kept = projected(gw, "w4a4", x, weight, k, n) / whole
    assert kept.min() >= 4 / 6 - 0.03 and kept.max() <= 1.05, (kept.min(), kept.max())


@pytest.mark.parametrize("kind", ["bf16", "fp8"])
@pytest.mark.parametrize("rows,hidden,mlp", [(9, 2816, 2176), (33, 2816, 2176), (64, 5376, 2048), (128, 2816, 384)])
def test_geglu_sums_quarters(gw, kind, rows, hidden, mlp):
    """Gate, up and GeGLU of few rows in one launch: four accumulators, the two middle ones are kept.  Up is 1, so that the product,
    which a BF16 down projection reads, is GeLU of a large gate value: that value."""
    from gewell_b200 import _lib
    x, gate, whole = operands(gw, kind, rows, hidden, mlp)
    one = hidden // 2
    x[:, one] = 1.0
    up = torch.zeros((mlp, hidden), dtype=torch.bfloat16, device="cuda")
    up[:, one] = 1.0
    if kind == "fp8":
        gate.data.view(mlp, hidden)[:, one] = 0
        gate = gw.Fp8Weight(gate.data, 1.0, 2.0 ** 11)
        whole *= 2.0 ** 11
        up = gw.Fp8Weight(gw.fp8_pack_weights(up, 1.0), 1.0, 1.0)
    else:
        gate[:, one] = 0
    down = torch.zeros((hidden, mlp), dtype=torch.bfloat16, device="cuda")
    chain = gw.MlpChain(hidden, mlp, rows, _lib.POLICY_ALWAYS)
    chain.prepare(rows)
    bound = [gw.make_projection(w, i, o) for w, i, o in ((gate, hidden, mlp), (up, hidden, mlp), (down, mlp, hidden))]
    gate_up = torch.empty((rows, 2 * mlp), dtype=torch.bfloat16, device="cuda")
    product, y = torch.empty((rows, mlp), dtype=torch.bfloat16, device="cuda"), torch.empty((rows, hidden), dtype=torch.bfloat16, device="cuda")
    lib = _lib.load()
    _lib.check(lib, lib.gw_mlp_chain_run(chain._chain, *map(ctypes.byref, bound), *(t.data_ptr() for t in (x, gate_up, product, y)),
                                         _lib.PHASE_DECODE, torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert gw.kernel_error() == 0
    kept = product.float() / whole
    assert kept.min() >= 0.45 and kept.max() <= 1.05, (kept.min(), kept.max())
