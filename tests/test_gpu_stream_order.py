"""What one call writes, the next call on the stream reads, also where it takes it as a weight: weight matrices, norm
vectors, the layer scalar and expert scales made by the framework's own kernels directly, or one launch, before their use.
The values alternate between two sets, so that a stale read gives the other set's result."""
import pytest
import torch

from tests.gpu_helpers import bf16_normal
from tests.test_gpu_moe import experts, experts_shared  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu

H = 2816
LARGE = 48 << 20           # elements of the tensor whose end is the weight: its writer runs for tens of microseconds
REPEATS = 12


@pytest.fixture(scope="module")
def gw():
    import gewell_b200
    return gewell_b200


def alternate(write, read, between=None):
    """write(i) produces the weight of set i, read() returns clones of what uses it."""
    expected = []
    for i in (0, 1):
        write(i)
        torch.cuda.synchronize()
        expected.append([t.clone() for t in read()])
        torch.cuda.synchronize()
    assert not all(torch.equal(a, b) for a, b in zip(*expected))
    results = []
    for i in range(REPEATS):
        write(i % 2)
        if between is not None:
            between()
        results.append([t.clone() for t in read()])
    torch.cuda.synchronize()
    for i, got in enumerate(results):
        for a, b in zip(got, expected[i % 2]):
            assert torch.equal(a, b), f"repeat {i}"


@pytest.fixture(scope="module")
def halves():
    """Addends of a large tensor; the sum with either of two deltas is the weight."""
    base = torch.randn(LARGE, device="cuda", dtype=torch.bfloat16) * 0.02
    return base, [torch.randn(LARGE, device="cuda", dtype=torch.bfloat16) * 0.02 for _ in (0, 1)], torch.empty_like(base)


def other_launch(gw):
    small = torch.ones(64, dtype=torch.bfloat16, device="cuda")
    return lambda: gw.add_bf16(small, small)


@pytest.mark.parametrize("one_between", [False, True])
@pytest.mark.parametrize("rows,k,n", [(1, H, H), (8, H, 4096), (8, H, 16384), (64, 5376, 2048)])
def test_add_then_bf16_projection(gw, halves, rows, k, n, one_between):
    """Streaming and swap-form projections over a weight that add has just written."""
    base, delta, out = halves
    weight = out[-n * k:].view(n, k)
    x = bf16_normal((rows, k), 1).cuda()
    plan = gw.Bf16Plan(rows, k, n)
    scratch = torch.empty(max(plan.scratch_bytes(), 256), dtype=torch.uint8, device="cuda")
    y = torch.empty((rows, n), dtype=torch.bfloat16, device="cuda")

    def read():
        plan.run(x, weight, y, scratch)
        return [y]
    alternate(lambda i: gw.add_bf16(base, delta[i], out), read, other_launch(gw) if one_between else None)
    assert gw.kernel_error() == 0


@pytest.mark.parametrize("writer", ["gemm", "geglu", "norm"])
def test_projection_over_another_kernels_output(gw, writer):
    """The direct predecessor -- a GEMM, GeGLU, a norm -- wrote the weight matrix."""
    rows, k, n = 8, H, 4096
    parts = [(bf16_normal((n, k), 10 + i, 0.1).cuda(), bf16_normal((n, k), 20 + i).cuda()) for i in (0, 1)]
    square = bf16_normal((k, k), 30, 0.02).cuda()
    made = gw.Bf16Plan(n, k, k)
    room = torch.empty(max(made.scratch_bytes(), 256), dtype=torch.uint8, device="cuda")
    weight = torch.empty((n, k), dtype=torch.bfloat16, device="cuda")
    x = bf16_normal((rows, k), 2).cuda()
    plan = gw.Bf16Plan(rows, k, n)
    scratch = torch.empty(max(plan.scratch_bytes(), 256), dtype=torch.uint8, device="cuda")
    y = torch.empty((rows, n), dtype=torch.bfloat16, device="cuda")
    from gewell_b200 import _lib
    library = _lib.load()

    def write(i):
        gate, up = parts[i]
        if writer == "gemm":
            made.run(gate, square, weight, room)
        elif writer == "norm":
            gw.rms_norm(gate, None, weight)
        else:
            _lib.check(library, library.gw_gelu_tanh_multiply_bf16(gate.data_ptr(), up.data_ptr(), weight.data_ptr(), n * k,
                                                                    torch.cuda.current_stream().cuda_stream))

    def read():
        plan.run(x, weight, y, scratch)
        return [y]
    alternate(write, read)
    assert gw.kernel_error() == 0


@pytest.mark.parametrize("rows,n", [(1, 2816), (8, 8192)])
def test_projection_over_rows_the_quantiser_has_packed(gw, rows, n):
    """Activation quantisation writes the layout of packed weights; its output as the weight of the next call."""
    k, scale = H, 0.01
    values = [bf16_normal((n, k), 40 + i, 0.05).cuda() for i in (0, 1)]
    packed, scales = gw.nvfp4_quantize_activations(values[0], scale)
    x = bf16_normal((rows, k), 3).cuda()
    plan = gw.Nvfp4Plan(rows, k, n)
    scratch = torch.empty(plan.scratch_bytes(), dtype=torch.uint8, device="cuda")
    y = torch.empty((rows, n), dtype=torch.bfloat16, device="cuda")
    from gewell_b200 import _lib
    library = _lib.load()

    def write(i):
        _lib.check(library, library.gw_nvfp4_quantize_activations(values[i].data_ptr(), n, k, scale, 0, packed.data_ptr(),
                                                                   scales.data_ptr(), torch.cuda.current_stream().cuda_stream))

    def read():
        plan.run(x, gw.Nvfp4Weight(packed, scales, 0.01, scale), y, scratch)
        return [y]
    alternate(write, read)
    assert gw.kernel_error() == 0


@pytest.mark.parametrize("one_between", [False, True])
def test_norm_weights_and_layer_scalar(gw, halves, one_between):
    base, delta, out = halves
    w = [out[LARGE - (i + 1) * H:LARGE - i * H] for i in range(3)]
    scalar = out[LARGE - 3 * H - 8:][:1]
    x, hidden = bf16_normal((16, H), 4).cuda(), bf16_normal((16, H), 5).cuda()

    def read():
        return [gw.rms_norm(x, w[0])]

    def read_three():
        return list(gw.rms_norm_feedforward(x, *w))

    def read_tail():
        return [gw.ffn_tail(x, x, w[0], w[1], w[2], scalar, hidden.clone())]
    between = other_launch(gw) if one_between else None
    for reader in (read, read_three):
        alternate(lambda i: gw.add_bf16(base, delta[i], out), reader, between)
    target = hidden.clone()                       # the clone above is a launch of its own; here nothing comes between

    def read_tail_in_place():
        return [gw.ffn_tail(x, x, w[0], w[1], w[2], scalar, target)]

    def write(i):
        target.copy_(hidden)
        gw.add_bf16(base, delta[i], out)
    alternate(write, read_tail_in_place, between)
    alternate(lambda i: gw.add_bf16(base, delta[i], out), read_tail, between)


def test_scale_in_place_then_norm(gw):
    big = torch.ones(LARGE, dtype=torch.bfloat16, device="cuda")
    weight = big[-H:]
    x = bf16_normal((4, H), 6).cuda()
    factor = [torch.tensor([f], dtype=torch.bfloat16, device="cuda") for f in (2.0, 0.5)]
    alternate(lambda i: gw.scale_bf16(big, factor[i]), lambda: [gw.rms_norm(x, weight)])


@pytest.mark.parametrize("rows", [7, 64, 300])
def test_expert_scales(gw, halves, experts_shared, rows):
    """Routing weights are the renormalised probabilities times the scales."""
    base, delta, out = halves
    table, _ = experts_shared
    scales = out[LARGE - 128:]
    x, scores = bf16_normal((rows, H), 7).cuda(), bf16_normal((rows, 128), 8).cuda()
    ws = gw.MoeWorkspace(rows)
    y = torch.empty((rows, H), dtype=torch.bfloat16, device="cuda")

    def read():
        ws.run(x, scores, scales, table, y, rows, has_nvfp4=True, fp4=True)
        return [y]
    alternate(lambda i: gw.add_bf16(base, delta[i], out), read)
    assert gw.kernel_error() == 0


@pytest.mark.parametrize("rows", [1, 8, 64])
def test_mlp_chain_over_weights_just_written(gw, rows):
    """The chain's first projection takes BF16 weights that add wrote; its later ones those of the sum before."""
    from gewell_b200 import _lib
    hidden, mlp = 1408, 4096
    base = bf16_normal((3 * mlp * hidden,), 9, 0.02).cuda()
    delta = [bf16_normal((3 * mlp * hidden,), 50 + i, 0.02).cuda() for i in (0, 1)]
    out = torch.empty_like(base)
    parts = [out[i * mlp * hidden:(i + 1) * mlp * hidden] for i in range(3)]
    bound = [gw.make_projection(p.view(o, i), i, o) for p, i, o in
             ((parts[0], hidden, mlp), (parts[1], hidden, mlp), (parts[2], mlp, hidden))]
    chain = gw.MlpChain(hidden, mlp, 64, _lib.POLICY_ALWAYS)
    chain.prepare(rows)
    x = bf16_normal((rows, hidden), 11).cuda()
    alternate(lambda i: gw.add_bf16(base, delta[i], out), lambda: [chain.run(*bound, x, _lib.PHASE_DECODE)])
    assert gw.kernel_error() == 0
