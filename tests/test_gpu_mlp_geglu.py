"""Gate, up and GeGLU in one prefill launch of the MLP chain, where a tile of tokens or channels ends, against the chain of
separate launches (GW_DENSE_NO_PAIR keeps the pair kernels out), which test_gpu_mlp_chain.py compares with the oracle."""
import pytest
import torch

from tests.gpu_helpers import assert_gemm_close, bf16_normal, bits

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gw():
    import gewell_b200
    return gewell_b200


def projections(gw, storage, hidden, mlp, joined):
    both = (bf16_normal((2 * mlp, hidden), 1) * 0.02).cuda()
    down = (bf16_normal((hidden, mlp), 2) * 0.02).cuda()
    gate, up = (both[:mlp], both[mlp:]) if joined else (both[:mlp].clone(), both[mlp:].clone())

    def fp8(w, input_scale, channel):
        rows = (w.float().abs().amax(dim=1) / 448).contiguous()
        if channel is not None:
            return gw.Fp8Weight(gw.fp8_pack_weights(w, 0.0, rows), input_scale, 1.0, (rows * input_scale).contiguous())
        return gw.Fp8Weight(gw.fp8_pack_weights(w, float(rows.max())), input_scale, float(rows.max()))

    if storage == "bf16":
        return gate, up, down
    if storage == "bf16 fp8":
        return gate, up, fp8(down, 16 / 448, None)
    if storage == "fp8":
        return fp8(gate.contiguous(), 6 / 448, None), fp8(up.contiguous(), 6 / 448, None), fp8(down, 16 / 448, None)
    if storage in ("fp8 channel", "fp8 bf16"):
        rows = (both.float().abs().amax(dim=1) / 448).contiguous()
        scales = (rows * (6 / 448)).contiguous()
        data = gw.fp8_pack_weights(both, 0.0, rows)
        pair = [gw.Fp8Weight(data[s], 6 / 448, 1.0, scales[s]) for s in (slice(0, mlp), slice(mlp, 2 * mlp))]
        return (*pair, down if storage == "fp8 bf16" else fp8(down, 16 / 448, rows))
    packed = gw.nvfp4_pack_weights(both, 6 / 2688)
    if joined:
        split = gw.nvfp4_scale_storage_bytes(mlp, hidden)
        gate = gw.Nvfp4Weight(packed.data[:mlp], packed.scales[:split], packed.input_scale, packed.weight_scale)
        up = gw.Nvfp4Weight(packed.data[mlp:], packed.scales[split:], packed.input_scale, packed.weight_scale)
    else:
        gate, up = gw.nvfp4_pack_weights(both[:mlp].contiguous(), 6 / 2688), gw.nvfp4_pack_weights(both[mlp:].contiguous(), 6 / 2688)
    return gate, up, gw.nvfp4_pack_weights(down, 16 / 2688)


@pytest.mark.parametrize("storage,joined", [("nvfp4", True), ("nvfp4", False), ("fp8", False), ("fp8 channel", True), ("fp8 bf16", True),
                                            ("bf16", True), ("bf16", False), ("bf16 fp8", True)])
@pytest.mark.parametrize("rows,hidden,mlp", [(129, 128, 128), (255, 256, 384), (256, 640, 128), (257, 384, 1152), (513, 1024, 256), (300, 2816, 2176)])
def test_fused_equals_separate_launches(gw, monkeypatch, storage, joined, rows, hidden, mlp):
    from gewell_b200 import _lib
    weights = projections(gw, storage, hidden, mlp, joined)
    bound = [gw.make_projection(w, i, o) for w, i, o in zip(weights, (hidden, hidden, mlp), (mlp, mlp, hidden))]
    x = bf16_normal((rows, hidden), rows).cuda()
    results = []
    for apart in (False, True):
        if apart:
            monkeypatch.setenv("GW_DENSE_NO_PAIR", "1")
        else:
            monkeypatch.delenv("GW_DENSE_NO_PAIR", raising=False)
        chain = gw.MlpChain(hidden, mlp, rows, _lib.POLICY_ALWAYS)
        chain.prepare(rows)
        y = chain.run(*bound, x, _lib.PHASE_PREFILL)
        torch.cuda.synchronize()
        assert gw.kernel_error() == 0
        results.append(bits(y))
    assert_gemm_close(results[0], results[1], f"{storage} {rows}x{hidden}->{mlp}")


@pytest.mark.parametrize("storage,joined", [("nvfp4", True), ("nvfp4", False), ("fp8", False), ("fp8 channel", True), ("fp8 bf16", True),
                                            ("bf16", False), ("bf16 fp8", True)])
@pytest.mark.parametrize("rows,hidden,mlp", [(9, 2816, 2176), (32, 256, 384), (33, 640, 1152), (65, 384, 256), (128, 384, 2176)])
def test_few_rows(gw, monkeypatch, storage, joined, rows, hidden, mlp):
    """Narrow MLPs from 9 rows on, BF16 from 33; test_dense_routes.py asserts the launches."""
    if storage.startswith("bf16") and rows <= 32:
        rows += 32
    test_fused_equals_separate_launches(gw, monkeypatch, storage, joined, rows, hidden, mlp)


@pytest.mark.parametrize("storage", ["fp8 channel", "bf16", "bf16 fp8"])
@pytest.mark.parametrize("rows,mlp", [(250, 9728), (300, 9600)])
def test_last_wave_in_pieces(gw, monkeypatch, storage, rows, mlp):
    """Two or a few tiles behind the last whole wave of 148 SMs, in pieces of 32 tokens."""
    test_fused_equals_separate_launches(gw, monkeypatch, storage, True, rows, 128, mlp)
