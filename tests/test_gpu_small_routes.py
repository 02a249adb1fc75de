"""Routing of at most 64 tokens (one cluster of eight blocks, a token per warp) at the edges of its blocks and warps."""
import numpy as np
import pytest
import torch

from oracle import codecs as C
from oracle import moe as omoe
from tests.gpu_helpers import to_f32
from tests.test_gpu_moe import E, make_scores

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 7, 8, 9, 56, 57, 63, 64])
@pytest.mark.parametrize("mode", ["normal", "ties", "uneven"])
def test_cluster_dispatch(rows, mode):
    import gewell_b200 as gw
    scores = make_scores(rows, mode)
    scales = C.bf16_round(1.0 + 0.1 * np.sin(np.arange(E, dtype=np.float32)))
    ws = gw.MoeWorkspace(64)
    ws.dispatch(scores.cuda(), torch.from_numpy(scales).to(torch.bfloat16).cuda(), rows)
    torch.cuda.synchronize()
    ids, weights = omoe.route(to_f32(scores), scales)
    order, offsets = omoe.permutation(ids)
    assert np.array_equal(ws.selected_experts().cpu().numpy()[:rows], ids)
    np.testing.assert_allclose(ws.routing_weights().cpu().numpy()[:rows], weights, rtol=3e-6, atol=0)
    assert np.array_equal(ws.offsets().cpu().numpy(), offsets)
    assert np.array_equal(ws.sorted_assignments().cpu().numpy()[: 8 * rows], order)
