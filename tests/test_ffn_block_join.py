"""A feed-forward block whose run fails brings its side stream back: work that follows on the caller's stream does not overlap
the shared MLP's, and a stream capture is left without a fork.  Every launch of a run fails in turn, on a CUDA runtime that only
records (tests/cpp/fake_cudart.cpp).  No GPU."""
import pytest

from tests.test_prepare import BLOCK, fake_runtime, run_child  # noqa: F401  (fixture)

JOIN = BLOCK[:BLOCK.index("for small, large")] + r'''
fake.fake_forked.restype = fake.fake_launch_failures_left.restype = ctypes.c_long
fake.fake_fail_launch.argtypes = [ctypes.c_long]
for rows in ROWS:
    check(prepare(rows))
    total = launches(run)
    assert fake.fake_forked() == 0
    reported = 0
    for n in range(1, total + 1):
        fake.fake_fail_launch(n)
        status = run()
        assert fake.fake_launch_failures_left() == 0
        assert fake.fake_forked() == 0, f"{rows} rows: launch {n} of {total} failed and the side stream was not joined"
        reported += status == _lib.GW_CUDA_ERROR
    assert reported >= 1
    assert launches(run) == total
'''


@pytest.mark.parametrize("rows", [8, 40, 129])
def test_failed_run_joins_the_side_stream(fake_runtime, rows):
    run_child(fake_runtime, JOIN.replace("ROWS", f"({rows},)"))


def test_router_memory_and_alignment(fake_runtime):
    """Beyond the block's buffers nothing is held for the router, and a router projection that no kernel takes is refused before
    anything is launched, at every row count."""
    run_child(fake_runtime, BLOCK[:BLOCK.index("for small, large")] + r'''
for name in ("gw_ffn_block_bytes", "gw_moe_bytes", "gw_projection_workspace_bytes"):
    getattr(lib, name).restype = ctypes.c_size_t
ws = ctypes.c_void_p()
check(lib.gw_projection_workspace_create((_lib.Projection * 3)(w.gate, w.up, w.down), 3, 256, _lib.POLICY_ALWAYS, None, ctypes.byref(ws)))
buffers = 256 * (5 * 2816 + 3 * 2112 + 128) * 2
assert lib.gw_ffn_block_bytes(block) == buffers + lib.gw_projection_workspace_bytes(ws) + lib.gw_moe_bytes(lib.gw_ffn_block_moe(block))
for rows in (8, 128, 129, 8):
    check(prepare(rows))
    w.router_proj = A + 8
    before = fake.fake_launches()
    assert run() == _lib.GW_INVALID_ARGUMENT and fake.fake_launches() == before
    w.router_proj = A
    check(run())
''')


def test_shared_mlp_of_few_nvfp4_rows_stays_on_the_swap_form(fake_runtime):
    """Gate, up and GeGLU in one launch from 65 rows on."""
    run_child(fake_runtime, BLOCK[:BLOCK.index("for small, large")] + r'''
fake.fake_launched.restype = ctypes.c_char_p
for rows, one_launch in ((9, False), (64, False), (65, True), (128, True), (129, True)):
    check(prepare(rows))
    fake.fake_launched()
    check(run())
    assert ("gemm_pair_kernelILb1E" in fake.fake_launched().decode()) == one_launch, rows
''')
