"""Which kernels a projection is launched on, from the host code alone: a CUDA runtime that only records
(tests/cpp/fake_cudart.cpp, 148 SMs) names them.  No GPU."""
import pytest

from tests.test_gpu_pair_split import SHARED
from tests.test_gpu_pair_wide import FEW_ROWS
from tests.test_gpu_stream_whole import STREAMED
from tests.test_prepare import CHILD, fake_runtime, run_child  # noqa: F401  (fixture)

NAMES = CHILD + r'''
fake.fake_launched.restype = ctypes.c_char_p


def kernels(run):
    """The kernels that a run launches, as the compiler mangles their names."""
    fake.fake_launched()
    check(run())
    return fake.fake_launched().decode().split()


def nvfp4_plan(rows, k, n):
    plan = ctypes.c_void_p()
    check(lib.gw_nvfp4_plan_create(rows, k, n, ctypes.byref(plan)))
    return lambda output: lib.gw_nvfp4_plan_run(plan, A, A, A, 0.01, 0.01, output, A, 1 << 40, None, 0)
'''

UNALIGNED = NAMES + r'''
swap_form = kernels(lambda: nvfp4_plan(128, 2816, 2816)(A))[-1]
assert "gemm_tc_kernel" in swap_form
for rows, k, n in ((128, 8192, 256), (129, 256, 128), (200, 2816, 2816), (257, 12352, 2560), (1000, 640, 384)):
    run = nvfp4_plan(rows, k, n)
    for offset in (0, 2, 8, 0, 14):
        names = kernels(lambda: run(A + offset))
        assert len(names) == 2
        assert (names[1] == swap_form) == (offset != 0), (rows, k, n, offset, names)
        assert ("gemm_pair" in names[1]) == (offset == 0), (rows, k, n, offset, names)
'''


@pytest.mark.parametrize("form", [None, "direct"])
def test_unaligned_nvfp4_output_keeps_off_vector_stores(fake_runtime, monkeypatch, form):
    """The kernels of more than 128 rows store sixteen bytes at a time; an output that is not 16-byte aligned takes the swap form."""
    script = UNALIGNED
    if form:
        monkeypatch.setenv("GW_DENSE_FORM", form)
        script = NAMES + r'''
for rows in (1, 40, 128, 300):
    run = nvfp4_plan(rows, 640, 384)
    direct, unaligned = kernels(lambda: run(A))[-1], kernels(lambda: run(A + 2))[-1]
    assert direct != unaligned and "gemm_tc_kernel" in unaligned, rows
'''
    run_child(fake_runtime, script)


GEGLU = NAMES + r'''
NV, F8, BF = _lib.STORAGE_NVFP4_W4A4, _lib.STORAGE_FP8_W8A8, _lib.STORAGE_BF16
for storage, kernel in ((NV, "gemm_pair_kernelILb1E"), (F8, "gemm_pair_wide_kernelILb1ELNS0_7WideOutE3"), (BF, "gemm_pair_wide_kernelILb0ELNS0_7WideOutE2")):
    for rows, hidden, mlp, fused in ((8, 2816, 2176, False), (9, 2816, 2176, storage != BF), (32, 256, 384, storage != BF),
                                     (33, 640, 1152, True), (41, 2816, 2176, True), (64, 256, 384, True), (65, 384, 256, True),
                                     (128, 384, 2176, True), (64, 2816, 9600, False), (129, 2816, 9600, True),
                                     (16, 5376, 2816, storage == F8),      # the swap form divides K of NVFP4 there
                                     (64, 5376, 2048, storage == F8), (96, 5376, 2048, storage != NV), (129, 5376, 2048, True)):
        chain = ctypes.c_void_p()
        check(lib.gw_mlp_chain_create(hidden, mlp, 256, _lib.POLICY_ALWAYS, ctypes.byref(chain)))
        check(lib.gw_mlp_chain_prepare(chain, rows))
        bound = [projection(storage, k, n) for k, n in ((hidden, mlp), (hidden, mlp), (mlp, hidden))]
        names = kernels(lambda: lib.gw_mlp_chain_run(chain, *map(ctypes.byref, bound), A, A, A, A, _lib.PHASE_PREFILL, None))
        assert any(kernel in name for name in names) == fused, (storage, rows, hidden, mlp, names)
'''


def test_narrow_mlps_of_few_rows_run_gate_up_and_geglu_in_one_launch(fake_runtime):
    run_child(fake_runtime, GEGLU)


PLANS = NAMES + r'''
def projection_kernels(kind, rows, k, n):
    """Of a projection by a plan of its own."""
    plan = ctypes.c_void_p()
    channel = kind.endswith("per channel")
    if kind == "nvfp4":
        run = nvfp4_plan(rows, k, n)
    elif kind.startswith("fp8"):
        check(lib.gw_fp8_plan_create(rows, k, n, int(channel), ctypes.byref(plan)))
        run = lambda output: lib.gw_fp8_plan_run(plan, A, A, 0.01, 0.01, A if channel else None, output, A, 1 << 40, None, 0)
    else:
        check(lib.gw_bf16_plan_create(rows, k, n, ctypes.byref(plan)))
        run = lambda output: lib.gw_bf16_plan_run(plan, A, A, output, A, 1 << 40, None)
    return kernels(lambda: run(A))


for kind, rows, k, n in SHAPES:
    names = projection_kernels(kind, rows, k, n)
    assert KERNEL in names[-1] and (not SPLIT or SPLIT in names[-1]), (kind, rows, k, n, names)
    if KERNEL == "decode_stream_kernel":
        assert len(names) == 1
'''


@pytest.mark.parametrize("shapes,kernel,split", [
    ([(kind, *shape) for kind, of in STREAMED.items() for shape in of], "decode_stream_kernel", None),
    ([("nvfp4", *shape) for shape in SHARED], "gemm_pair_kernel", "ILb0ELb0ELb1E"),
    (FEW_ROWS, "gemm_pair_wide_kernel", None)], ids=["streamed", "shared K", "few rows on pairs"])
def test_shapes_of_the_gpu_tests_take_the_route_under_test(fake_runtime, shapes, kernel, split):
    run_child(fake_runtime, f"SHAPES, KERNEL, SPLIT = {shapes!r}, {kernel!r}, {split!r}\n" + PLANS)


GRIDS = PLANS[:PLANS.index("for kind, rows, k, n in SHAPES")] + r'''
fake.fake_grid.restype = ctypes.c_long
# (kind, rows, K, N): blocks of the launch, whether pieces are summed by themselves
for shape, grid, pieces in (
        (("nvfp4", 1, 1024, 4864), 38, False), (("fp8", 1, 512, 4864), 38, False), (("fp8", 1, 1024, 512), 8, False),      # short K
        (("nvfp4", 1, 2816, 512), 16, False), (("nvfp4", 1, 2816, 8192), 148, False), (("bf16", 1, 2816, 4096), 128, False),
        (("nvfp4", 1, 5376, 1024), 32, True), (("fp8", 8, 2816, 1024), 32, True), (("bf16", 8, 5376, 2048), 64, True),       # few blocks, long K
        (("nvfp4", 1, 5376, 4096), 128, False), (("fp8", 8, 5376, 43008), 148, True)):
    names = projection_kernels(*shape)
    assert len(names) == 1 and "decode_stream_kernel" in names[0], (shape, names)
    assert fake.fake_grid() == grid and ("ELi1ELb0ELb1E" in names[0]) == pieces, (shape, fake.fake_grid(), names)
'''


def test_division_of_the_streaming_kernel(fake_runtime):
    """Blocks of a short K come together; pieces are summed by themselves where a warp has more of them than equal ranges would give it."""
    run_child(fake_runtime, GRIDS)
