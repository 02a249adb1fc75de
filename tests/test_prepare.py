"""A prepare() that fails leaves its object as it was: the next run() works on the row count of the last prepare() that
succeeded, in every part of it.  Every allocation of a prepare() fails in turn, on a CUDA runtime that only counts
(tests/cpp/fake_cudart.cpp); the number of launches of a run tells the row count each part works on.  A prepare() that
succeeds has waited for what it filled: streams need not be ordered behind the default one.  No GPU."""
import os
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

CHILD = r'''
import ctypes, os, sys
sys.path.insert(0, os.environ["GW_ROOT"])
from gewell_b200 import _lib
fake = ctypes.CDLL(os.environ["GW_FAKE"])
for name in ("fake_launches", "fake_allocations_left", "fake_unfinished"):
    getattr(fake, name).restype = ctypes.c_long
fake.fake_fail_allocation.argtypes = [ctypes.c_long]
lib = _lib.load()
check = lambda status: _lib.check(lib, status)
A = 0x7000_0000_0000                       # any address: nothing touches it


def projection(storage, k, n, physical=None):
    p = _lib.Projection()
    p.storage, p.input, p.output, p.physical_output = storage, k, n, physical or n
    p.bf16 = p.nvfp4_data = p.fp8_data = A
    p.nvfp4_scales = A + (1 << 32)
    p.nvfp4_input_scale = p.nvfp4_weight_scale = p.fp8_input_scale = p.fp8_weight_scale = 0.01
    return p


def launches(run):
    before = fake.fake_launches()
    check(run())
    return fake.fake_launches() - before


def each_allocation_fails(prepare, run, small, large):
    """From `small` rows, prepare(large) fails at its 1st, 2nd, ... allocation until it has no more."""
    check(prepare(small))
    assert fake.fake_unfinished() == 0, "set-up that a run on another stream may overtake"
    at_small = launches(run)
    failures = 0
    while True:
        fake.fake_fail_allocation(failures + 1)
        status = prepare(large)
        spent = fake.fake_allocations_left() == 0
        fake.fake_fail_allocation(0)
        if not spent:
            break
        assert status == _lib.GW_CUDA_ERROR, status
        failures += 1
        assert launches(run) == at_small, f"allocation {failures} of prepare({large}) from {small} rows"
    check(status)
    assert fake.fake_unfinished() == 0
    assert launches(run) != at_small and failures >= 1
'''

PROJECTIONS = CHILD + r'''
p = projection(_lib.STORAGE_NVFP4_W4A4, 2816, 4096)
q = projection(_lib.STORAGE_NVFP4_W4A4, 4096, 2816)
ws = ctypes.c_void_p()
check(lib.gw_projection_workspace_create((_lib.Projection * 2)(p, q), 2, 256, _lib.POLICY_PREFILL, None, ctypes.byref(ws)))
prepare = lambda rows: lib.gw_projection_workspace_prepare(ws, rows, _lib.PHASE_DECODE)
run = lambda: lib.gw_projection_workspace_run(ws, ctypes.byref(p), A, A)
for small, large in ((200, 5), (5, 24), (24, 5), (40, 5)):
    each_allocation_fails(prepare, run, small, large)
'''

CHAIN = CHILD + r'''
gate, up, down = (projection(_lib.STORAGE_NVFP4_W4A4, k, n) for k, n in ((640, 1408), (640, 1408), (1408, 640)))
chain = ctypes.c_void_p()
check(lib.gw_mlp_chain_create(640, 1408, 256, _lib.POLICY_PREFILL, ctypes.byref(chain)))
prepare = lambda rows: lib.gw_mlp_chain_prepare(chain, rows)
run = lambda: lib.gw_mlp_chain_run(chain, *map(ctypes.byref, (gate, up, down)), A, A, A, A, _lib.PHASE_DECODE, None)
for small, large in ((200, 5), (5, 24), (24, 5), (40, 5)):
    each_allocation_fails(prepare, run, small, large)
'''

BLOCK = CHILD + r'''
NV = _lib.STORAGE_NVFP4_W4A4
experts = (_lib.ExpertWeights * 128)()
for e in experts:
    e.gate = e.up = projection(NV, 2816, 704, 768)
    e.down = projection(NV, 704, 2816)
table = ctypes.c_void_p()
check(lib.gw_moe_expert_table_create(experts, 128, ctypes.byref(table)))
w = _lib.FfnBlockWeights()
for name in ("pre_feedforward_norm", "router_scale", "pre_feedforward_norm_2", "post_feedforward_norm_1", "post_feedforward_norm_2",
             "post_feedforward_norm", "layer_scalar", "router_proj", "router_per_expert_scale"):
    setattr(w, name, A)
w.gate = w.up = projection(NV, 2816, 2112, 2176)
w.down = projection(NV, 2112, 2816)
w.experts, w.has_nvfp4 = table, 1
block = ctypes.c_void_p()
check(lib.gw_ffn_block_create(ctypes.byref(w), 1, 256, _lib.POLICY_ALWAYS, 0, None, ctypes.byref(block)))
prepare = lambda rows: lib.gw_ffn_block_prepare(block, rows, _lib.PHASE_DECODE)
run = lambda: lib.gw_ffn_block_run(block, ctypes.byref(w), A)
for small, large in ((8, 40), (40, 8)):
    each_allocation_fails(prepare, run, small, large)
'''


@pytest.fixture(scope="module")
def fake_runtime(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    library = tmp_path_factory.mktemp("fake") / "libfakecudart.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", str(ROOT / "tests" / "cpp" / "fake_cudart.cpp"), "-o",
                    str(library)], check=True)
    return library


def run_child(fake_runtime, script):
    env = dict(os.environ, LD_PRELOAD=str(fake_runtime), GW_FAKE=str(fake_runtime), GW_ROOT=str(ROOT))
    done = subprocess.run([sys.executable, "-c", script], env=env, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stdout + done.stderr


@pytest.mark.parametrize("script", [PROJECTIONS, CHAIN, BLOCK], ids=["projections", "mlp chain", "feed-forward block"])
def test_failed_prepare_leaves_the_row_count(fake_runtime, script):
    run_child(fake_runtime, script)
