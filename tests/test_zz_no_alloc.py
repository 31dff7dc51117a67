"""The allocation-free allocator entry point (rdkv_knapsack_batched_static) against the
regular one, called through the C ABI.

Who needs it: code that must run the bit allocator from a place where device memory may
not be allocated any more — an inference engine whose memory plan is frozen after
warm-up, a host callback, a plugin handed nothing but input and output buffers.  The
regular entry point wants a small scratch buffer from the caller; this one keeps it
inside the library.  Both must choose exactly the same bits.

The file name sorts last on purpose: a run that stops at the first failure has then
already been through every other test.
"""
import ctypes as C
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu


def _call(static: bool, scores, budget, out, eps, max_iters=60, tol=0.01):
    from rdkv_b200 import _lib
    lib = _lib.lib()
    opts = [0.0, 2.0, 4.0, 8.0, 16.0]
    c_bits = (C.c_float * 5)(*opts)
    c_eps = (C.c_float * 5)(*[eps[int(b)] for b in opts])
    B, T = scores.shape
    stream = torch.cuda.current_stream().cuda_stream
    if static:
        st = lib.rdkv_knapsack_batched_static(scores.data_ptr(), scores.stride(0), B, T, budget.data_ptr(), c_bits,
                                              c_eps, 5, max_iters, tol, out.data_ptr(), stream)
    else:
        scratch = torch.empty(3 * B, dtype=torch.int32, device="cuda")
        st = lib.rdkv_knapsack_batched(scores.data_ptr(), scores.stride(0), B, T, budget.data_ptr(), c_bits, c_eps,
                                       5, max_iters, tol, out.data_ptr(), scratch.data_ptr(), stream)
    return st


def test_static_scratch_variant_matches_regular_entry_point_twice():
    from rdkv_b200 import _lib, synth
    eps = synth.ALLOC_EPSILON
    lib = _lib.lib()
    assert lib.rdkv_knapsack_static_max_rows() == 4096
    # two calls in a row with different shapes and budgets: the shared scratch keeps the first
    # call's contents, the second call must not be disturbed by them
    for seed, rows, T, budgets in ((31, 96, 4096, (2.0, 0.5)), (32, 17, 700, (6.0, 1.0))):
        scores = synth.make_scores(rows, T, seed=seed, device="cuda")
        budget = torch.full((rows,), budgets[0], dtype=torch.float32, device="cuda")
        budget[::3] = budgets[1]
        want = torch.empty((rows, T), dtype=torch.int64, device="cuda")
        got = torch.full((rows, T), -1, dtype=torch.int64, device="cuda")
        assert _call(False, scores, budget, want, eps) == 0
        assert _call(True, scores, budget, got, eps) == 0
        torch.cuda.synchronize()
        assert torch.equal(got, want)          # integer choices: bit-exact, like every allocator test
    # more rows than the built-in scratch holds: refused, nothing launched
    big = torch.ones((4097, 8), dtype=torch.float32, device="cuda")
    out = torch.empty((4097, 8), dtype=torch.int64, device="cuda")
    bud = torch.full((4097,), 2.0, dtype=torch.float32, device="cuda")
    assert _call(True, big, bud, out, eps) == 3


# (rows, length) of every kernel the call chooses from, behind a warm-up of another shape
SHAPES = [(8, 100), (300, 100), (8, 200), (300, 200), (300, 1000), (100, 5000), (40, 20000), (8, 40000), (300, 20000),
          (100, 32769), (30, 65537), (8, 131073), (3, 300000)]

CHILD = """
import sys
import torch
from rdkv_b200 import _lib, synth
from test_zz_no_alloc import SHAPES, _call
n = max(r * t for r, t in SHAPES)
scores = torch.rand(n, device="cuda")
out = torch.empty(n, dtype=torch.int64, device="cuda")
budget = torch.full((4096,), 2.0, device="cuda")
def call(rows, length, eps):
    assert _call(True, scores[:rows * length].view(rows, length), budget[:rows], out, eps) == 0
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]
eps = dict(synth.ALLOC_EPSILON)
free = call(4, 700, eps)
told = [(r, t, call(r, t, eps)) for r, t in SHAPES]
eps[8] = -eps[8]                                             # (the kernels for negative distortions)
told += [(r, t, call(r, t, eps)) for r, t in ((3, 700), (3, 300000))]
sys.exit(f"{free} bytes free after the warm-up, then {told}" if any(f != free for _, _, f in told) else 0)
"""


def test_one_warm_up_call_loads_every_kernel():
    """After one call of one shape the device's free memory stays where it is, whatever shapes follow (in a
    fresh process: what a process has loaded it keeps)."""
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([os.path.dirname(here), here]), CUDA_MODULE_LOADING="LAZY")
    got = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True, timeout=300)
    assert got.returncode == 0, got.stdout + got.stderr
