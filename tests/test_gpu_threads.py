"""Calls of different sizes from several host threads at the same time.

ctypes gives up the interpreter lock during a call, so the launchers really run side by side.  What a
launcher sets on a KERNEL (its limit of dynamic shared memory) is shared by all threads: one call must
not take away what another one is about to launch with.  To spend the time in the launchers and not in
Python, the library calls of one ordinary call are recorded with their arguments and then repeated from
several threads (on one stream: the repetitions write the same values to the same buffers)."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu

THREADS, CALLS = 3, 1500                                     # per recorded call


class _Recorder:
    """Stands for the loaded library: passes every call on and writes it down with what it returned."""

    def __init__(self, real):
        self.real, self.calls = real, []

    def __getattr__(self, name):
        fn = getattr(self.real, name)

        def call(*args):
            got = fn(*args)
            self.calls.append((fn, args, got))
            return got
        return call


@pytest.fixture
def side_by_side(monkeypatch):
    """Runs ordinary calls (each returning its result tensors) once and then repeats their library calls
    from several threads each: no repetition may be refused, and the results stay."""
    from rdkv_b200 import _lib, blockwise, decode, k_kernel, knapsack_solver, packing, scoring
    modules = (blockwise, decode, k_kernel, knapsack_solver, packing, scoring)

    def run(calls):
        kept, recorded, results = [], [], []
        empty = torch.empty
        with monkeypatch.context() as m:
            # (scratch that a call lets go of has to stay its own for the repetitions)
            m.setattr(torch, "empty", lambda *a, **k: (kept.append(empty(*a, **k)), kept[-1])[1])
            for call in calls:
                recorder = _Recorder(_lib.lib())
                for module in modules:
                    m.setattr(module, "lib", lambda recorder=recorder: recorder)
                results.append(call())
                recorded.append(recorder.calls)
        wants = [[t.clone() for t in r] for r in results]
        torch.cuda.synchronize()
        start, refused = threading.Barrier(THREADS * len(calls)), []

        def work(library_calls):
            start.wait(60)
            for _ in range(CALLS):
                for fn, args, got in library_calls:
                    again = fn(*args)
                    if again != got:
                        refused.append((fn.__name__, again))

        threads = [threading.Thread(target=work, args=(r,)) for r in recorded for _ in range(THREADS)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        assert not refused, f"{len(refused)} calls refused, first {refused[0]}"
        assert all(torch.equal(a, b) for r, w in zip(results, wants) for a, b in zip(r, w))
    return run


@pytest.mark.parametrize("rows,lengths", [(2, (131072, 32768)), (150, (32768, 20000)), (2, (2000, 4000))])
def test_allocator_rows_of_two_lengths(side_by_side, rows, lengths):
    from rdkv_b200 import synth
    from rdkv_b200.knapsack_solver import knapsack_bit_allocation_batched

    def call_of(length):
        scores = synth.make_scores(rows, length, seed=length, device="cuda")
        return lambda: (knapsack_bit_allocation_batched(scores, 2.0, epsilon=synth.ALLOC_EPSILON, max_iters=0),)

    side_by_side([call_of(n) for n in lengths])
