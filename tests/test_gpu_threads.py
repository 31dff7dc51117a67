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


# (row widths of one kernel instance: whole words; any width)
@pytest.mark.parametrize("widths", [((16, 24, 24), (4, 8, 8)), ((23, 31, 35), (3, 17, 40))])
@pytest.mark.parametrize("form", ["one CTA per unit", "persistent", "live counts", "scores"])
def test_decode_of_two_row_widths(side_by_side, widths, form):
    from rdkv_b200 import synth
    from rdkv_b200.decode import DecodeTable, packed_decode_attention
    from rdkv_b200.k_kernel import k_mixed_qk_dot
    from rdkv_b200.packing import pack_kv

    def call_of(w):
        K, V = synth.make_kv(4, 200, seed=5)
        kb = synth.make_k_bits(4, seed=5, mix=tuple(zip((8, 4, 2), w)))
        pl, nv = pack_kv(K.cuda(), V.cuda(), synth.make_v_bits(4, 200, 150, seed=5).cuda(), kb.cuda(), 4)
        q = synth.make_q(16, seed=3, batch=1).cuda()
        if form == "scores":
            k_mixed_qk_dot(q[0], pl, pl.T_eff_k)             # (its table is built by the first call)
            return lambda: (k_mixed_qk_dot(q[0], pl, pl.T_eff_k),)
        table = DecodeTable([pl], [nv], 16, persistent=form == "persistent", live_counts=form == "live counts")
        return lambda: (packed_decode_attention(q, table),)

    side_by_side([call_of(w) for w in widths])


@pytest.mark.parametrize("k_passes", [1, 3])
def test_packing_of_two_widths(side_by_side, k_passes):
    from rdkv_b200 import synth
    from rdkv_b200.packing import pack_kv_layers

    batches = []

    def call_of(widths, kept):
        K, V = synth.make_kv(2, 700, seed=kept)
        vb = synth.make_v_bits(2, 700, kept, seed=kept).cuda()
        kb = synth.make_k_bits(2, seed=kept, mix=tuple(zip((8, 4, 2), widths))).cuda()
        K, V = K.cuda(), V.cuda()

        def call():
            batches.append(pack_kv_layers([K], [V], vb[None], kb[None], 4, build_mask=False, k_passes=k_passes))
            pl, _ = batches[-1][0]
            return pl.K_2bit, pl.K_4bit, pl.K_8bit, pl.K_ch_scale, pl.K_ch_zp
        return call

    side_by_side([call_of((8, 12, 8), 90), call_of((40, 48, 40), 640)])


def test_window_scores_of_two_sizes(side_by_side):
    from rdkv_b200.scoring import obs_window_scores

    def call_of(window):
        gen = torch.Generator(device="cuda").manual_seed(window)
        q = torch.randn(1, 8, window, 128, generator=gen, device="cuda").half()
        k = torch.randn(1, 2, 1000, 128, generator=gen, device="cuda").half()
        return lambda: obs_window_scores(q, k)

    side_by_side([call_of(32), call_of(64)])


def test_block_scores_of_two_sizes(side_by_side):
    from rdkv_b200.blockwise import _score_block

    def call_of(tokens):
        gen = torch.Generator(device="cuda").manual_seed(tokens)
        q = torch.randn(8, tokens, 128, generator=gen, device="cuda").half()
        k = torch.randn(1, 2, tokens, 128, generator=gen, device="cuda").half()
        return lambda: _score_block(q, k, num_kv_groups=4, causal=False)

    side_by_side([call_of(64), call_of(256)])
