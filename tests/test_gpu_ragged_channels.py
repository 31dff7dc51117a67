"""Decode over layers whose K rows have any number of bytes at any address: every way the fused kernel
reads K codes (one span of whole words, two spans and many spans at any byte), odd row counts that
put V scales on odd half-words, and heads of very different lengths, against the oracle."""
import numpy as np
import pytest
import torch

from helpers import assert_attn_close, layer_to_np, to_np

pytestmark = pytest.mark.gpu

# channels per head of 8, 4 and 2 bits: aligned single spans, odd widths, empty segments, two spans at the
# limit, more than two spans
CHANNELS = [(16, 24, 24), (24, 31, 27), (23, 31, 35), (5, 32, 0), (0, 3, 61), (32, 64, 32), (1, 0, 0), (33, 40, 50), (3, 17, 100)]


def _layer(counts, T, kept, seed, g, H=2):
    from rdkv_b200 import synth
    from rdkv_b200.packing import pack_kv
    K, V = synth.make_kv(H, T, seed=seed)
    vb = synth.make_v_bits(H, T, max(kept), seed=seed, per_head_N=kept)
    kb = synth.make_k_bits(H, seed=seed, mix=tuple(zip((8, 4, 2), counts)))
    if sum(counts) > 4:                                      # another count in the second head: padded slots
        kb[1, torch.nonzero(kb[1] == (8 if counts[0] else 4))[0]] = 0
    return pack_kv(K.cuda(), V.cuda(), vb.cuda(), kb.cuda(), g)


@pytest.mark.parametrize("counts", CHANNELS)
@pytest.mark.parametrize("kept", [(301, 77), (1, 640)])
def test_k_rows_of_any_width(counts, kept):
    from oracle import ref_attention as RA
    from rdkv_b200 import synth
    from rdkv_b200.decode import DecodeTable, packed_decode_attention
    g, H = 4, 2
    layers = [_layer(counts, 700, list(kept), 11, g), _layer(counts, 701, list(kept)[::-1], 12, g)]
    q = synth.make_q(H * g, seed=5, batch=2)
    wants = [RA.decode_attention(q[i].numpy(), layer_to_np(pl), to_np(nv))[0] for i, (pl, nv) in enumerate(layers)]
    for persistent in (False, True):
        table = DecodeTable([p for p, _ in layers], [n for _, n in layers], H * g, persistent=persistent)
        assert table._all_fast, "the packed rows lie in copyable 16-byte blocks"
        out = packed_decode_attention(q.cuda(), table)
        table.check_status()
        for i, want in enumerate(wants):
            assert_attn_close(to_np(out[i]), want, f"view {i}, persistent {persistent}")
    # without a snapshot (counts and scales read by every CTA) and through the two separate operators
    live = DecodeTable([p for p, _ in layers], [n for _, n in layers], H * g, live_counts=True)
    out = packed_decode_attention(q.cuda(), live)
    for i, want in enumerate(wants):
        assert_attn_close(to_np(out[i]), want, f"live view {i}")


@pytest.mark.parametrize("counts", [(16, 24, 24), (23, 31, 35), (3, 17, 100), (1, 0, 0)])
@pytest.mark.parametrize("tails", [(1, 15), (16, 17), (31, 33), (47, 49), (63, 64), (65, 127), (129, 500)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_tail_tiles(counts, tails, dtype):
    """Tail lengths at the edges of a warp's 16 rows and of a tile, for stages of several sizes, whole units
    and chunks; rows behind the live ones are not numbers and must not show."""
    from oracle import ref_attention as RA
    from rdkv_b200 import synth
    from rdkv_b200.decode import DecodeTable, packed_decode_attention
    g, H, cap = 4, 2, 512
    layers = [_layer(counts, 400, [201, 77], 11, g), _layer(counts, 401, [5, 300], 12, g)]
    gen = torch.Generator().manual_seed(sum(tails))
    q = synth.make_q(H * g, seed=6, batch=2, dtype=dtype)
    new = torch.randn(2, 2, H, cap, 128, generator=gen).to(dtype)            # K, V
    wants = [RA.decode_attention(q[i].float().numpy(), layer_to_np(pl), to_np(nv), new[0, i, :, :tails[i]].float().numpy(),
                                 new[1, i, :, :tails[i]].float().numpy())[0] for i, (pl, nv) in enumerate(layers)]
    for i in range(2):
        new[:, i, :, tails[i]:] = float("nan")
    new = new.cuda()
    n_new = torch.tensor(tails, dtype=torch.int32, device="cuda")
    for n_chunks in (None, 3):
        table = DecodeTable([p for p, _ in layers], [n for _, n in layers], H * g, n_chunks=n_chunks)
        out = packed_decode_attention(q.cuda(), table, new_k=new[0], new_v=new[1], n_new=n_new)
        table.check_status()
        for i, want in enumerate(wants):
            assert_attn_close(to_np(out[i]), want, f"view {i}, chunks {n_chunks}")


@pytest.mark.parametrize("rows", [128, 129, 257, 1061, 2600])
@pytest.mark.parametrize("counts", [(16, 24, 24), (23, 31, 35)])
def test_few_units_in_many_chunks(rows, counts):
    """A launch of few units is cut into up to 16 chunks each, the last of them short or empty: against
    whole units."""
    from rdkv_b200 import synth
    from rdkv_b200.decode import DecodeTable, packed_decode_attention
    g, H = 4, 2
    pl, nv = _layer(counts, rows + 20, [rows, max(1, rows // 3)], 7, g)
    q = synth.make_q(H * g, seed=8, batch=1).cuda()
    table = DecodeTable([pl], [nv], H * g)
    k, chunk, n_whole = table.plan(1)
    assert k * chunk >= rows and k <= 16 and (n_whole == 0) == (k > 1)
    whole = packed_decode_attention(q, DecodeTable([pl], [nv], H * g, n_chunks=1))
    assert_attn_close(to_np(packed_decode_attention(q, table)), to_np(whole), f"{k} chunks of {chunk}")
    table.check_status()


@pytest.mark.parametrize("rows", [1, 127, 128, 255, 256, 700, 2048])
@pytest.mark.parametrize("heads,g", [(1, 4), (2, 8), (8, 4), (3, 16)])
def test_weighted_sum_in_clusters(rows, heads, g):
    """The V operator cuts a head's rows over a cluster of CTAs: lengths at the edges of the cut, empty
    chunks, more query heads than one pass takes."""
    from oracle import ref_attention as RA
    from rdkv_b200.v_kernel import v_dequant_weighted_sum_dispatch
    kept = [max(1, rows * (h + 1) // heads) for h in range(heads)]
    pl, nv = _layer((16, 24, 24), rows + 40, kept, 3, g, H=heads) if heads > 1 else _layer_one(rows, kept, g)
    w = torch.rand(heads * g, pl.T_eff_k, generator=torch.Generator().manual_seed(1)) / rows
    got = v_dequant_weighted_sum_dispatch(w.cuda(), pl, V16=None if nv is None else nv[0], n_v16_per_head=pl.n_v16_per_head,
                                          max_T_v=pl.T_eff)
    assert_attn_close(to_np(got), RA.v_weighted_sum(w.numpy(), layer_to_np(pl), to_np(nv)), f"{rows} rows")
    again = v_dequant_weighted_sum_dispatch(w.cuda(), pl, V16=None if nv is None else nv[0], n_v16_per_head=pl.n_v16_per_head,
                                            max_T_v=pl.T_eff)
    assert torch.equal(got, again), "the order of the sums is fixed"


def _layer_one(rows, kept, g):
    from rdkv_b200 import synth
    from rdkv_b200.packing import pack_kv
    K, V = synth.make_kv(1, rows + 40, seed=3)
    vb = synth.make_v_bits(1, rows + 40, kept[0], seed=3)
    return pack_kv(K.cuda(), V.cuda(), vb.cuda(), synth.make_k_bits(1, seed=3).cuda(), g)
