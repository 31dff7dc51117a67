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
    # without a snapshot (counts and scales read by every CTA)
    live = DecodeTable([p for p, _ in layers], [n for _, n in layers], H * g, live_counts=True)
    out = packed_decode_attention(q.cuda(), live)
    for i, want in enumerate(wants):
        assert_attn_close(to_np(out[i]), want, f"live view {i}")


@pytest.mark.parametrize("counts", CHANNELS)
@pytest.mark.parametrize("kept", [(301, 77), (1, 640)])
def test_separate_operators_on_rows_of_any_width(counts, kept):
    """The score operator writes the columns below ``T_eff`` of a wider buffer whose rows start off 16-byte
    boundaries, and nothing else; the V operator takes the same layer."""
    from oracle import ref_attention as RA
    from oracle.ref_packing import unpack_k
    from rdkv_b200 import synth
    from rdkv_b200.k_kernel import _scores_table, k_mixed_qk_dot_into
    from rdkv_b200.v_kernel import v_dequant_weighted_sum_dispatch
    g, H = 4, 2
    pl, nv = _layer(counts, 700, list(kept), 11, g)
    q = synth.make_q(H * g, seed=5)
    layer = layer_to_np(pl)
    want = RA.k_scores(q.numpy(), layer, pl.T_eff_k)
    # two roundings to fp16 a product, of the folded query here and of the oracle's dequantised K (2^-11
    # each), and fp32 sums of up to 224 terms, some of them below fp16's normal numbers
    size = np.einsum("hd,htd->ht", np.abs(q.numpy().astype(np.float32)), np.repeat(np.abs(unpack_k(layer, 128)[0].astype(np.float32)), g, 0))
    bound = size / np.sqrt(128.0) * 2.0 ** -10 + 3e-4
    assert _scores_table(pl, H * g) is not None, "the fused kernel takes the layer"
    for t_eff in (pl.T_eff_k, pl.T_eff_k - 5, 1):
        buf = torch.full((H * g, pl.T_eff_k + 13), 7.0, device="cuda")
        k_mixed_qk_dot_into(q.cuda(), pl, t_eff, buf[:, 3:3 + pl.T_eff_k])
        got = to_np(buf)
        assert (np.abs(got[:, 3:3 + t_eff] - want[:, :t_eff]) <= bound[:, :t_eff]).all()
        assert (got[:, :3] == 7.0).all() and (got[:, 3 + t_eff:] == 7.0).all()
    w = torch.rand(H * g, pl.T_eff_k, generator=torch.Generator().manual_seed(2)) / 300
    out = v_dequant_weighted_sum_dispatch(w.cuda(), pl, V16=None if nv is None else nv[0], n_v16_per_head=pl.n_v16_per_head, max_T_v=pl.T_eff)
    assert_attn_close(to_np(out), RA.v_weighted_sum(w.numpy(), layer, to_np(nv)), "weighted sum")


@pytest.mark.parametrize("counts", [(16, 24, 24), (23, 31, 35), (3, 17, 100), (5, 32, 0), (1, 0, 0)])
@pytest.mark.parametrize("persistent", [False, True])
@pytest.mark.parametrize("n_chunks", [None, 3])
def test_parts_windows_and_records_of_any_width(counts, persistent, n_chunks):
    """Sequence parts and row windows cut a head's rows anywhere, with odd widths at any byte: every record
    against the oracle's, and the records of all parts merged against the unsplit result."""
    from oracle import ref_attention as RA
    from rdkv_b200 import synth
    from rdkv_b200.decode import DecodeTable, lse_combine, packed_decode_attention
    g, H = 4, 2
    layers = [_layer(counts, 700, [301, 77], 11, g), _layer(counts, 701, [5, 640], 12, g)]
    q = synth.make_q(H * g, seed=5, batch=2)
    host = [(layer_to_np(pl), to_np(nv)) for pl, nv in layers]
    table = DecodeTable([p for p, _ in layers], [n for _, n in layers], H * g, persistent=persistent, n_chunks=n_chunks)
    unsplit = packed_decode_attention(q.cuda(), table)

    def record(**cut):
        rec = torch.full((2 * H * g, 132), float("nan"), device="cuda")
        packed_decode_attention(q.cuda(), table, out_partial=rec, **cut)
        r = to_np(rec).reshape(2, H * g, 132)
        for i, (pl, nv) in enumerate(host):
            o, m, l = RA.decode_attention(q[i].numpy(), pl, nv, **cut)
            live = l > 0
            assert np.array_equal(np.isfinite(r[i, :, 0]), live)
            assert_attn_close(r[i][live, 4:] / r[i][live, 1:2], o[live], f"{cut} view {i}")
        return rec

    for cut in (dict(rows=(0, 1)), dict(rows=(37, 138)), dict(rows=(63, 300)), dict(rows=(299, 700))):
        record(**cut)
    recs = [record(seq_part=(i, 3)) for i in range(3)]
    merged = lse_combine(torch.stack(recs, dim=1)).view(2, H * g, 128)
    assert_attn_close(to_np(merged), to_np(unsplit), "parts merged")
    windows = []                                             # of the last part's rows
    for rows in ((0, 13), (13, 98), (98, 1 << 20)):
        windows.append(torch.empty((2 * H * g, 132), device="cuda"))
        packed_decode_attention(q.cuda(), table, out_partial=windows[-1], seq_part=(2, 3), rows=rows)
    assert_attn_close(to_np(lse_combine(torch.stack(windows, dim=1))), to_np(lse_combine(recs[2][:, None])), "windows of a part merged")
    table.check_status()


@pytest.mark.parametrize("counts", [(23, 31, 35), (3, 17, 100), (1, 0, 0)])
def test_additive_mask_of_any_width(counts):
    """The additive mask (finite values and -inf) with K rows of any width."""
    from oracle import ref_attention as RA
    from rdkv_b200 import synth
    from rdkv_b200.decode import DecodeTable, packed_decode_attention
    g, H = 4, 2
    layers = [_layer(counts, 700, [301, 77], 11, g), _layer(counts, 701, [5, 640], 12, g)]
    for i, (pl, _) in enumerate(layers):
        gen = torch.Generator().manual_seed(i)
        pl.softmax_mask += torch.randn(pl.softmax_mask.shape, generator=gen).cuda()
        pl.softmax_mask[torch.rand(pl.softmax_mask.shape, generator=gen).cuda() < 0.2] = float("-inf")
        pl.softmax_mask[:, 0] = 0.0                          # (every head keeps a row)
    q = synth.make_q(H * g, seed=5, batch=2)
    table = DecodeTable([p for p, _ in layers], [n for _, n in layers], H * g, use_mask=True)
    out = packed_decode_attention(q.cuda(), table)
    table.check_status()
    for i, (pl, nv) in enumerate(layers):
        assert_attn_close(to_np(out[i]), RA.decode_attention(q[i].numpy(), layer_to_np(pl), to_np(nv))[0], f"view {i}")


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
