"""Prefill kernels at the sizes where they change their way of working: partition (tiles of 256 elements,
eight kept in shared memory, clusters of CTAs), allocator (a warp per short row, clusters and buckets for long ones),
batched packing of layers of different shapes, budgets, unpacking; against the oracle, bit for bit."""
import numpy as np
import pytest
import torch

from helpers import cuda, layer_to_np, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [1, 7, 255, 256, 257, 4096, 4097, 32769, 131072, 263000])
@pytest.mark.parametrize("dtype", [torch.int8, torch.int16, torch.int32, torch.int64])
def test_partition(length, dtype):
    from rdkv_b200.packing import _partition_pair, partition_by_bits
    rng = np.random.default_rng(length)
    rows = 3
    tok = rng.choice([0, 0, 2, 4, 8, 16, 1, -2, 3], size=(rows, length + 1))
    if dtype == torch.int64 and length > 2:
        tok[0, 1], tok[1, 1] = (1 << 32) + 4, -(1 << 33) + 2                 # the low word of neither counts
    ch = rng.choice([0, 2, 4, 8, 16], size=(rows, 128))
    maps = torch.from_numpy(tok).to(dtype).cuda()[:, 1:]                     # rows off 16-byte boundaries
    for mode, bits in ((0, maps), (1, maps)):
        order, counts = partition_by_bits(bits, mode)
        for r in range(rows):
            row = to_np(bits[r]).astype(np.int64)
            cls = [np.flatnonzero(row == b) for b in (2, 4, 8, 16)]
            if mode == 1:
                cls = cls[:2] + [np.flatnonzero((row == 8) | (row == 16)), np.zeros(0, np.int64)]
            want = np.concatenate(cls)
            assert to_np(counts[r]).tolist() == [len(c) for c in cls]
            assert np.array_equal(to_np(order[r])[:len(want)], want) and (to_np(order[r])[len(want):] == -1).all()
    t_order, t_rank, c_order, counts = _partition_pair(maps, cuda(ch))
    for r in range(rows):
        row = to_np(maps[r]).astype(np.int64)
        want = np.concatenate([np.flatnonzero(row == b) for b in (2, 4, 8, 16)])
        n_comp = int(np.isin(row, (2, 4, 8)).sum())
        assert np.array_equal(to_np(t_order[r])[:len(want)], want)
        rank = np.cumsum((row > 0) & (row != 16)) - 1                        # (every positive value but 16, as the reference counts)
        assert np.array_equal(to_np(t_rank[r])[:n_comp], rank[want[:n_comp]])
        assert to_np(counts[rows + r]).tolist() == [int((ch[r] == 2).sum()), int((ch[r] == 4).sum()), int(np.isin(ch[r], (8, 16)).sum()), 0]


@pytest.mark.parametrize("length", [1, 33, 128, 129, 256, 257, 2048, 4096, 8191, 16385, 65537])
@pytest.mark.parametrize("kind", ["lognormal", "softmax", "ties", "zeros", "negative", "tiny"])
def test_allocator_lengths(length, kind):
    """Row lengths at which a row moves from a warp to a CTA and to clusters; rows whose scores sit in a
    few buckets, on ties, at zero, below it and near the smallest numbers."""
    from oracle.ref_knapsack import knapsack_batched
    from rdkv_b200 import synth
    from rdkv_b200.knapsack_solver import knapsack_bit_allocation_batched
    gen = torch.Generator().manual_seed(length)
    s = synth.make_scores(3, length, seed=length)
    if kind == "softmax":
        s = torch.softmax(6 * torch.randn(3, length, generator=gen), dim=1)
    elif kind == "ties":
        s = torch.randint(0, 4, (3, length), generator=gen).float()
    elif kind == "zeros":
        s[:, ::3] = 0.0
    elif kind == "negative":
        s = torch.randn(3, length, generator=gen)
    elif kind == "tiny":
        s = s * 1e-37
    for budget, kw in ((2.0, {}), (torch.tensor([0.4, 3.3, 9.0]), dict(max_iters=60)),
                       (3.0, dict(bit_options=torch.tensor([2.0, 4.0, 8.0])))):
        got = knapsack_bit_allocation_batched(s.cuda(), budget.cuda() if torch.is_tensor(budget) else budget, epsilon=synth.ALLOC_EPSILON, **kw)
        want_kw = {k: (v.numpy() if torch.is_tensor(v) else v) for k, v in kw.items()}
        want = knapsack_batched(s.numpy(), budget.numpy() if torch.is_tensor(budget) else budget, synth.ALLOC_EPSILON, **want_kw)
        assert np.array_equal(to_np(got), want)


@pytest.mark.parametrize("rows", [1, 2, 16, 17])
@pytest.mark.parametrize("length", [1, 40, 128, 129, 256])
def test_short_rows_end_their_doublings_together(rows, length):
    """One CTA takes up to 16 short rows and replays the batch-wide exit of the doubling loop: rows that can
    never meet their budget alone, and next to rows that can."""
    from oracle.ref_knapsack import knapsack_batched
    from rdkv_b200 import synth
    from rdkv_b200.knapsack_solver import knapsack_bit_allocation_batched
    s = synth.make_scores(rows, length, seed=rows + length)
    s[::2] *= 1e6
    opts = torch.tensor([2., 4., 8., 16.])
    for budget in (torch.ones(rows), 1.0 + 3.0 * (torch.arange(rows) % 3).float()):
        got = knapsack_bit_allocation_batched(s.cuda(), budget.cuda(), epsilon=synth.ALLOC_EPSILON, max_iters=20, bit_options=opts)
        want = knapsack_batched(s.numpy(), budget.numpy(), synth.ALLOC_EPSILON, max_iters=20, bit_options=(2, 4, 8, 16))
        assert np.array_equal(to_np(got), want)


@pytest.mark.parametrize("length", [1, 2, 3, 1000, 32768, 40001])
def test_budgets_and_logical_bits(length):
    from oracle.ref_blockwise import logical_layer_bits
    from rdkv_b200 import _lib
    from rdkv_b200.knapsack_solver import k_average_bits_per_head, k_budgets_from_v_bits
    gen = torch.Generator().manual_seed(length)
    bits = torch.tensor([0, 0, 0, 2, 4, 8, 16])[torch.randint(0, 7, (5, length + 1), generator=gen)].cuda()
    bits[0] = 0
    for v in (bits, bits[:, 1:]):
        want = k_average_bits_per_head(777, 128, 0.37, (v > 0).sum(dim=1))
        assert torch.equal(k_budgets_from_v_bits(777, 128, 0.37, v), want)
    L, H = 2, 3
    vb = torch.tensor([0, 2, 4, 8, 16])[torch.randint(0, 5, (L, H, length), generator=gen)].cuda()
    kb = torch.tensor([0, 2, 4, 8, 16])[torch.randint(0, 5, (L, H, 128), generator=gen)].cuda()
    out = torch.empty(L, dtype=torch.int64, device="cuda")
    _lib.check(_lib.lib().rdkv_logical_bits(vb.data_ptr(), kb.data_ptr(), L, H, length, 128, out.data_ptr(), _lib.stream_ptr(out.device)), "logical")
    assert out.tolist() == [logical_layer_bits(to_np(vb[i]), to_np(kb[i]), 128) for i in range(L)]


@pytest.mark.parametrize("layers", [1, 3, 9])
@pytest.mark.parametrize("strided", [False, True])
def test_layers_of_different_shapes(layers, strided):
    """Layers whose channel counts differ go out together, a few per launch; every layer equals the
    oracle's.  Strided: keys and values as halves of one tensor, rows off 16-byte boundaries."""
    from oracle import ref_packing as RP
    from rdkv_b200 import synth
    from rdkv_b200.packing import pack_kv_layers
    H, T, g = 2, 515, 4
    Ks, Vs, vbs, kbs = [], [], [], []
    for i in range(layers):
        K, V = synth.make_kv(H, T, seed=i)
        if strided:
            both = torch.zeros(1, H, T, 259, dtype=torch.float16)
            both[..., 1:129], both[..., 130:258] = K, V
            both = both.cuda()
            Ks.append(both[..., 1:129]); Vs.append(both[..., 130:258])
        else:
            Ks.append(K.cuda()); Vs.append(V.cuda())
        vbs.append(synth.make_v_bits(H, T, 200 + 3 * i, seed=i, per_head_N=[200 + 3 * i, 5 + i]))
        kbs.append(synth.make_k_bits(H, seed=i, mix=((8, 5 + 3 * i), (4, 20 + i), (2, 30 - i))))
    batch = pack_kv_layers(Ks, Vs, torch.stack(vbs).cuda(), torch.stack(kbs).cuda(), g)
    for i, (pl, nv) in enumerate(batch):
        want, want_nv = RP.pack_kv(to_np(Ks[i]), to_np(Vs[i]), vbs[i].numpy(), kbs[i].numpy(), g)
        got = layer_to_np(pl)
        for name in ("K_2bit", "K_4bit", "K_8bit", "K_ch_scale", "K_ch_zp", "V_2bit", "V_4bit", "V_8bit", "V_scale", "V_zp",
                     "softmax_mask", "seg_bounds_per_head", "n_v16_per_head", "T_eff_per_head", "K_ch_perm_padded_idx_for_Q"):
            a, b = got[name], want[name]
            assert (a is None and b is None) or np.array_equal(a, b), (i, name)
        row = vbs[i][0].numpy()                                              # the first head's V order among its compressed tokens
        rank = np.cumsum((row > 0) & (row != 16)) - 1
        assert np.array_equal(got["sort_idx"], rank[np.concatenate([np.flatnonzero(row == b) for b in (2, 4, 8)])])
        assert np.array_equal(to_np(nv), want_nv)


@pytest.mark.parametrize("rows", [1, 15, 127, 128, 129, 300])
@pytest.mark.parametrize("mix", [((8, 24), (4, 31), (2, 27)), ((8, 1),), ((4, 2), (2, 126)), ((16, 100), (8, 28))])
def test_unpack_rows(rows, mix):
    """Row counts around the 128 rows of a CTA, K rows of odd widths, layers of different lengths in one
    launch (17: more than one launch takes)."""
    from oracle import ref_packing as RP
    from rdkv_b200 import synth
    from rdkv_b200.decompress import unpack_k_mixed, unpack_trizone_to_past_kv
    from rdkv_b200.packing import TriZoneCache, pack_kv
    H, g = 2, 2
    pairs, wants = [], []
    for i in range(17 if rows == 129 else 2):
        T = rows + 9 + i
        K, V = synth.make_kv(H, T, seed=i)
        vb = synth.make_v_bits(H, T, rows, seed=i, per_head_N=[rows, max(1, rows - 2 * i - 1)])
        kb = synth.make_k_bits(H, seed=i, mix=mix)
        pairs.append(pack_kv(K.cuda(), V.cuda(), vb.cuda(), kb.cuda(), g))
        want, want_nv = RP.pack_kv(K.numpy(), V.numpy(), vb.numpy(), kb.numpy(), g)
        wants.append((RP.unpack_k(want, 128), RP.unpack_v(want, want_nv, 128)))
    none = [None] * len(pairs)
    cache = TriZoneCache(tuple(p for p, _ in pairs), [v for _, v in pairs], none, none, 0)
    for (k, v), (pl, _), (want_k, want_v) in zip(unpack_trizone_to_past_kv(cache, head_dim=128), pairs, wants):
        assert np.array_equal(to_np(k).view(np.uint16), want_k.view(np.uint16))
        assert np.array_equal(to_np(v).view(np.uint16), want_v.view(np.uint16))
        assert torch.equal(unpack_k_mixed(pl, 128), k)


@pytest.mark.parametrize("n8", [300, 365, 366, 383, 384, 450])
def test_unpack_wide_rows(n8):
    """K rows packed for larger channel targets than a head has channels: up to the widest that the
    128-channel kernel has shared memory for, and wider ones, which the general kernel takes."""
    from rdkv_b200.decompress import unpack_k_mixed
    from rdkv_b200.packing import PackedKVLayer, pack_k_mixed
    H, T = 2, 131
    K = torch.randn(1, H, T, 128, generator=torch.Generator().manual_seed(n8)).half().cuda()
    bits = torch.full((128,), 8, device="cuda")
    none = torch.empty(1, H, 0, 1, dtype=torch.float16, device="cuda")

    def unpacked(target):
        k2, k4, k8, scale, zp, sort_idx, perm, (_, _, n) = pack_k_mixed(K, bits, n_ch_8_target=target)
        assert n == 128 and k8.shape[-1] == target
        layer = PackedKVLayer(k2, k4, k8, scale, zp, sort_idx, (0, 0, target), perm, None, None, None, none, none, sort_idx[:0],
                              (0, 0, 0), 0, T_eff_k=T, K_ch_sort_idx_per_head=sort_idx.repeat(H, 1),
                              K_ch_seg_bounds_per_head=torch.tensor([[0, 0, 128]] * H, dtype=torch.int32, device="cuda"))
        return unpack_k_mixed(layer, 128)

    assert torch.equal(unpacked(n8), unpacked(128))


@pytest.mark.parametrize("dtype", [torch.int16, torch.int32, torch.float32])
def test_bit_maps_of_other_types_and_strides(dtype):
    """Maps that are not contiguous 64-bit integers give what the same maps as such give: the bits a packed
    layer stands for, the layers themselves, the K budgets."""
    from rdkv_b200 import synth
    from rdkv_b200.knapsack_solver import k_budgets_from_v_bits
    from rdkv_b200.packing import pack_selected
    H, T, g, L = 2, 203, 4, 2
    K, V, vb, kb = [], [], [], []
    for i in range(L):
        k, v = synth.make_kv(H, T, seed=i)
        K.append(k.cuda()); V.append(v.cuda())
        vb.append(synth.make_v_bits(H, T, 90, seed=i).to(torch.int64).cuda())
        kb.append(synth.make_k_bits(H, seed=i).to(torch.int64).cuda())

    def fields(pairs):
        return [t for pl, v16 in pairs for t in (pl.K_2bit, pl.K_4bit, pl.K_8bit, pl.V_2bit, pl.V_4bit, pl.V_8bit, v16,
                                                 pl.allocation_v_bits, pl.allocation_k_bits)]

    want, want_bits = pack_selected(K, V, vb, kb, g)
    budgets = k_budgets_from_v_bits(60, 128, 0.5, vb[0])
    for change in (lambda m: m.to(dtype), lambda m: m.to(dtype).t().contiguous().t(), lambda m: m.t().contiguous().t()):
        got, got_bits = pack_selected(K, V, [change(m) for m in vb], [change(m) for m in kb], g)
        assert torch.equal(got_bits, want_bits)
        assert all(torch.equal(a, b) for a, b in zip(fields(got), fields(want)))
        assert torch.equal(k_budgets_from_v_bits(60, 128, 0.5, change(vb[0])), budgets)


@pytest.mark.parametrize("k_passes", [0, 1, 3])
def test_pass_choice_for_layers_of_different_shapes(k_passes):
    """Layers with tensors of their own take every ``k_passes``, also 1 where their rows do not fit a cluster's
    shared memory; the bytes are the same."""
    from rdkv_b200 import synth
    from rdkv_b200.packing import pack_kv, pack_kv_layers
    H, T, g = 1, 26000, 2
    Ks, Vs, vbs, kbs = [], [], [], []
    for i in range(2):
        K, V = synth.make_kv(H, T, seed=i)
        Ks.append(K.cuda()); Vs.append(V.cuda())
        vbs.append(synth.make_v_bits(H, T, 25000, seed=i).cuda())
        kbs.append(synth.make_k_bits(H, seed=i, mix=((8, 30 + i), (4, 40), (2, 30))).cuda())
    batch = pack_kv_layers(Ks, Vs, torch.stack(vbs), torch.stack(kbs), g, build_mask=False, k_passes=k_passes)
    for i, (pl, _) in enumerate(batch):
        want, _ = pack_kv(Ks[i], Vs[i], vbs[i], kbs[i], g, build_mask=False)
        for name in ("K_2bit", "K_4bit", "K_8bit", "K_ch_scale", "K_ch_zp"):
            assert torch.equal(getattr(pl, name), getattr(want, name)), name


@pytest.mark.parametrize("tokens,window,g", [(33, 32, 4), (128, 8, 4), (129, 16, 8), (1000, 32, 8), (5000, 5, 3)])
@pytest.mark.parametrize("causal", [True, False])
def test_normalised_window_scores(tokens, window, g, causal):
    """The division by the window positions that see a key, inside the second pass: the fp32 quotient of the
    plain call's scores, for tiles of 128 keys that end inside the window and windows staged by plain loads."""
    from rdkv_b200.scoring import obs_window_scores
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    q = torch.randn(1, 2 * g, window, 128, generator=gen, device="cuda").half()
    k = torch.randn(1, 2, tokens, 128, generator=gen, device="cuda").half()
    plain, channel = obs_window_scores(q, k, causal=causal, check_status=True)
    token, channel_n = obs_window_scores(q, k, causal=causal, normalise=True, check_status=True)
    seen = torch.full((tokens,), float(window), device="cuda")
    if causal:
        seen[tokens - window:] = torch.arange(window, 0, -1, device="cuda", dtype=torch.float32)
    assert torch.equal(token, plain / seen) and torch.equal(channel, channel_n)
