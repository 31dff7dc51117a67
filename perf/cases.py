"""Performance cases of the packed-KV path: what a serving program has the library do.

A prompt is prefilled: every layer's tokens and channels are scored from the observation window
(``obs_window_scores``), bits are allotted (``knapsack_bit_allocation_batched``) and the layer is packed
(``select_and_pack``, or ``pack_kv_layers`` where the bits are at hand).  Then tokens are decoded against
the packed cache: layer by layer inside a model (``packed_decode_attention`` with the uncompressed tail,
the new token and the rotary embedding), all layers at once, from host buffers, or through the two
separate K-side and V-side operators.  Blocks of decoded tokens are compressed again
(``compress_block``), and a cache can be turned back into fp16 keys and values
(``unpack_trizone_to_past_kv``).

Shapes are those of the repository's configurations: 8 KV heads (fewer on a rank of a sharded model)
with 4 or 8 query heads each, head_dim 128, contexts up to 131072, budgets of 256 to 8192 kept tokens a
head.  ``ragged`` caches have what the bit allocator leaves in earnest: another number of kept tokens in
every head and other channel counts in every head; the others have the configurations' fixed mix.
How many elements get how many bits belongs to the case (it decides the shapes of the results); which
ones they are, and all values, come from the seed.
"""
import math

import numpy as np
import torch

from rdkv_b200 import synth
from rdkv_b200.blockwise import BlockwiseRDKVConfig, compress_block
from rdkv_b200.decode import DecodeTable, packed_decode_attention, packed_decode_attention_host
from rdkv_b200.decompress import unpack_trizone_to_past_kv
from rdkv_b200.k_kernel import k_mixed_qk_dot_into
from rdkv_b200.knapsack_solver import (DEFAULT_EPSILON_K, DEFAULT_EPSILON_V, k_average_bits_per_head,
                                       knapsack_bit_allocation_batched)
from rdkv_b200.packing import TriZoneCache, pack_kv, pack_kv_layers, select_and_pack
from rdkv_b200.scoring import obs_window_scores
from rdkv_b200.v_kernel import v_dequant_weighted_sum_dispatch_into

D = 128
DEV = "cuda"
DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
PACKED_FIELDS = ("K_2bit", "K_4bit", "K_8bit", "K_ch_scale", "K_ch_zp", "K_ch_perm_padded_idx_for_Q",
                 "V_2bit", "V_4bit", "V_8bit", "V_scale", "V_zp", "seg_bounds_per_head", "n_v16_per_head")


# ── the cases ────────────────────────────────────────────────────────────────

def listed():
    return [
        # One token of one sequence in one layer: what an interactive chat pays 32 times per token.  The
        # smallest call; latency, launches and host work are all there is.
        dict(name="block_b1", op="block", batch=1, heads=8, gqa=4, kept=1024, tail=37, ragged=True, dtype="fp16"),
        # The same for a batch of 16 sequences at different positions: a server's inner loop.
        dict(name="block_b16", op="block", batch=16, heads=8, gqa=4, kept=2048, tail=517, ragged=True, dtype="bf16"),
        # All 32 layers of 16 sequences in one launch (the benchmark's decode step).
        dict(name="step_32x16", op="step", views=512, heads=8, gqa=4, kept=2048, ragged=False, dtype="bf16"),
        # Long contexts of a 72B model, 80 layers of 4 sequences, heads as the allocator leaves them.
        dict(name="step_80x4_long", op="step", views=320, heads=8, gqa=8, kept=8192, ragged=True, dtype="bf16"),
        # Queries and results in pinned host memory (a scheduler on the host): 32 layers of 4 sequences.
        dict(name="host_32x4", op="host", views=128, heads=8, gqa=4, kept=2048, ragged=False, dtype="bf16"),
        # The drop-in pair of operators with the caller's own mask and softmax between them.
        dict(name="two_stage", op="two_stage", heads=8, gqa=4, kept=2048, ragged=True, dtype="fp16"),
        # Prefill of one layer: scores of a 32K prompt from a window of 32 queries.
        dict(name="obs_32k", op="obs", tokens=32768, heads=8, gqa=4, window=32, dtype="fp16"),
        # Bit allocation of 32 layers x 8 heads at 32K tokens, and of their K channels.
        dict(name="alloc_256x32k", op="alloc", rows=256, tokens=32768, bits=2.0),
        # Prefill of one layer: pool, allot, pack (the call a prefill loop makes per layer).
        dict(name="select_32k", op="select", tokens=32768, heads=8, gqa=4, budget=2048),
        # Packing of the layers of a long prompt whose bits are at hand (a pipeline stage of four layers).
        dict(name="pack_4x128k", op="pack", layers=4, tokens=131072, heads=8, gqa=4, kept=8192, ragged=True),
        # A cache handed back to plain attention code.
        dict(name="unpack_16", op="unpack", layers=16, heads=8, gqa=4, kept=2048, ragged=True),
        # A finished block of 64 decoded tokens compressed in four layers: the smallest encode call.
        dict(name="recompress_64", op="recompress", layers=4, tokens=64, heads=8, gqa=4, budget=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["block", "block", "step", "host", "two_stage", "obs", "alloc", "select", "pack", "unpack", "recompress"])
    heads, gqa = rng.choice([8, 8, 4, 2]), rng.choice([4, 8])
    case = dict(op=op, heads=heads, gqa=gqa)
    if op == "block":
        case.update(batch=_log_int(rng, 1, 64), kept=_log_int(rng, 256, 8192), tail=rng.randint(0, 1023),
                    ragged=rng.random() < 0.75, dtype=rng.choice(["fp16", "bf16"]))
    elif op in ("step", "host"):
        kept = _log_int(rng, 256, 8192)
        most = min(512, 320 * 8192 * 8 // (kept * heads)) if op == "step" else min(128, 128 * 2048 * 8 // (kept * heads))
        case.update(views=_log_int(rng, 16, max(17, most)), kept=kept, ragged=rng.random() < 0.5, dtype=rng.choice(["fp16", "bf16"]))
    elif op == "two_stage":
        case.update(kept=_log_int(rng, 256, 8192), ragged=rng.random() < 0.75, dtype=rng.choice(["fp16", "bf16"]))
    elif op == "obs":
        case.update(tokens=_log_int(rng, 1024, 131072), window=rng.choice([8, 16, 32, 32]), dtype=rng.choice(["fp16", "bf16"]))
    elif op == "alloc":
        rows = rng.choice([8, 64, 256, 640])
        del case["heads"], case["gqa"]
        case.update(rows=rows, tokens=_log_int(rng, 1024, min(131072, 256 * 32768 // rows)), bits=round(rng.uniform(0.5, 4.0), 2))
    elif op == "select":
        tokens = _log_int(rng, 1024, 131072)
        case.update(tokens=tokens, budget=max(64, int(tokens * rng.uniform(0.03, 0.25))))
    elif op == "pack":
        tokens = _log_int(rng, 2048, 131072)
        case.update(layers=max(1, min(4, 4 * 131072 * 8 // (tokens * heads))), tokens=tokens,
                    kept=max(128, int(tokens * rng.uniform(0.05, 0.25))), ragged=rng.random() < 0.75)
    elif op == "unpack":
        kept = _log_int(rng, 256, 8192)
        case.update(layers=rng.choice([4, 8, 16, 32]) if kept < 4096 else 4, kept=kept, ragged=rng.random() < 0.75)
    else:
        tokens = rng.choice([64, 128])
        case.update(layers=rng.randint(1, 4), tokens=tokens, budget=rng.randint(tokens // 8, tokens // 2))
    return case


# ── inputs ───────────────────────────────────────────────────────────────────

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _kv(heads, tokens, gen):
    """Keys with four outlier channels a head, values; fp16 (the configurations' distributions)."""
    K = torch.randn(1, heads, tokens, D, generator=gen, device=DEV)
    V = torch.randn(1, heads, tokens, D, generator=gen, device=DEV)
    ch = (torch.arange(heads, device=DEV)[:, None] * 16 + torch.tensor(synth.OUTLIER_BASE, device=DEV)) % D
    gain = torch.ones(heads, D, device=DEV).scatter_(1, ch, 10.0)
    return (K * gain[None, :, None, :]).half(), V.half()


def _bits_by_rank(scores, counts):
    """Bits handed out by descending score: ``counts`` [rows, 4] elements of 16, 8, 4 and 2 bits."""
    rank = torch.argsort(torch.argsort(scores, dim=1, descending=True), dim=1)
    edges = torch.as_tensor(np.cumsum(counts, axis=1), device=scores.device)
    widths = torch.tensor([16, 8, 4, 2, 0], device=scores.device)
    return widths[(rank[:, :, None] >= edges[:, None, :]).sum(dim=2)]


def _bit_maps(rng, gen, heads, tokens, kept, ragged):
    """(v_bits [heads, tokens], k_bits [heads, 128]), int64 as the allocator returns them.  ``rng`` gives
    the counts, ``gen`` the places."""
    n = np.full(heads, kept) if not ragged else rng.integers(max(1, kept * 3 // 4), kept + 1, heads)
    if ragged:
        share = np.stack([np.full(heads, 1 / 8), rng.uniform(0.15, 0.35, heads), rng.uniform(0.3, 0.45, heads)], axis=1)
        k_counts = np.stack([np.zeros(heads), rng.integers(8, 25, heads), rng.integers(16, 33, heads), rng.integers(12, 37, heads)], axis=1)
    else:
        share = np.tile([1 / 8, 1 / 4, 3 / 8], (heads, 1))
        k_counts = np.tile([0, 16, 24, 24], (heads, 1))
    v_counts = np.floor(share * n[:, None]).astype(np.int64)
    v_counts = np.concatenate([v_counts, (n - v_counts.sum(axis=1))[:, None]], axis=1)
    tok = torch.randn(heads, tokens, generator=gen, device=DEV)
    ch = torch.randn(heads, D, generator=gen, device=DEV)
    return _bits_by_rank(tok, v_counts), _bits_by_rank(ch, k_counts.astype(np.int64))


def _packed(views, heads, gqa, kept, ragged, seed, mask=False):
    """Packed layers of ``views`` (sequence, layer) pairs.  The context is only a little longer than what
    is kept of it: evicted tokens leave no trace in a packed cache."""
    gen, rng = _gen(seed), np.random.default_rng([heads, kept])
    tokens = kept + kept // 8 + 16
    layers, values = [], []
    for at in range(0, views, 8):
        some = [_kv(heads, tokens, gen) + _bit_maps(rng, gen, heads, tokens, kept, ragged) for _ in range(min(8, views - at))]
        if ragged:
            pairs = [pack_kv(k, v, vb, kb, gqa, build_mask=mask) for k, v, vb, kb in some]
        else:
            K, V, vb, kb = zip(*some)
            pairs = list(pack_kv_layers(K, V, torch.stack(vb), torch.stack(kb), gqa, build_mask=mask))
        for pl, nv in pairs:
            layers.append(pl)
            values.append(nv)
    return layers, values


def _token_scores(rng, gen, heads, tokens):
    """Lognormal token scores in clusters of 64 tokens whose order the seed chooses.  A cluster starts and
    ends with a few tokens that hardly count, so that pooling does not mix neighbouring clusters and
    every order leads to the same counts of bits."""
    n = -(-tokens // 64)
    scores = np.exp(1.5 * rng.standard_normal((heads, n, 64)))
    scores[:, :, :4] = scores[:, :, -4:] = 1e-3
    scores[:, -1, tokens - 64 * (n - 1) - 4:] = 1e-3       # (the last, cut cluster stays where it is)
    order = torch.argsort(torch.rand(heads, n - 1, generator=gen, device=DEV), dim=1)
    scores = torch.from_numpy(scores).float().to(DEV)
    moved = torch.gather(scores[:, :-1], 1, order[:, :, None].expand(-1, -1, 64))
    return torch.cat([moved, scores[:, -1:]], dim=1).reshape(heads, -1)[:, :tokens].contiguous()


def _queries(shape, gen, dtype):
    return (torch.randn(*shape, generator=gen, device=DEV) / D ** 0.5 * 4).to(dtype)


def prepare(case, seed):
    op, s = case["op"], dict(op=case["op"])
    heads, gqa = case.get("heads"), case.get("gqa")
    gen = _gen(seed + 1)
    dtype = DTYPES.get(case.get("dtype"))
    if op in ("block", "step", "host"):
        views = case["batch"] if op == "block" else case["views"]
        layers, values = _packed(views, heads, gqa, case["kept"], case["ragged"], seed)
        s["table"] = DecodeTable(layers, values, heads * gqa)
        s["q"] = _queries((views, heads * gqa, D), gen, dtype)
        s["out"] = torch.empty(views, heads * gqa, D, device=DEV)
    if op == "host":
        s["q"], s["out"] = s["q"].cpu().pin_memory(), torch.empty(s["out"].shape).pin_memory()
    if op == "block":
        views, cap = case["batch"], (case["tail"] // 64 + 1) * 64
        s["new_k"], s["new_v"] = (torch.randn(views, heads, cap, D, generator=gen, device=DEV).to(dtype) for _ in range(2))
        s["k_cur"], s["v_cur"] = (torch.randn(views, heads, D, generator=gen, device=DEV).to(dtype) for _ in range(2))
        # sequences of a batch are at positions of their own: live tail rows per view on the device
        s["n_new"] = case["tail"] if views == 1 else torch.randint(case["tail"] // 2, case["tail"] + 1, (views,), generator=gen,
                                                                   device=DEV, dtype=torch.int32)
        angle = torch.randint(1000, 30000, (views, 1), generator=gen, device=DEV) * (
            5e5 ** (-torch.arange(D // 2, device=DEV) / (D // 2)))
        s["rope"] = (torch.cos(angle), torch.sin(angle))
    elif op == "two_stage":
        (layer,), (v16,) = _packed(1, heads, gqa, case["kept"], case["ragged"], seed, mask=True)
        s.update(layer=layer, v16=None if v16 is None else v16[0], q=_queries((heads * gqa, D), gen, dtype),
                 scores=torch.zeros(heads * gqa, layer.T_eff_k, device=DEV), out=torch.empty(heads * gqa, D, device=DEV))
    elif op == "obs":
        k, _ = _kv(heads, case["tokens"], gen)
        s.update(q=torch.randn(1, heads * gqa, case["window"], D, generator=gen, device=DEV).to(dtype), k=k.to(dtype))
    elif op == "alloc":
        s.update(v=synth.make_scores(case["rows"], case["tokens"], seed=seed, device=DEV),
                 k=synth.make_scores(case["rows"], D, seed=seed + 1, device=DEV), bits=case["bits"], budget=case["tokens"] // 8)
    elif op == "select":
        k, v = _kv(heads, case["tokens"], gen)
        rng = np.random.default_rng([heads, case["tokens"]])
        channel = torch.from_numpy(np.exp(1.5 * rng.standard_normal((heads, D)))).float().to(DEV)
        order = torch.argsort(torch.rand(heads, D, generator=gen, device=DEV), dim=1)
        s.update(k=k, v=v, token=_token_scores(rng, gen, heads, case["tokens"]), channel=torch.gather(channel, 1, order),
                 gqa=gqa, budget=case["budget"])
    elif op == "pack":
        rng = np.random.default_rng([heads, case["kept"]])
        kv = [_kv(heads, case["tokens"], gen) for _ in range(case["layers"])]
        maps = [_bit_maps(rng, gen, heads, case["tokens"], case["kept"], case["ragged"]) for _ in kv]
        s.update(K=[k for k, _ in kv], V=[v for _, v in kv], v_bits=torch.stack([a for a, _ in maps]),
                 k_bits=torch.stack([b for _, b in maps]), gqa=gqa)
    elif op == "unpack":
        layers, values = _packed(case["layers"], heads, gqa, case["kept"], case["ragged"], seed)
        none = [None] * len(layers)
        s["cache"] = TriZoneCache(tuple(layers), values, none, none, 4 * case["kept"])
    elif op == "recompress":
        T = case["tokens"]
        # keys, queries and token scores that lead to the case's counts; the seed chooses the heads'
        # order, the channels' signs and the values
        base = _gen(heads * T)
        s["kv"], s["queries"], s["token"] = [], [], []
        for i in range(case["layers"]):
            order = torch.randperm(heads, generator=gen, device=DEV)
            sign = torch.randint(0, 2, (heads, 1, D), generator=gen, device=DEV) * 2 - 1
            k, _ = _kv(heads, T, base)
            v = torch.randn(1, heads, T, D, generator=gen, device=DEV).half()
            q = torch.randn(heads, gqa * T, D, generator=base, device=DEV).half()
            s["kv"].append(torch.cat([(k[:, order] * sign).half(), v], dim=3))
            s["queries"].append((q[order] * sign).half().reshape(heads * gqa, T, D))
            s["token"].append(synth.make_scores(heads, T, seed=T + i, device=DEV)[order])
        s["config"] = BlockwiseRDKVConfig(block_size=T, block_budget_tokens=case["budget"], k_budget_ratio=0.5, obs_window=32,
                                          pool_kernel_size=5, pool_padding="reflect", v_bit_options=None, k_bit_options=None,
                                          epsilon_v=DEFAULT_EPSILON_V, epsilon_k=DEFAULT_EPSILON_K)
        s["gqa"] = gqa
    return s


# ── one pass ─────────────────────────────────────────────────────────────────

def _layer_outputs(layer, v16):
    return [getattr(layer, f) for f in PACKED_FIELDS] + [v16]


def run(s):
    op = s["op"]
    if op == "block":
        out = packed_decode_attention(s["q"], s["table"], out=s["out"], new_k=s["new_k"], new_v=s["new_v"], n_new=s["n_new"],
                                      k_cur=s["k_cur"], v_cur=s["v_cur"], rope=s["rope"])
        return out, s["new_k"], s["new_v"]                 # (the new token's rows were appended)
    if op == "step":
        return packed_decode_attention(s["q"], s["table"], out=s["out"])
    if op == "host":
        return packed_decode_attention_host(s["q"], s["table"], s["out"])
    if op == "two_stage":
        layer, scores = s["layer"], s["scores"]
        k_mixed_qk_dot_into(s["q"], layer, layer.T_eff_k, scores)
        weights = torch.softmax(scores + layer.softmax_mask, dim=-1)
        v_dequant_weighted_sum_dispatch_into(weights, layer, s["out"], V16=s["v16"], n_v16_per_head=layer.n_v16_per_head,
                                             max_T_v=layer.T_eff)
        return weights, s["out"]
    if op == "obs":
        return obs_window_scores(s["q"], s["k"], normalise=True)
    if op == "alloc":
        v_bits = knapsack_bit_allocation_batched(s["v"], s["bits"], epsilon=synth.ALLOC_EPSILON, max_iters=60)
        kept = (v_bits > 0).sum(dim=1)
        k_bits = knapsack_bit_allocation_batched(s["k"], k_average_bits_per_head(s["budget"], D, 0.5, kept),
                                                 epsilon=synth.ALLOC_EPSILON, max_iters=60)
        return v_bits, k_bits
    if op == "select":
        layer, v16, t_eff = select_and_pack(s["k"], s["v"], s["token"], s["channel"], gqa_factor=s["gqa"],
                                            token_budget=s["budget"], k_budget_ratio=0.5)
        return _layer_outputs(layer, v16) + [layer.softmax_mask, layer.sort_idx, layer.K_ch_sort_idx_per_head, t_eff]
    if op == "pack":
        batch = pack_kv_layers(s["K"], s["V"], s["v_bits"], s["k_bits"], s["gqa"])
        return [_layer_outputs(*batch[i]) + [batch[i][0].softmax_mask] for i in range(len(batch))]
    if op == "unpack":
        return unpack_trizone_to_past_kv(s["cache"], head_dim=D)
    block = compress_block(target_kv=s["kv"], query_block=s["queries"], token_scores_by_layer=s["token"], block_id=0,
                           token_start=0, token_end=s["kv"][0].shape[2] - 1, config=s["config"], num_kv_groups=s["gqa"])
    return [_layer_outputs(pl, nv) for pl, nv in zip(block.packed, block.new_v_only)], block.logical_bits_per_layer


# ── what a pass cannot do without ────────────────────────────────────────────

def _cache_bytes(heads, kept, ragged):
    """Packed bytes of one (sequence, layer): K codes 34 and V rows 99.5 bytes a kept token on average
    (the fixed mix; ragged heads keep 7/8 of ``kept`` on average)."""
    n = kept * 7 / 8 if ragged else kept
    return heads * (n * 133.5 + 256)


def work(case):
    op, heads, gqa = case["op"], case.get("heads"), case.get("gqa")
    if op in ("block", "step", "host", "two_stage"):
        views = {"block": case.get("batch"), "two_stage": 1}.get(op) or case["views"]
        n = case["kept"] * (7 / 8 if case["ragged"] else 1)
        tail = case.get("tail", 0) * (1 if views == 1 else 0.75)
        moved = views * (_cache_bytes(heads, case["kept"], case["ragged"]) + heads * (tail * 512 + 1024 * (op == "block")))
        moved += views * heads * gqa * D * 6               # 16-bit queries in, fp32 results out
        if op == "two_stage":
            moved += 4 * heads * gqa * n * 4               # scores out and in, weights out and in
        return {"bytes": moved, "flops": views * heads * gqa * (2 * n * 64 + 2 * n * D + 4 * tail * D)}
    if op == "obs":
        T = case["tokens"]
        return {"bytes": heads * T * D * 2 + heads * gqa * case["window"] * D * 2 + heads * (T + D) * 4,
                "flops": 2.0 * heads * gqa * case["window"] * T * D}
    if op == "alloc":
        return {"bytes": case["rows"] * (case["tokens"] + D) * 12, "flops": 0}
    if op == "select":
        T = case["tokens"]
        kept = min(T, 6 * case["budget"])                  # (at 2 and 4 bits a token keeps far more than the budget's fp16 tokens)
        return {"bytes": heads * (T * 4 + kept * 512 + kept * 90), "flops": 0}
    if op == "pack":
        n = case["kept"] * (7 / 8 if case["ragged"] else 1)
        return {"bytes": case["layers"] * heads * (case["tokens"] * 8 + n * 512 + n * 133.5), "flops": 0}
    if op == "unpack":
        n = case["kept"] * (7 / 8 if case["ragged"] else 1)
        return {"bytes": case["layers"] * heads * (n * 133.5 + case["kept"] * 512), "flops": 0}
    T = case["tokens"]
    return {"bytes": case["layers"] * heads * (T * 512 + gqa * T * 256 + T * 120), "flops": 0}


def tolerance(case):
    """About four times what the path differs by from the same formula in fp64 (decode: on the dequantised
    cache) or from torch's own 16-bit matmul and softmax (scores), over the ranges above."""
    if case["op"] in ("block", "step", "host"):
        return {"rel": 1.6e-3, "max": 2e-2}                # softmax weights and V scales meet as fp16 products
    if case["op"] == "two_stage":
        return {"rel": 6e-3, "max": 2.5e-2}                # weights far below 1 as fp16 operands
    if case["op"] == "obs":                                # scores and weights are rounded to the inputs' type
        return {"rel": 1e-4, "max": 4e-3} if case["dtype"] == "fp16" else {"rel": 1.4e-3, "max": 3e-2}
    return "exact"                                         # packed bytes, parameters, bit choices, fp16 rows


# ── the same results in 64 bits ──────────────────────────────────────────────

def _codes(packed, bits):
    """Codes of packed rows [..., bytes] -> [..., bytes * 8 / bits]: part i of the columns holds the bits
    from i * bits on of every byte."""
    return torch.cat([(packed >> (bits * i)) & (2 ** bits - 1) for i in range(8 // bits)], dim=-1).double()


def _dense(layer, v16, gqa):
    """[(keys [n, 128], values [n, 128])] of the layer's heads, live rows only, from its packed bytes."""
    heads, T_v = layer.K_ch_scale.shape[1], layer.T_eff
    parts = [_codes(t[0], b) for t, b in ((layer.K_2bit, 2), (layer.K_4bit, 4), (layer.K_8bit, 8)) if t is not None]
    slots = (torch.cat(parts, dim=-1) - layer.K_ch_zp[0].double()) * layer.K_ch_scale[0].double()
    out = []
    for h, ((n2, n4, n8), n16) in enumerate(zip(layer.seg_bounds_per_head.tolist(), layer.n_v16_per_head.tolist())):
        keys = torch.zeros(slots.shape[1], D, dtype=torch.float64, device=DEV)
        keys.index_add_(1, layer.K_ch_perm_padded_idx_for_Q[h * gqa], slots[h])
        n = n2 + n4 + n8
        rows = [_codes(t[0, h, :m], b) for t, m, b in ((layer.V_2bit, n2, 2), (layer.V_4bit, n4, 4), (layer.V_8bit, n8, 8)) if m]
        values = (torch.cat(rows) - layer.V_zp[0, h, :n].double()) * layer.V_scale[0, h, :n].double() if rows else keys[:0]
        if n16:
            values = torch.cat([values, v16[0, h, :n16].double()])
        out.append((torch.cat([keys[:n], keys[T_v:T_v + n16]]), values))
    return out


def _rotated(x, cos, sin):
    lo, hi = x[..., :D // 2], x[..., D // 2:]
    return torch.cat([lo * cos - hi * sin, hi * cos + lo * sin], dim=-1)


def _exact_decode(s, gqa):
    table, q = s["table"], s["q"].to(DEV).double()
    out = torch.empty(q.shape, dtype=torch.float64, device=DEV)
    for i, (layer, v16) in enumerate(table.source):
        qi = q[i]
        if "rope" in s:
            cos, sin = (t[i].double() for t in s["rope"])
            qi, k_cur = _rotated(qi, cos, sin), _rotated(s["k_cur"][i].double(), cos, sin)
            n_new = int(s["n_new"]) if not torch.is_tensor(s["n_new"]) else int(s["n_new"][i])
        for h, (keys, values) in enumerate(_dense(layer, v16, gqa)):
            if "rope" in s:
                keys = torch.cat([keys, s["new_k"][i, h, :n_new].double(), k_cur[h:h + 1]])
                values = torch.cat([values, s["new_v"][i, h, :n_new].double(), s["v_cur"][i, h:h + 1].double()])
            at = slice(h * gqa, (h + 1) * gqa)
            out[i, at] = torch.softmax(qi[at] @ keys.T / D ** 0.5, dim=-1) @ values
    return out


def exact(case, seed):
    """What ``run`` returns for ``prepare(case, seed)``, from the packed bytes (decode) or the inputs (scores) in
    64 bits; None where the outputs are whole numbers, bytes and the fp16 parameters that go with them."""
    op, gqa = case["op"], case.get("gqa")
    if op not in ("block", "step", "host", "two_stage", "obs"):
        return None
    s = prepare(case, seed)
    if op == "obs":
        q, k = s["q"].double(), s["k"].double()
        heads, W, T = k.shape[1], q.shape[2], k.shape[2]
        token = torch.empty(1, heads, T, dtype=torch.float64, device=DEV)
        unseen = torch.arange(T, device=DEV) > (T - W + torch.arange(W, device=DEV))[:, None]
        for h in range(heads):
            scores = (q[0, h * gqa:(h + 1) * gqa] @ k[0, h].T / D ** 0.5).masked_fill(unseen, float("-inf"))
            token[0, h] = torch.softmax(scores, dim=-1).sum(dim=(0, 1)) / (~unseen).sum(dim=0)
        channel = q.reshape(1, heads, -1, D).square().mean(dim=2) * k.square().mean(dim=2)
        return token, channel
    if op == "two_stage":
        layer, T_v = s["layer"], s["layer"].T_eff
        weights = torch.zeros(s["scores"].shape, dtype=torch.float64, device=DEV)
        out = torch.empty(s["out"].shape, dtype=torch.float64, device=DEV)
        for h, (keys, values) in enumerate(_dense(layer, None if s["v16"] is None else s["v16"][None], gqa)):
            at, n = slice(h * gqa, (h + 1) * gqa), int(layer.seg_bounds_per_head[h].sum())
            w = torch.softmax(s["q"][at].double() @ keys.T / D ** 0.5, dim=-1)
            weights[at, :n], weights[at, T_v:T_v + w.shape[1] - n] = w[:, :n], w[:, n:]
            out[at] = w @ values
        return weights, out
    out = _exact_decode(s, gqa)
    return (out, None, None) if op == "block" else out
