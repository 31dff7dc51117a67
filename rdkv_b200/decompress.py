"""Packed cache -> fp16 (K, V): drop-ins for the reference's decompressor.

Mirrors ``unpack_k_mixed`` (obkv_accel/packing.py:581-709), ``unpack_v_segment``
(:1427-1444) and ``unpack_trizone_to_past_kv`` with its helpers
(obkv_accel/trizone_decompress.py:43-333): same names, arguments and results, computed
by one CUDA launch per call for one layer (``rdkv_unpack_layer``) and per 16 layers of a
cache (``rdkv_unpack_layers``).  Tensors must be on a CUDA device.
"""
from __future__ import annotations

import ctypes as C
from typing import List, Optional, Tuple

import torch
from torch import Tensor

from ._lib import LayerView, UnpackJob, check, lib, ptr, require_cuda, stream_ptr
from .packing import PackedKVLayer, TriZoneCache, _squeeze_h, layer_view


def _is_perhead_layout(pl: PackedKVLayer) -> bool:
    """True when ``pl`` came out of ``_pad_and_stack_per_head_layers`` (trizone_decompress.py:86-88)."""
    return pl.seg_bounds_per_head is not None


def _launch(view: LayerView, H_kv: int, D: int, rows: int, device, *, want_k: bool, want_v: bool,
            sort_idx: Optional[Tensor] = None, sort_stride: int = 0, ch_counts: Optional[Tensor] = None,
            n_ch=(0, 0, 0)) -> Tuple[Optional[Tensor], Optional[Tensor]]:
    k_out = torch.empty((1, H_kv, rows, D), dtype=torch.float16, device=device) if want_k else None
    v_out = torch.empty((1, H_kv, rows, D), dtype=torch.float16, device=device) if want_v else None
    if rows > 0:
        check(lib().rdkv_unpack_layer(C.byref(view), H_kv, D, ptr(sort_idx), sort_stride, ptr(ch_counts),
                                      int(n_ch[0]), int(n_ch[1]), int(n_ch[2]), ptr(k_out), ptr(v_out),
                                      rows * D, rows, stream_ptr(device)), "rdkv_unpack_layer")
    return k_out, v_out


def _k_channel_maps(pl: PackedKVLayer):
    """(sort_idx int64, head stride, per-head counts int32 or None, shared counts)."""
    n_ch = tuple(int(x) for x in pl.K_ch_seg_bounds)
    if pl.K_ch_seg_bounds_per_head is not None:
        assert pl.K_ch_sort_idx_per_head is not None, "per-head layout requires K_ch_sort_idx_per_head"
        si = pl.K_ch_sort_idx_per_head.to(torch.int64).contiguous()
        cnt = pl.K_ch_seg_bounds_per_head.to(torch.int32).contiguous()
        return si, si.stride(0), cnt, n_ch
    si = pl.K_ch_sort_idx
    if si is None or si.numel() == 0:
        return None, 0, None, n_ch
    return si.to(torch.int64).contiguous(), 0, None, n_ch


def unpack_k_mixed(packed: PackedKVLayer, D: int) -> Tensor:
    """Reverse of pack_k_mixed / pack_k_mixed_per_head: ``[1, H_kv, T_eff, D]`` fp16 with the kept
    channels scattered back to their original positions and zeros elsewhere (packing.py:581-709)."""
    if packed.K_ch_scale is None:
        raise ValueError("unpack_k_mixed: K_ch_scale missing")
    require_cuda(packed.K_ch_scale, "K_ch_scale")
    H_kv = _squeeze_h(packed.K_ch_scale).shape[0]
    T_eff = int(packed.T_eff_k) if packed.T_eff_k > 0 else int(packed.T_eff)
    device = packed.K_ch_scale.device
    si, stride, cnt, n_ch = _k_channel_maps(packed)
    if si is None or sum(n_ch) == 0:
        return torch.zeros(1, H_kv, T_eff, D, dtype=torch.float16, device=device)
    view, keep = layer_view(packed, t_k=T_eff)
    k, _ = _launch(view, H_kv, D, T_eff, device, want_k=True, want_v=False, sort_idx=si, sort_stride=stride,
                   ch_counts=cnt, n_ch=n_ch)
    del keep
    return k


def unpack_v_segment(V_packed: Tensor, V_scale: Tensor, V_zp: Tensor, n_bits: int) -> Tensor:
    """Reverse of one V segment: unpack + dequantise -> fp16 ``[..., N, D]`` (packing.py:1427-1444)."""
    if n_bits not in (2, 4, 8):
        raise ValueError(f"Unsupported n_bits={n_bits}")
    require_cuda(V_packed, "V_packed")
    lead = V_packed.shape[:-2]
    n, width = int(V_packed.shape[-2]), int(V_packed.shape[-1])
    D = width * (8 // n_bits)
    heads = 1
    for x in lead:
        heads *= int(x)
    codes = V_packed.reshape(heads, n, width).contiguous()
    sc = V_scale.reshape(heads, n).to(torch.float16).contiguous()
    zp = V_zp.reshape(heads, n).to(torch.float16).contiguous()
    out = torch.empty((heads, n, D), dtype=torch.float16, device=V_packed.device)
    if heads == 0 or n == 0:
        return out.reshape(*lead, n, D)
    v = LayerView()
    name = {2: "v2", 4: "v4", 8: "v8"}[n_bits]
    setattr(v, name, codes.data_ptr())
    setattr(v, name + "_head_stride", codes.stride(0))
    setattr(v, name + "_bytes", codes.numel())
    v.v_scale, v.v_zp, v.v_meta_head_stride, v.v_meta_bytes = sc.data_ptr(), zp.data_ptr(), sc.stride(0), sc.numel() * 2
    v.n2, v.n4, v.n8 = (n if n_bits == 2 else 0), (n if n_bits == 4 else 0), (n if n_bits == 8 else 0)
    v.max_t_v, v.t_k = n, n
    check(lib().rdkv_unpack_layer(C.byref(v), heads, D, None, 0, None, 0, 0, 0, None, ptr(out), n * D, n,
                                  stream_ptr(out.device)), "rdkv_unpack_layer")
    return out.reshape(*lead, n, D)


def _v_stripe(pl: PackedKVLayer, V16: Optional[Tensor], head_dim: int, rows: int, *, with_zone_b: bool) -> Tensor:
    H_kv = _squeeze_h(pl.V_scale).shape[0]
    device = pl.V_scale.device
    view, keep = layer_view(pl, V16 if with_zone_b else None, t_k=rows)
    _, v = _launch(view, H_kv, head_dim, rows, device, want_k=False, want_v=True)
    del keep
    return v


def _unpack_v_zone_a(pl: PackedKVLayer) -> Tensor:
    """Shared layout: the 2/4/8-bit V segments dequantised and concatenated along T, in ``sort_idx``
    order: ``[1, H_kv, T_v, D]`` fp16 (trizone_decompress.py:43-83)."""
    N_2, N_4, N_8 = (int(x) for x in pl.seg_bounds)
    T_v = int(pl.T_eff)
    assert N_2 + N_4 + N_8 == T_v, f"V seg_bounds {(N_2, N_4, N_8)} must sum to T_v={T_v}"
    H_kv = pl.V_scale.shape[1]
    if T_v == 0:
        return torch.empty(1, H_kv, 0, 1, dtype=torch.float16, device=pl.V_scale.device)
    for t, n_bits in ((pl.V_2bit, 2), (pl.V_4bit, 4), (pl.V_8bit, 8)):
        if t is not None and t.numel() > 0:
            D = int(t.shape[-1]) * (8 // n_bits)
            break
    else:
        return torch.empty(1, H_kv, 0, 1, dtype=torch.float16, device=pl.V_scale.device)
    return _v_stripe(pl, None, D, T_v, with_zone_b=False)


def _unpack_v_perhead(pl: PackedKVLayer, *, head_dim: int) -> Tensor:
    """Per-head layout: ``[1, H_kv, max_T_v, head_dim]`` fp16, head h's rows ``[0, T_v_h)`` dequantised
    and the rest zeros (trizone_decompress.py:91-144)."""
    return _v_stripe(pl, None, head_dim, int(pl.T_eff), with_zone_b=False)


def _fill_view(v: LayerView, pl: PackedKVLayer, V16: Optional[Tensor], rows: int) -> Optional[list]:
    """The fields of ``rdkv_layer_view`` the decompressor reads, straight from a layer whose tensors are
    ``[1,H_kv,...]`` with contiguous rows (what this library packs).  Returns the temporaries to keep alive; None
    for any other layer, which takes :func:`rdkv_b200.packing.layer_view`."""
    n2c, n4c, n8c = pl.K_ch_seg_bounds
    v.n_ch2_pad, v.n_ch4_pad, v.n_ch8 = (n2c + 3) // 4 * 4, (n4c + 1) // 2 * 2, n8c
    for name, stride_name, t in (("k2", "k2_head_stride", pl.K_2bit if n2c else None), ("k4", "k4_head_stride", pl.K_4bit if n4c else None),
                                 ("k8", "k8_head_stride", pl.K_8bit if n8c else None), ("v2", "v2_head_stride", pl.V_2bit),
                                 ("v4", "v4_head_stride", pl.V_4bit), ("v8", "v8_head_stride", pl.V_8bit),
                                 ("v16", "v16_head_stride", V16)):
        if t is None or t.numel() == 0:
            continue
        if t.dim() != 4 or t.shape[0] != 1 or t.stride(3) != 1:
            return None
        require_cuda(t, name)
        setattr(v, name, t.data_ptr())
        setattr(v, stride_name, t.stride(1))
    ks, kz, vs, vz = pl.K_ch_scale, pl.K_ch_zp, pl.V_scale, pl.V_zp
    if not (ks.dim() == kz.dim() == vs.dim() == vz.dim() == 4 and ks.is_contiguous() and kz.is_contiguous()
            and vs.shape[3] == vz.shape[3] == 1 and vs.stride(2) == vz.stride(2) == 1 and vs.stride(1) == vz.stride(1)):
        return None
    for name, t in (("k_scale", ks), ("k_zp", kz), ("v_scale", vs), ("v_zp", vz)):
        if t.numel():
            require_cuda(t, name)
            setattr(v, name, t.data_ptr())
    v.v_meta_head_stride = vs.stride(1)
    keep = []

    if V16 is not None and V16.numel() > 0:
        v.n_v16_shared = int(V16.shape[-2])
    for name, t in (("v_seg_bounds", pl.seg_bounds_per_head), ("n_v16", pl.n_v16_per_head if v.n_v16_shared else None)):
        if t is not None:
            if t.dtype != torch.int32 or not t.is_contiguous():
                t = t.to(torch.int32).contiguous()
                keep.append(t)
            require_cuda(t, name)
            setattr(v, name, t.data_ptr())
    v.n2, v.n4, v.n8 = (int(x) for x in pl.seg_bounds)
    v.max_t_v, v.t_k = int(pl.T_eff), rows
    return keep


def _unpack_layers(layers, V16s, D: int, first: int = 0) -> List[Tuple[Tensor, Tensor]]:
    """(K, V) fp16 stripes of every layer, the fp16-V rows included: ``unpack_k_mixed`` and ``_v_stripe``
    of all of them in one call.  ``first``: the number of the first of them in its cache."""
    jobs = (UnpackJob * max(1, len(layers)))()
    out, keep, n = [], [], 0
    devices = set()
    for i, (pl, V16) in enumerate(zip(layers, V16s)):
        if pl.K_ch_scale is None:
            raise ValueError("unpack_k_mixed: K_ch_scale missing")
        require_cuda(pl.K_ch_scale, "K_ch_scale")
        device = pl.K_ch_scale.device
        H = int(pl.K_ch_scale.shape[1] if pl.K_ch_scale.dim() == 4 and pl.K_ch_scale.shape[0] == 1 else pl.K_ch_scale.shape[0])
        rows_k = int(pl.T_eff_k) if pl.T_eff_k > 0 else int(pl.T_eff)
        n16 = int(pl.n_v16) if _is_perhead_layout(pl) else (int(V16.shape[2]) if V16 is not None and V16.numel() > 0 else 0)
        rows = int(pl.T_eff) + n16
        assert rows_k == rows, (f"layer {first + i}: K T-dim {rows_k} != V T-dim {rows} "
                                f"(T_v={pl.T_eff}, n_v16={pl.n_v16}, T_eff_k={pl.T_eff_k})")
        si, stride, cnt, n_ch = _k_channel_maps(pl)
        no_k = si is None or sum(n_ch) == 0
        K = (torch.zeros if no_k else torch.empty)((1, H, rows, D), dtype=torch.float16, device=device)
        V = torch.empty((1, H, rows, D), dtype=torch.float16, device=device)
        out.append((K, V))
        if rows == 0:
            continue
        job = jobs[n]
        tmp = _fill_view(job.view, pl, V16, rows)
        if tmp is None:
            job.view, tmp = layer_view(pl, V16, t_k=rows)
        keep.append((tmp, si, cnt))
        if not no_k:
            job.k_sort_idx, job.k_sort_idx_head_stride, job.k_ch_counts = si.data_ptr(), stride, ptr(cnt)
            job.n_ch2, job.n_ch4, job.n_ch8 = n_ch
            job.k_out = K.data_ptr()
        job.H_kv, job.v_out, job.out_head_stride, job.rows_out = H, V.data_ptr(), rows * D, rows
        devices.add(device)
        n += 1
    for device in devices:
        stream = stream_ptr(device)
    if n:
        check(lib().rdkv_unpack_layers(jobs, n, D, stream), "rdkv_unpack_layers")
    del keep
    return out


def unpack_trizone_to_past_kv(dual_cache: TriZoneCache, *, head_dim: int, device: Optional[torch.device] = None,
                              dtype: torch.dtype = torch.float16, return_masks: bool = False,
                              H_q: Optional[int] = None, max_new_tokens: int = 0,
                              mask_dtype: torch.dtype = torch.float16):
    """Reverse a ``TriZoneCache`` into HF legacy ``past_key_values``: a tuple of ``(K_i, V_i)``, each
    ``[1, H_kv, T_eff_k_i, head_dim]``; with ``return_masks`` also the per-layer ``[1, H_q, 1,
    T_eff_k_i + max_new_tokens]`` additive masks of the per-head layout (``None`` for shared-layout
    layers).  Same contract as trizone_decompress.py:185-333.

    Stripes that stay as they are unpacked (no other ``device`` or ``dtype``) are the result and come from
    one launch per 16 layers.  Stripes that are moved or converted are unpacked and let go one layer at a
    time: a cache that does not fit the GPU in fp16 can be unpacked to the host."""
    past_kv: List[Tuple[Tensor, Tensor]] = []
    masks_list: List[Optional[Tensor]] = []
    layers = list(dual_cache.packed)
    V16s = [dual_cache.new_v_only[i] if i < len(dual_cache.new_v_only) else None for i in range(len(layers))]
    target = None if device is None else torch.device(device)
    stay = dtype == torch.float16 and (target is None or all(
        pl.K_ch_scale is not None and target.type == pl.K_ch_scale.device.type
        and target.index in (None, pl.K_ch_scale.device.index) for pl in layers))
    dense = _unpack_layers(layers, V16s, head_dim) if stay else None
    for i, pl in enumerate(layers):
        K_full, V_full = dense[i] if stay else _unpack_layers([pl], V16s[i:i + 1], head_dim, i)[0]
        per_head = _is_perhead_layout(pl)
        if device is not None:
            K_full, V_full = K_full.to(device), V_full.to(device)
        if dtype != torch.float16:
            K_full, V_full = K_full.to(dtype), V_full.to(dtype)
        past_kv.append((K_full, V_full))                   # (contiguous: allocated as they are)
        if return_masks:
            if per_head and pl.softmax_mask is not None:
                mask_2d = pl.softmax_mask
                mask_H_q = int(mask_2d.shape[0])
                if H_q is not None:
                    assert H_q == mask_H_q, f"layer {i}: caller H_q={H_q} != softmax_mask H_q={mask_H_q}"
                target = device if device is not None else mask_2d.device
                mask_4d = mask_2d.to(device=target, dtype=mask_dtype).view(1, mask_H_q, 1, int(mask_2d.shape[1]))
                if max_new_tokens > 0:
                    pad = torch.zeros(1, mask_H_q, 1, max_new_tokens, dtype=mask_dtype, device=target)
                    mask_4d = torch.cat([mask_4d, pad], dim=-1)
                masks_list.append(mask_4d.contiguous())
            else:
                masks_list.append(None)
    if return_masks:
        return tuple(past_kv), masks_list
    return tuple(past_kv)
