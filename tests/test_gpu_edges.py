"""Prefill kernels at the sizes where they change their way of working, against the oracle, bit for bit."""
import numpy as np
import pytest
import torch

from helpers import to_np

pytestmark = pytest.mark.gpu


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
