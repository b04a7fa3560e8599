"""Edges of the one-cluster selection (runs of a warp, its largest input, ties across blocks) and of the F16 candidate scoring
(ragged last block, missing blocks, fewer positions than a warp's tile)."""
import numpy as np
import pytest
import torch

import oracle_lib as ol
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 257, 8192, 8193, 32768, 32769])
@pytest.mark.parametrize("kind", ["normal", "ties", "holes"])
def test_topk_cluster_edges(n, kind):
    from macseek_b200 import _lib, attn
    from macseek_b200.core import Enc
    orc, rng, e = ol.Oracle(), np.random.default_rng(n), Enc()
    v = rng.standard_normal(n).astype(np.float32)
    if kind == "ties":
        v = np.float32(1.0) + rng.integers(0, 3, n).astype(np.float32) * np.float32(2.0 ** -23)   # differ in the last bits only
    if kind == "holes":
        v[rng.integers(0, n, n // 2)] = -np.inf
    scratch = torch.zeros(_lib.lib.msb_topk_scratch_bytes(n) // 4 + 1, dtype=torch.int32, device="cuda")
    sc = torch.from_numpy(v).cuda()
    for k in (1, 512, 2048):
        out = torch.full((k,), -7, dtype=torch.int32, device="cuda")
        attn.encode_topk(e, sc, n, k, out, scratch)
        e.wait()
        assert np.array_equal(out.cpu().numpy(), orc.topk_sorted(v, k)), k


@pytest.mark.parametrize("heads", [32, 64])
def test_f16_candidate_scores(heads):
    from macseek_b200 import attn
    from macseek_b200.core import Enc
    orc, e = ol.Oracle(), Enc()
    length, k = 4003, 256
    sh = attn.Shape(D=512, heads=64, index_heads=heads, topk=k, key_type=attn.KEY_F16, elem_type=attn.ELEM_F16)
    tab = np.zeros((1, 32, 2), np.float32)
    tab[:, :, 0] = 1.0
    st = attn.DecodeState(sh, length, tab)
    keys = synth.randn(length * 128, 1).reshape(length, 128).astype(np.float16)
    q, w = synth.randn(heads * 128, 2).reshape(heads, 128) * np.float32(1e-3), synth.randn(heads, 3)      # small queries: every term counts
    st.ikey[:length] = torch.from_numpy(keys).cuda()
    cand = np.full(sh.cand_blocks, -1, np.int32)
    cand[:101] = np.sort(np.random.default_rng(4).choice(length // 8 + 1, 101, replace=False))
    cand[100] = length // 8                                  # the block that ends after 3 keys
    st.cand_list.copy_(torch.from_numpy(cand))
    attn.encode_index_decode_list(e, st, torch.from_numpy(q).cuda(), torch.from_numpy(w).cuda(), 0, length, actq=False)
    e.wait()
    qp, wp = orc.index_q(q, w, tab[0], False, heads, 128)
    ref = orc.index_scores(qp, wp, keys.astype(np.float32))
    masked = np.full(length, -np.inf, np.float32)
    for b in cand[:101]:
        masked[8 * b:min(length, 8 * b + 8)] = ref[8 * b:min(length, 8 * b + 8)]
    assert np.array_equal(st.topk.cpu().numpy(), orc.topk_sorted(masked, k))
    virt = st.dec_scores[:8 * 101].cpu().numpy().reshape(101, 8)
    for i, b in enumerate(cand[:101]):
        seg = ref[8 * b:min(length, 8 * b + 8)]
        assert np.max(np.abs(virt[i, :len(seg)] - seg)) <= 2e-6 * np.max(np.abs(ref)) and np.all(virt[i, len(seg):] == -np.inf)
