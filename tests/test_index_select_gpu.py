"""Edges of the one-cluster selection (runs of a warp, its largest input, ties across blocks) and of the F16 candidate scoring
(ragged last block, missing blocks, fewer positions than a warp's tile)."""
import numpy as np
import pytest
import torch

import oracle_lib as ol
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 257, 8192, 8193, 16384, 16385, 32768, 32769])
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


@pytest.mark.parametrize("key_type", ["f16", "fp8"])
@pytest.mark.parametrize("listed", [False, True])
def test_refused_index_decode_leaves_the_scratch_zeroed(key_type, listed):
    """k too large, no output, a scratch too small: refused before anything is added to the scratch's histogram, so that the
    next call selects what it would have selected."""
    from macseek_b200 import _lib, attn
    from macseek_b200.core import Enc, ptr
    orc, e = ol.Oracle(), Enc()
    length, k, heads = 2000, 512, 32
    kt = attn.KEY_F16 if key_type == "f16" else attn.KEY_FP8
    keys = torch.from_numpy(synth.randn(length * 128, 1).reshape(length, 128)).cuda()
    keys = keys.half() if key_type == "f16" else keys.to(torch.float8_e4m3fn).view(torch.uint8)
    q, w = torch.from_numpy(synth.randn(heads * 128, 2)).cuda(), torch.from_numpy(synth.randn(heads, 3)).cuda()
    cs = torch.zeros(32, 2, device="cuda")
    cs[:, 0] = 1.0
    qp, wp, sc = torch.zeros(heads, 128, device="cuda"), torch.zeros(heads, device="cuda"), torch.zeros(length, device="cuda")
    cand = torch.arange(length // 8, dtype=torch.int32, device="cuda")
    out = torch.full((4096,), -7, dtype=torch.int32, device="cuda")
    need = _lib.lib.msb_topk_scratch_bytes(length)
    scratch = torch.zeros(need // 4 + 1, dtype=torch.int32, device="cuda")       # always the whole room, whatever size is named

    def call(kk, dst, size):
        if listed:
            return _lib.lib.msb_index_decode_list(kt, ptr(keys), length, ptr(q), ptr(w), ptr(cs), 0, heads, kk, ptr(cand), cand.numel(),
                                                  ptr(qp), ptr(wp), ptr(sc), ptr(dst), ptr(scratch), size, e.handle)
        return _lib.lib.msb_index_decode(kt, ptr(keys), length, ptr(q), ptr(w), ptr(cs), 0, heads, kk, ptr(qp), ptr(wp), ptr(sc), ptr(dst),
                                         ptr(scratch), size, 0, e.handle)

    for kk, dst, size in ((4096, out, need), (0, out, need), (k, None, need), (k, out, 64), (k, out, need - 4)):
        assert call(kk, dst, size) != 0
        e.wait()
        assert int(scratch.abs().max()) == 0
    assert call(k, out, need) == 0
    e.wait()
    assert np.array_equal(out[:k].cpu().numpy(), orc.topk_sorted(sc.cpu().numpy(), k))
    assert int(scratch.abs().max()) == 0


@pytest.mark.parametrize("heads", [32, 64])
@pytest.mark.parametrize("listed", [False, True])
def test_f16_scores_are_as_precise_as_fp32_sums(heads, listed):
    """Against float64: 128 fp32 additions one after the other are 2.2e-7 off here, the bound is a third more."""
    from macseek_b200 import _lib
    from macseek_b200.core import Enc, ptr
    n, k, e = 16384, 512, Enc()
    g = torch.Generator(device="cuda")
    g.manual_seed(heads)
    keys = torch.randn(n, 128, device="cuda", generator=g).half()
    q, w = torch.randn(heads, 128, device="cuda", generator=g), torch.randn(heads, device="cuda", generator=g)
    cs = torch.zeros(32, 2, device="cuda")
    cs[:, 0] = 1.0
    qp, wp, sc = torch.zeros(heads, 128, device="cuda"), torch.zeros(heads, device="cuda"), torch.zeros(n, device="cuda")
    out, cand = torch.zeros(k, dtype=torch.int32, device="cuda"), torch.arange(n // 8, dtype=torch.int32, device="cuda")
    need = _lib.lib.msb_topk_scratch_bytes(n)
    scratch = torch.zeros(need // 4 + 1, dtype=torch.int32, device="cuda")
    if listed:
        _lib.check(_lib.lib.msb_index_decode_list(1, ptr(keys), n, ptr(q), ptr(w), ptr(cs), 0, heads, k, ptr(cand), n // 8, ptr(qp), ptr(wp),
                                                  ptr(sc), ptr(out), ptr(scratch), need, e.handle))
    else:
        _lib.check(_lib.lib.msb_index_decode(1, ptr(keys), n, ptr(q), ptr(w), ptr(cs), 0, heads, k, ptr(qp), ptr(wp), ptr(sc), ptr(out),
                                             ptr(scratch), need, 0, e.handle))
    e.wait()
    want = (torch.relu(q.double() @ keys.double().T) * (w.double() * (128 * heads) ** -0.5)[:, None]).sum(0)
    assert float((sc.double() - want).norm() / want.norm()) <= 3e-7
