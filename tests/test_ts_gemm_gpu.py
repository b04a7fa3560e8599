"""Edges of the contractions that decode raw blocks into tensor memory, and of the block-pair GEMM beside them: tile and piece
remainders, matrices at 2-byte addresses, a split K, more expert groups than fit in shared memory."""
import numpy as np
import pytest
import torch

import oracle_lib as ol
import synth

pytestmark = pytest.mark.gpu

KQ = (ol.Q6_K, ol.Q5_K, ol.IQ1_S, ol.IQ2_XXS)


def r16(a):
    return a.astype(np.float16).astype(np.float64)


def at_offset(a, off):
    """device copy of the bytes of `a`, `off` bytes after an aligned address"""
    b = torch.zeros(a.nbytes + 64, dtype=torch.uint8, device="cuda")
    v = b[off:off + a.nbytes]
    v.copy_(torch.from_numpy(a.view(np.uint8).reshape(-1).copy()))
    return v


@pytest.mark.parametrize("t", [ol.Q6_K, ol.Q5_K, ol.Q8_0, ol.IQ4_NL, ol.IQ1_S, ol.IQ2_XXS, ol.BF16, ol.F16, ol.F32])
def test_matmul_edges(t):
    from macseek_b200 import quant as q
    from macseek_b200.core import Enc
    orc = ol.Oracle()
    k1 = 256 if t in KQ else 128          # one and three pieces of K, then a long K (split over a cluster)
    shapes = [(1, k1, 1), (255, 3 * k1, 16), (257, k1, 17), (300, 3 * k1, 64), (513, 2816, 65), (511, 5 * k1, 128),
              (40, 3 * k1, 129), (256, 2560, 300), (520, k1, 1500), (777, 1280, 2049)]
    for i, (rows, cols, n) in enumerate(shapes):
        acc = i % 2 == 1
        off = 0 if t == ol.F16 else 4 if t == ol.F32 else 2 * (i % 3)
        W = synth.random_weights(t, rows, cols, 70 + i)
        X = synth.randn(n * cols, 71 + i).reshape(n, cols)
        Y0 = synth.randn(n * rows, 72 + i).reshape(n, rows)
        wd = orc.dequant(t, W, rows * cols).reshape(rows, cols).astype(np.float64)
        wh = wd if t == ol.F32 else r16(wd)
        base = Y0 if acc else 0.0
        want = r16(X) @ wh.T + base
        mag = np.abs(X.astype(np.float64)) @ np.abs(wd).T + np.abs(base)
        Y = torch.from_numpy(Y0.copy()).cuda()
        scratch = torch.zeros(q.matmul_scratch_bytes(t, rows, cols, n), dtype=torch.uint8, device="cuda")
        e = Enc()
        q.encode_matmul(e, t, at_offset(W, off), rows, cols, torch.from_numpy(X).cuda(), Y, n, acc, scratch)
        e.wait()
        err = float(np.max(np.abs(Y.cpu().numpy() - want) / (mag + 1e-12)))
        assert err <= 1e-5, (rows, cols, n, err)


@pytest.mark.parametrize("n_exp,off,n", [(3, 2, 40), (700, 0, 1400)])
def test_moe_prefill_groups_and_alignment(n_exp, off, n):
    from macseek_b200 import quant as q
    from macseek_b200.core import Enc
    orc = ol.Oracle()
    D, I, t = 256, 256, ol.IQ2_XXS
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    base = [synth.random_weights(t, 256, 256, 90 + i) for i in range(9)]      # three distinct experts, used in turn
    mats = [at_offset(m, off) for m in base]
    a = q.MoePrefillArgs(D, I)
    a.t_gate_up, a.t_down, a.t_shared = t, t, t
    a.n_tokens, a.k_per_token, a.has_shared = n, 1, False
    for j in range(n_exp):
        s = q.ExpertSlot()
        s.gate, s.up, s.down = mats[3 * (j % 3)], mats[3 * (j % 3) + 1], mats[3 * (j % 3) + 2]
        a.slots.append(s)
    # two tokens of every expert: a group is made for each that has entries, and 16 KB hold 682
    expert = np.repeat(np.arange(n_exp), 2) if n_exp > 3 else np.array([0] * 1 + [1] * 16 + [2] * 23)
    assert n_exp == 3 or np.unique(expert).size > 682
    a.offs = [int(v) for v in np.searchsorted(expert, np.arange(n_exp + 1))]
    X, Y0 = synth.randn(n * D, 5).reshape(n, D), synth.randn(n * D, 6).reshape(n, D)
    a.tok, a.wt, a.slot_of = dev(np.arange(n, dtype=np.int32)), dev(np.full(n, 0.5, np.float32)), dev(np.arange(n, dtype=np.int32))
    a.X, a.Y = dev(X), dev(Y0)
    a.scratch = torch.zeros(q.moe_prefill_scratch_bytes(n, n, n_exp, D, I), dtype=torch.uint8, device="cuda")
    e = Enc()
    q.encode_moe_prefill(e, a)
    e.wait()
    w = [r16(orc.dequant(t, m, 65536).reshape(256, 256).astype(np.float64)) for m in base]
    want, mag = Y0.astype(np.float64), np.abs(Y0).astype(np.float64)
    for i in range(n):
        wg, wu, wd = w[3 * (expert[i] % 3):3 * (expert[i] % 3) + 3]
        x = r16(X[i])
        g, u = np.minimum(wg @ x, 10.0), np.clip(wu @ x, -10.0, 10.0)
        h = r16((g / (1 + np.exp(-g)) * u * 0.5).astype(np.float32))
        want[i] += wd @ h
        mag[i] += np.abs(wd) @ np.abs(h)
    assert float(np.max(np.abs(a.Y.cpu().numpy() - want) / (mag + 1e-9))) <= 1e-3
