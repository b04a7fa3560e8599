"""Sampling head on the GPU, mirroring the reference's own test (tests/test_arch_sample.mm): argmax over several rows
with ties and edge maxima and repeated launches, Gumbel-max sampling (the winner reproduced from the restated noise, and
the empirical distribution against softmax(l / T)), top-k + log-sum-exp bit-exact ids / values, log-softmax (also in
place), the CPU top-p sampler, and a top-k logits dump written from the kernel's output."""
import numpy as np
import pytest
import torch

import oracle_lib as ol

pytestmark = pytest.mark.gpu
V = 129280


@pytest.fixture(scope="module")
def orc():
    return ol.Oracle()


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def test_argmax_rows_ties_edges_repeats(orc):
    from macseek_b200 import arch
    from macseek_b200.core import Enc
    rows = 6
    rng = np.random.default_rng(99)
    l = (4.0 * rng.standard_normal((rows, V))).astype(np.float32)
    l[0, 0] = 100.0
    l[1, V - 1] = 100.0
    l[2, 5000] = 50.0; l[2, 90000] = 50.0            # tie -> lowest index
    l[3, 2019] = 60.0; l[3, 2020] = 60.0             # tie across a chunk boundary
    ld = dev(l)
    idx, val = torch.zeros(rows, dtype=torch.int32, device="cuda"), torch.zeros(rows, device="cuda")
    s = arch.sample_scratch(rows)
    e = Enc()
    for rep in range(3):
        idx.fill_(-1)
        arch.encode_argmax_rows(e, ld, rows, V, idx, val, s)
        e.wait()
        for r in range(rows):
            want = orc.argmax(l[r])
            assert int(idx[r]) == want and float(val[r]) == l[r, want], (rep, r)
    # 300 back-to-back launches on one stream (ticket reuse): all agree
    R = 300
    si = torch.zeros(R, rows, dtype=torch.int32, device="cuda")
    for i in range(R):
        arch.encode_argmax_rows(e, ld, rows, V, si[i], None, s)
    e.wait()
    assert torch.equal(si, idx.unsqueeze(0).expand(R, rows))


def test_gumbel_winner_and_distribution(orc):
    from macseek_b200 import arch
    from macseek_b200.core import Enc
    e = Enc()
    # (1) which element wins is reproducible from the restated noise (float vs double log: skip rows with a near-tie)
    rng = np.random.default_rng(5)
    rows, n = 4, 5000
    l = rng.standard_normal((rows, n)).astype(np.float32)
    idx, val = torch.zeros(rows, dtype=torch.int32, device="cuda"), torch.zeros(rows, device="cuda")
    s = arch.sample_scratch(16)
    seed, T = 0x0123456789ABCDEF, 0.8
    arch.encode_argmax_rows(e, dev(l), rows, n, idx, val, s, T, seed)
    e.wait()
    checked = 0
    for r in range(rows):
        noisy = np.array([l[r, i] / np.float32(T) + orc.gumbel(i, seed, r) for i in range(n)])
        o = np.argsort(-noisy)
        # the winner's noise is large (u close to 1), where the float -log(-log(u)) of the kernel (the reference's
        # formula) is only good to ~1e-3 absolute: skip near-ties below that, compare the value to that
        if noisy[o[0]] - noisy[o[1]] > 5e-3:
            assert int(idx[r]) == int(o[0]) and abs(float(val[r]) - noisy[o[0]]) < 2e-3
            checked += 1
    assert checked >= 2
    # (2) empirical distribution over a small vocabulary against softmax(l / T): chi-square, 6 dof, p = 0.001
    Vs, N, per = 7, 20000, 16
    lv = np.array([1.0, 2.0, 0.5, 2.5, -1.0, 1.5, 0.0], np.float32)
    l16 = dev(np.tile(lv, (per, 1)))
    bi = torch.zeros(per, dtype=torch.int32, device="cuda")
    out = torch.zeros(N // per, per, dtype=torch.int32, device="cuda")
    for it in range(N // per):
        arch.encode_argmax_rows(e, l16, per, Vs, out[it], None, s, T, 0x1234567 + it * 7919)
    e.wait()
    cnt = np.bincount(out.cpu().numpy().reshape(-1), minlength=Vs)
    p = np.exp(lv / T - orc.logsumexp(lv, 1.0 / T))
    chi2 = float(((cnt - p * N) ** 2 / (p * N)).sum())
    assert chi2 < 22.5, (chi2, cnt / N, p)


def test_topk_lse_and_top_p(orc, tmp_path):
    from macseek_b200 import arch, logits_dump
    from macseek_b200.core import Enc
    rows, k = 3, 64
    rng = np.random.default_rng(7)
    l = (3.0 * rng.standard_normal((rows, V))).astype(np.float32)
    for i in range(10):
        l[1, 4040 * i + 7] = 20.0                   # ties across chunks
    ld = dev(l)
    ov, oi = torch.zeros(rows, 64, device="cuda"), torch.zeros(rows, 64, dtype=torch.int32, device="cuda")
    ol_ = torch.zeros(rows, device="cuda")
    s = arch.sample_scratch(rows)
    e = Enc()
    for T in (1.0, 0.7):
        for rep in range(2):
            arch.encode_sample_topk(e, ld, rows, V, k, T, ov, oi, ol_, s)
            e.wait()
            for r in range(rows):
                rv, ri = orc.topk_desc(l[r], k)
                assert np.array_equal(oi[r].cpu().numpy().astype(np.uint32), ri), (T, r)
                assert np.array_equal(ov[r].cpu().numpy().view(np.uint32), rv.view(np.uint32))
                want = orc.logsumexp(l[r], 1.0 / T)
                assert abs(float(ol_[r]) - want) <= 1e-4 * abs(want) + 1e-5
    # smaller k and a short row
    arch.encode_sample_topk(e, ld[0, :1000].contiguous(), 1, 1000, 5, 1.0, ov, oi, ol_, s)
    e.wait()
    rv, ri = orc.topk_desc(l[0, :1000], 5)
    assert np.array_equal(oi[0, :5].cpu().numpy().astype(np.uint32), ri)
    # CPU top-p sampler on the T = 0.7 result of row 0: library function == oracle, frequencies == nucleus probabilities
    arch.encode_sample_topk(e, ld, rows, V, k, 0.7, ov, oi, ol_, s)
    e.wait()
    v0, i0, lse0 = ov[0].cpu().numpy(), oi[0].cpu().numpy(), float(ol_[0])
    p = np.exp(v0.astype(np.float64) / 0.7 - lse0)
    keep = int(np.searchsorted(np.cumsum(p), 0.3) + 1)
    N = 20000
    cnt = np.zeros(k)
    for it in range(N):
        u = (it + 0.5) / N
        tok = arch.sample_top_p(v0, i0, k, lse0, 0.7, 0.3, u)
        if it % 97 == 0:
            assert tok == orc.sample_top_p(v0, i0.astype(np.uint32), k, lse0, 0.7, 0.3, u)
        pos = int(np.where(i0 == tok)[0][0])
        assert pos < keep
        cnt[pos] += 1
    assert np.all(np.abs(cnt[:keep] / N - p[:keep] / p[:keep].sum()) < 1e-3)
    assert arch.sample_top_p(v0, i0, k, lse0, 0.0, 0.3, 0.99) == int(i0[0])
    # a top-k dump of these positions (temperature 1) reads back as written
    arch.encode_sample_topk(e, ld, rows, V, k, 1.0, ov, oi, ol_, s)
    e.wait()
    path = str(tmp_path / "t.logits")
    logits_dump.write_topk(path, [1, 2, 3, 4], V, oi.cpu().numpy(), ov.cpu().numpy(), ol_.cpu().numpy(), first_pos=1)
    d = logits_dump.read(path)
    assert d["k"] == 64 and np.array_equal(d["ids"], oi.cpu().numpy()) and np.array_equal(d["lse"], ol_.cpu().numpy())
    # bad arguments
    from macseek_b200 import _lib
    with pytest.raises(_lib.MsbError):
        arch.encode_sample_topk(e, ld, rows, V, 65, 1.0, ov, oi, ol_, s)
    with pytest.raises(_lib.MsbError):
        arch.encode_sample_topk(e, ld, rows, V, 8, 1.0, ov, oi, ol_, s[:16])


def _topk_rows():
    """Rows at the edges of the cluster's form: its smallest and largest V and what lies beside them, every number of registers per
    thread, ties (more than the list holds, at the k-th place, at zero of both signs), rows of few numbers."""
    rng = np.random.default_rng(23)
    for V_, k in ((16384, 64), (16385, 64), (16385, 1), (32768, 33), (65536, 64), (65537, 7), (131072, 64), (131073, 64),
                  (163840, 64), (163841, 5)):
        yield "normal", rng.standard_normal(V_).astype(np.float32), k
    base = rng.standard_normal(100003).astype(np.float32)
    yield "equal", np.full(100003, -2.5, np.float32), 64
    x = base.copy(); x[rng.choice(x.size, 5000, replace=False)] = 9.0; x[77777] = 10.0
    yield "ties", x, 40
    x = -np.abs(base); x[rng.choice(x.size, 3000, replace=False)] = 0.0; x[rng.choice(x.size, 3000, replace=False)] = -0.0
    yield "zeros", x, 64
    x = np.full(100003, np.nan, np.float32); x[[5, 40000, 99999]] = [1.0, -1.0, np.inf]
    yield "few", x, 64
    x = np.full(100003, -np.inf, np.float32); x[1000:1900] = base[:900]
    yield "one block", x, 64
    x = base.copy(); x[::3] = np.nan; x[1] = np.inf
    yield "nan", x, 50


@pytest.mark.parametrize("rows", [1, 3])
def test_topk_at_the_edges_of_its_forms(rows):
    from macseek_b200 import arch
    from macseek_b200.core import Enc
    e, s = Enc(), arch.sample_scratch(rows)
    for name, x, k in _topk_rows():
        l = np.stack([np.roll(x, 11 * r) for r in range(rows)])
        ov, oi = torch.zeros(rows, 64, device="cuda"), torch.zeros(rows, 64, dtype=torch.int32, device="cuda")
        lse = torch.zeros(rows, device="cuda")
        arch.encode_sample_topk(e, dev(l), rows, l.shape[1], k, 0.8, ov, oi, lse, s)
        e.wait()
        for r in range(rows):
            valid = np.flatnonzero(~np.isnan(l[r]))
            order = valid[np.lexsort((valid, -l[r][valid]))][:k]          # descending, ties by index
            n = order.size
            assert np.array_equal(oi[r, :n].cpu().numpy(), order), (name, l.shape[1], k, r)
            assert np.array_equal(ov[r, :n].cpu().numpy().view(np.uint32), l[r][order].view(np.uint32)), (name, r)
            assert (oi[r, n:k].cpu().numpy() == -1).all() and np.isneginf(ov[r, n:k].cpu().numpy()).all(), (name, r)
            if np.isfinite(l[r]).all():
                z = l[r].astype(np.float64) / 0.8
                want = z.max() + np.log(np.exp(z - z.max()).sum())
                assert abs(float(lse[r]) - want) <= 1e-5 * abs(want) + 1e-5, (name, r)


@pytest.mark.parametrize("rows,V_,k", [(20, 40000, 40), (33, 70000, 64), (64, 129280, 64), (5, 16385, 64), (2, 163840, 3), (66, 40000, 64)])
def test_topk_of_more_rows_than_run_at_once_and_of_masked_rows(rows, V_, k):
    """Up to 64 rows by clusters, of which 15 run at once, or by groups; every third row has all but a few hundred or one of its logits
    masked with -inf, some are masked whole."""
    from macseek_b200 import arch
    from macseek_b200.core import Enc
    g = torch.Generator(device="cuda"); g.manual_seed(rows + V_)
    x = 3 * torch.randn(rows, V_, device="cuda", generator=g)
    for r in range(0, rows, 3):
        keep = [300, 1, 0][r // 3 % 3]
        at = torch.randperm(V_, device="cuda", generator=g)[keep:]
        x[r, at] = -float("inf")
    ov, oi = torch.zeros(rows, 64, device="cuda"), torch.zeros(rows, 64, dtype=torch.int32, device="cuda")
    lse = torch.zeros(rows, device="cuda")
    e, s = Enc(), arch.sample_scratch(rows)
    for _ in range(2):
        arch.encode_sample_topk(e, x, rows, V_, k, 0.8, ov, oi, lse, s)
    e.wait()
    l = x.cpu().numpy()
    for r in range(rows):
        order = np.lexsort((np.arange(V_), -l[r]))[:k]               # -inf is a number: lowest index first
        assert np.array_equal(oi[r, :k].cpu().numpy(), order), r
        assert np.array_equal(ov[r, :k].cpu().numpy(), l[r][order]), r
        z = l[r].astype(np.float64) / 0.8
        if np.isneginf(z.max()):
            assert np.isneginf(float(lse[r])), r
            continue
        want = z.max() + np.log(np.exp(z - z.max()).sum())
        # exponents of at most 2^5 in fp32, a sum of positive terms: 1e-5, a tenth of what the sampler is given elsewhere
        assert abs(float(lse[r]) - want) <= 1e-5 * max(1.0, abs(want)), r


def test_log_softmax_and_in_place(orc):
    from macseek_b200 import arch
    from macseek_b200.core import Enc
    rows = 3
    rng = np.random.default_rng(11)
    l = (3.0 * rng.standard_normal((rows, V))).astype(np.float32)
    ld, out = dev(l), torch.zeros(rows, V, device="cuda")
    e = Enc()
    arch.encode_log_softmax(e, ld, out, rows, V)
    arch.encode_log_softmax(e, ld, ld, rows, V)       # in place
    e.wait()
    assert torch.equal(out, ld)
    for r in range(rows):
        want = orc.log_softmax(l[r])
        assert np.max(np.abs(out[r].cpu().numpy() - want)) <= 2e-5
