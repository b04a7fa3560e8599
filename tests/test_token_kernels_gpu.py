"""Edges of the per-token kernels: sampling top-k and log-softmax at ties, short and ragged rows; routing lists over many
experts; hyper-connection steps of several tokens at once."""
import numpy as np
import pytest
import torch

import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def orc():
    return ol.Oracle()


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("V", (1, 63, 128, 129, 4097, 33333, 131073, 262144))
@pytest.mark.parametrize("data", ("normal", "equal", "two_levels", "sorted", "one_granule"))
def test_topk_edges(orc, V, data):
    from macseek_b200 import arch
    from macseek_b200.core import Enc
    rng = np.random.default_rng(V)
    x = rng.standard_normal(V).astype(np.float32)
    if data == "equal":
        x[:] = -0.0
        x[::3] = 0.0                              # compares equal to -0
    elif data == "two_levels":                    # more ties at the threshold than granules
        x[:] = 1.0
        x[rng.choice(V, max(1, min(V, 40) // 2), replace=False)] = 2.0
    elif data == "sorted":
        x = np.sort(x)
    elif data == "one_granule":                   # the whole top inside one run of 128
        x = np.abs(x) * -1
        x[:min(V, 128)] = np.linspace(1, 2, min(V, 128), dtype=np.float32)
    e = Enc()
    s = arch.sample_scratch(2)
    xd = dev(np.stack([x, x[::-1]]))
    ov, oi, lse = torch.zeros(2, 64, device="cuda"), torch.zeros(2, 64, dtype=torch.int32, device="cuda"), torch.zeros(2, device="cuda")
    for k in (1, 33, 64):
        arch.encode_sample_topk(e, xd, 2, V, k, 1.0, ov, oi, lse, s)
        e.wait()
        for r in range(2):
            row = np.ascontiguousarray(x if r == 0 else x[::-1])
            order = np.lexsort((np.arange(V), -row))[:k]
            n = order.size
            assert np.array_equal(oi[r, :n].cpu().numpy(), order), (k, r)
            assert np.array_equal(ov[r, :n].cpu().numpy().view(np.uint32), row[order].view(np.uint32))
            assert (oi[r, n:k].cpu().numpy() == -1).all()
            assert abs(float(lse[r]) - orc.logsumexp(row)) <= 1e-4 * abs(orc.logsumexp(row)) + 1e-5


@pytest.mark.parametrize("V,rows", ((1, 2), (7, 2), (8193, 2), (163840, 2), (200001, 2), (1, 40), (1025, 300), (20000, 40)))
def test_log_softmax_edges(orc, V, rows):
    from macseek_b200 import arch
    from macseek_b200.core import Enc
    x = (3 * np.random.default_rng(V).standard_normal((rows, V))).astype(np.float32)
    xd, out = dev(x), torch.zeros(rows, V, device="cuda")
    e = Enc()
    arch.encode_log_softmax(e, xd, out, rows, V)
    e.wait()
    for r in range(rows):
        assert np.max(np.abs(out[r].cpu().numpy() - orc.log_softmax(x[r]))) <= 3e-5


@pytest.mark.parametrize("n,k,E", ((3, 2, 2049), (700, 3, 5000), (1025, 8, 64), (2048, 4, 1)))
def test_route_lists_edges(orc, n, k, E):
    from macseek_b200 import arch
    from macseek_b200.core import Enc
    rng = np.random.default_rng(n)
    ids = rng.integers(0, E, (n, k)).astype(np.int32)
    w = rng.random((n, k)).astype(np.float32)
    L = arch.RouteLists.create(n, k, E)
    e = Enc()
    arch.encode_route_lists(e, dev(ids), dev(w), n, L)
    e.wait()
    for g, r in zip((L.counts, L.offsets, L.entry, L.tok, L.w, L.slot_of), orc.route_lists(ids, w, n, k, E)):
        assert np.array_equal(g.cpu().numpy().view(np.uint32), r.view(np.uint32))


@pytest.mark.parametrize("D", (1024, 5120))
@pytest.mark.parametrize("n", (2, 9, 10, 41))
def test_hc_step_tokens(orc, D, n):
    from macseek_b200 import arch
    from macseek_b200.core import Enc
    rng = np.random.default_rng(D + n)
    f = lambda *s: rng.standard_normal(s).astype(np.float32)
    h, xs, mp = 2 * f(n, 4, D), f(n, D), np.abs(f(n, 24)) * 0.5 + np.float32(0.05)
    fn, scale, base, gain = f(24, 4 * D) * np.float32(0.02), np.array([0.7, 1.3, 0.9], np.float32), f(24), 1 + f(D) * np.float32(0.1)
    e = Enc()
    hd, mo, xo, scratch = dev(h), torch.zeros(n, 24, device="cuda"), torch.zeros(n, D, device="cuda"), arch.hc_scratch(n)
    arch.encode_hc_step(e, hd, hd, dev(xs), dev(mp), dev(fn), dev(scale), dev(base), mo, dev(gain), xo, D, scratch, n)
    e.wait()
    for t in range(n):
        rh, rm, rx = orc.hc_step(h[t].reshape(-1), xs[t], mp[t], fn.reshape(-1), scale, base, gain, D)
        assert np.max(np.abs(hd[t].cpu().numpy().reshape(-1) - rh)) <= 2e-6 * np.max(np.abs(rh))
        assert np.max(np.abs(mo[t].cpu().numpy() - rm)) <= 2e-5
        assert np.max(np.abs(xo[t].cpu().numpy() - rx)) <= 1e-5 * np.max(np.abs(rx))


@pytest.mark.parametrize("D", (512, 1024, 4096, 5120))
@pytest.mark.parametrize("n", (1, 12))
def test_hc_step_adds_the_blocks_sums_in_double(D, n):
    """Three columns in different sixteenths of the width carry 2^24, 1 and -2^24: their sum is 1, in float it would be 0."""
    from macseek_b200 import arch
    from macseek_b200.core import Enc
    h = torch.zeros(n, 4, D, device="cuda")
    h[:, 0, 0], h[:, 0, D // 16], h[:, 0, D // 8] = 2.0 ** 24, 1.0, -2.0 ** 24
    fn = torch.zeros(24, 4, D, device="cuda")
    fn[:, 0] = 1.0
    rstd = 1.0 / np.sqrt(2.0 ** 49 / (4 * D))
    scale = torch.full((3,), 1.0 / rstd, device="cuda")
    mp, mo = torch.zeros(n, 24, device="cuda"), torch.zeros(n, 24, device="cuda")
    mp[:, 0] = 1.0
    e = Enc()
    arch.encode_hc_step(e, h, h, None, mp, fn, scale, torch.zeros(24, device="cuda"), mo, None, None, D, arch.hc_scratch(n), n)
    e.wait()
    pre = 1.0 / (1.0 + np.exp(-1.0))                      # of scale * sum * rstd = 1
    assert np.max(np.abs(mo[:, :4].cpu().numpy() - pre)) <= 1e-5 and np.max(np.abs(mo[:, 4:8].cpu().numpy() - 2 * pre)) <= 1e-5


@pytest.mark.parametrize("n", (1, 40))
def test_hc_step_sinkhorn_against_float64(n):
    """The 4 x 4 mixing matrix alone: no product with fn (its rows are zero), any base.  An element is rounded by 40 products or
    divisions (2^-24 each), by the exponential (4 of them) and by its argument (2^-24 of it); a line's sum can bring in twice
    what an element has itself."""
    from macseek_b200 import arch
    from macseek_b200.core import Enc
    D, e = 1024, Enc()
    for spread in (0.1, 1.0, 4.0):
        h = torch.randn(n, 4, D, device="cuda")
        base = spread * torch.randn(24, device="cuda")
        mo = torch.zeros(n, 24, device="cuda")
        arch.encode_hc_step(e, h, h, None, torch.ones(n, 24, device="cuda"), torch.zeros(24, 4 * D, device="cuda"), torch.ones(3, device="cuda"),
                            base, mo, None, None, D, arch.hc_scratch(n), n)
        e.wait()
        c = torch.softmax(base[8:].double().view(4, 4), 1) + 1e-6
        for it in range(20):
            if it:
                c = c / (c.sum(1, keepdim=True) + 1e-6)
            c = c / (c.sum(0, keepdim=True) + 1e-6)
        got = mo[:, 8:].double().view(n, 4, 4)
        span = float(base[8:].max() - base[8:].min())
        assert float(((got - c) / c).abs().max()) <= 3 * (40 + 4 + span) * 2.0 ** -24, spread
