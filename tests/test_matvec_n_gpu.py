"""Edges of the tensor-core projection of 2 to 16 tokens: row tiles of 16, groups of four tokens, units past the last group of
four, rows brought in runs of units, several passes, matrices at 2-byte addresses, activations whose extremes use the fixed
point's whole range."""
import numpy as np
import pytest
import torch

import oracle_lib as ol
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [ol.Q6_K, ol.Q5_K, ol.Q8_0, ol.IQ4_NL, ol.IQ1_S, ol.IQ2_XXS])
def test_matvec_n_edges(t):
    from macseek_b200 import quant as q
    from macseek_b200.core import Enc
    orc = ol.Oracle()
    odd = t in (ol.Q8_0, ol.IQ4_NL)                   # 32-element blocks: any number of units
    shapes = [(1, 256, 2), (15, 1056 if odd else 1024, 3), (17, 2304, 4), (33, 768, 5), (600, 96 if odd else 256, 16),
              (5000, 512, 9), (40, 5120, 8), (100, 12288, 13), (31, 20480, 16)]
    for i, (rows, cols, n) in enumerate(shapes):
        W = synth.random_weights(t, rows, cols, 40 + i)
        x = synth.randn(n * cols, 41 + i).reshape(n, cols).copy()
        x[0, :32] = 0.0
        x[1, :32] = np.where(np.arange(32) % 2, 1.0, -1.0)        # both extremes
        x[1, 32:64] = np.linspace(-0.99, 1.0, 32)
        acc = bool(i & 1)
        y0 = synth.randn(n * rows, 42 + i).reshape(n, rows)
        ry, mag = orc.matvec(t, W, rows, cols, x, 1)
        if acc:
            ry, mag = ry + y0, mag + np.abs(y0)
        off = 2 * (i % 4)
        Wd = torch.zeros(W.nbytes + 64, dtype=torch.uint8, device="cuda")[off:off + W.nbytes]
        Wd.copy_(torch.from_numpy(W.view(np.uint8).reshape(-1).copy()))
        yd = torch.from_numpy(y0.copy()).cuda()
        e = Enc()
        q.encode_matvec_n(e, t, Wd, rows, cols, torch.from_numpy(x).cuda(), yd, n, acc)
        e.wait()
        assert orc.max_norm_err(yd.cpu().numpy(), ry, mag) <= 2e-5, (rows, cols, n)


@pytest.mark.parametrize("t", [ol.Q6_K, ol.Q5_K, ol.Q8_0, ol.IQ4_NL, ol.IQ1_S, ol.IQ2_XXS])
@pytest.mark.parametrize("scale", [2.0 ** -105, 1e-30, 1e30, 1.5 * 2.0 ** 126])
def test_matvec_n_keeps_the_range_of_one_token(t, scale):
    """Units of very small and very large activations: as one token at a time gives them."""
    from macseek_b200 import quant as q, synthetic
    from macseek_b200.core import Enc
    if t in (ol.Q6_K, ol.Q5_K, ol.IQ1_S):
        scale = min(scale, 2.0 ** 112)       # their codes (and Q6_K scales, up to 2^12) meet the activation before the block's scale
    rows, cols, n, e = 64, 512, 3, Enc()
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    W = synthetic.random_weights(t, rows, cols, g, lo=1e-4, hi=5e-4)         # weights well below 1: the products stay in range
    x = torch.from_numpy(synth.randn(n * cols, 8).reshape(n, cols)).cuda()
    x = x / x.abs().amax()
    x[:, :32] *= scale                       # one unit; the largest products are not summed with others of their size
    x[:, 32:] *= min(scale, 1.0)
    if scale > 1:
        x[:, 1:32] *= 1e-6                   # (a sum of 32 would leave the range of float)
    one, many = torch.zeros(n, rows, device="cuda"), torch.zeros(n, rows, device="cuda")
    for i in range(n):
        q.encode_matvec(e, t, W, rows, cols, x[i].contiguous(), one[i])
    q.encode_matvec_n(e, t, W, rows, cols, x, many, n)
    e.wait()
    assert float(one.abs().max()) > 0 and bool(torch.isfinite(one).all())
    assert float((many.double() - one.double()).norm() / one.double().norm()) <= 1e-4



@pytest.mark.parametrize("cols", [65536, 65792, 86016])
@pytest.mark.parametrize("n", [1, 3])
def test_widest_q5k_rows(cols, n):
    """Both layouts of the quantised activations, and the widest row that fits shared memory."""
    from macseek_b200 import quant as q
    from macseek_b200.core import Enc
    orc, rows, e = ol.Oracle(), 5, Enc()
    W, x = synth.random_weights(ol.Q5_K, rows, cols, 3), synth.randn(n * cols, 4).reshape(n, cols)
    y = torch.zeros(n, rows, device="cuda")
    q.encode_matvec_n(e, ol.Q5_K, torch.from_numpy(W.view(np.uint8).reshape(-1).copy()).cuda(), rows, cols, torch.from_numpy(x).cuda(), y, n)
    e.wait()
    ry, mag = orc.matvec(ol.Q5_K, W, rows, cols, x, 1)
    assert orc.max_norm_err(y.cpu().numpy(), ry, mag) <= 2e-5
