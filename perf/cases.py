"""The work a user of this package has it do, as timed cases: one dict per case, made ready by prepare() and run by run().

Every pass goes through the public entry points of the host modules (quant, arch, attn, moe_layer, dec_layer), with the
shapes of the package's own configurations: the benchmark's layer (hidden 4096, experts of 2048, 64 x 128 FP8 index heads,
rows of 512 + 64 bf16) and the reference model's (hidden 5120, experts of 2304, 32 index heads with F16 keys, rows of 512
f16).  Weights are the seeded synthetic blocks of `synthetic`, made on the device.

Kinds of case:
  decode       one token through whole layers and the output head, replayed from a CUDA graph as the benchmark does
  matvec       a projection of 1 .. 16 tokens (single-stream decode, several streams, speculative drafts)
  matmul       a prefill projection, activations given as F32 or as half
  moe_prefill  the MoE part of a prefill chunk: router selection, routing lists, their offsets to the host (the call takes
               them there), grouped expert GEMMs
  moe_decode   one token through router + experts, called eagerly
  attend       one token's index decode (plain or restricted to candidate blocks) and sparse attention, called eagerly
  sample       the sampling head on rows of logits
  mix          hyper-connection boundaries of a layer, and for single tokens the KV compressor
"""
import functools
import math

import torch

from macseek_b200 import arch, attn, dec_layer, moe_layer, quant as q, synthetic
from macseek_b200.core import Enc
from macseek_b200.shapes import BLOCK, QType, row_bytes

E_BENCH = {"dim": 4096, "inter": 2048, "experts": 384, "k": 8, "t_gate_up": "IQ1_S", "t_down": "IQ2_XXS", "t_shared": "Q8_0"}
E_REF = {"dim": 5120, "inter": 2304, "experts": 384, "k": 6, "t_gate_up": "IQ1_S", "t_down": "IQ1_S", "t_shared": "Q6_K"}


def listed():
    return [
        # the benchmark's decode step at its 200K-token context (two of its 43 layers and the whole head)
        {"name": "decode_200k", "kind": "decode", "layers": 2, "kv_len": 200000},
        # the same step early in a conversation: every key is selected, launches and latency are what is left
        {"name": "decode_1500", "kind": "decode", "layers": 2, "kv_len": 1500},
        # the smallest projection of the benchmark's sweep: one launch, a 3 MB matrix
        {"name": "matvec_iq1s", "kind": "matvec", "t": "IQ1_S", "rows": 4096, "cols": 4096, "n": 1, "norm": False},
        # a projection for a few streams at once (the sweep's batch of 4)
        {"name": "matvec_q6k_4", "kind": "matvec", "t": "Q6_K", "rows": 16384, "cols": 4096, "n": 4, "norm": False},
        # prefill projections: a full chunk, and a short prompt of odd length
        {"name": "matmul_q6k_4096", "kind": "matmul", "t": "Q6_K", "rows": 4096, "cols": 4096, "n": 4096, "half": False},
        {"name": "matmul_q8_77", "kind": "matmul", "t": "Q8_0", "rows": 5120, "cols": 4096, "n": 77, "half": False},
        # MoE prefill: a full chunk of the reference model's layer with its benchmark's routing (every expert gets tokens),
        # and a chunk of odd length of the benchmark layer with a skewed router
        dict(E_REF, name="moe_prefill_4096", kind="moe_prefill", n=4096, routing="sample"),
        dict(E_BENCH, name="moe_prefill_999", kind="moe_prefill", n=999, routing="bias"),
        # one token of the reference model's MoE and attention, call by call
        dict(E_REF, name="moe_decode", kind="moe_decode"),
        {"name": "attend_50k", "kind": "attend", "shape": "reference", "kv_len": 50003, "cand": False},
        # the sampling head's top-k over one token's logits
        {"name": "sample_topk", "kind": "sample", "what": "topk", "rows": 1, "vocab": 129280, "k": 64},
        # what one token's layer does around its two halves: both hyper-connection boundaries and the compressor
        {"name": "mix_1", "kind": "mix", "dim": 5120, "n": 1, "ratio": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "matvec", "matvec", "matmul", "matmul", "moe_prefill", "moe_prefill", "moe_decode", "attend",
                       "sample", "mix"])
    if kind == "decode":
        return {"kind": kind, "layers": rng.choice([1, 2]), "kv_len": _log(rng, 64, 200000)}
    if kind == "matvec":
        t = rng.choice(["Q6_K", "Q8_0", "Q5_K", "IQ4_NL", "IQ2_XXS", "IQ1_S", "BF16"])
        n = rng.choice([1, 1, rng.randint(2, 16)])
        return {"kind": kind, "t": t, "rows": _log(rng, 512, 40000), "cols": 256 * rng.randint(4, 48), "n": n,
                "norm": n == 1 and rng.random() < 0.5}
    if kind == "matmul":
        t = rng.choice(["Q6_K", "Q8_0", "Q5_K", "IQ4_NL", "IQ2_XXS", "IQ1_S", "BF16", "F16"])
        return {"kind": kind, "t": t, "rows": _log(rng, 512, 8192), "cols": 256 * rng.randint(4, 32), "n": _log(rng, 17, 4096),
                "half": rng.random() < 0.5}
    if kind == "moe_prefill":
        return dict(rng.choice([E_BENCH, E_REF]), kind=kind, n=_log(rng, 16, 3500), routing=rng.choice(["sample", "bias"]))
    if kind == "moe_decode":
        return dict(rng.choice([E_BENCH, E_REF]), kind=kind, t_down=rng.choice(["IQ1_S", "IQ2_XXS"]),
                    t_shared=rng.choice(["Q8_0", "Q6_K"]), k=rng.randint(4, 8), experts=rng.randint(64, 384))
    if kind == "attend":
        kv = _log(rng, 300, 200000)
        return {"kind": kind, "shape": rng.choice(["reference", "benchmark"]), "kv_len": kv, "cand": kv > 20000 and rng.random() < 0.5}
    if kind == "sample":
        return {"kind": kind, "what": rng.choice(["topk", "argmax", "log_softmax"]), "rows": rng.choice([1, rng.randint(2, 16)]),
                "vocab": _log(rng, 32000, 160000), "k": rng.randint(1, 64)}
    return {"kind": kind, "dim": rng.choice([4096, 5120]), "n": rng.choice([1, _log(rng, 2, 256)]), "ratio": rng.choice([1, 2])}


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


@functools.lru_cache(maxsize=4)
def _rope(n):
    return torch.from_numpy(attn.make_rope_table(n, True)).cuda()


# ---------------------------------------------------------------------------------------------------- prepare / run
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_decode(c, seed):
    cfg = dec_layer.DecConfig(n_layers=c["layers"], kv_len=c["kv_len"])
    dev = torch.device("cuda", torch.cuda.current_device())
    model = dec_layer.SyntheticModel(cfg, seed=seed, device=dev)
    h_in = torch.randn(cfg.dim, device=dev, generator=_gen(seed + 1))
    stream = torch.cuda.Stream(device=dev)
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        model.bufs.h.copy_(h_in)
        model.forward_token(Enc(stream))
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            model.bufs.h.copy_(h_in)
            model.forward_token(Enc(torch.cuda.current_stream()))
    stream.synchronize()
    slot = (cfg.kv_len - 1) % cfg.window
    out = {"logits": model.bufs.logits, "next_id": model.bufs.next_id, "h": model.bufs.h,
           "window_rows": [st.win[slot] for st in model.state]}
    return {"run": _run_decode, "graph": graph, "model": model, "h_in": h_in, "out": out}


def _run_decode(s):
    s["graph"].replay()
    return s["out"]


def _prepare_matvec(c, seed):
    g, t = _gen(seed), QType[c["t"]]
    s = {"run": _run_matvec, "c": c, "t": t, "e": Enc()}
    s["W"] = synthetic.random_weights(t, c["rows"], c["cols"], g)
    s["x"] = torch.randn(c["n"], c["cols"], device="cuda", generator=g)
    s["gain"] = 1 + 0.1 * torch.randn(c["cols"], device="cuda", generator=g)
    s["y"] = torch.zeros(c["n"], c["rows"], device="cuda")
    return s


def _run_matvec(s):
    c = s["c"]
    if c["norm"]:
        q.encode_matvec_rmsnorm(s["e"], s["t"], s["W"], c["rows"], c["cols"], s["x"], s["gain"], 1e-6, s["y"])
    elif c["n"] == 1:
        q.encode_matvec(s["e"], s["t"], s["W"], c["rows"], c["cols"], s["x"], s["y"])
    else:
        q.encode_matvec_n(s["e"], s["t"], s["W"], c["rows"], c["cols"], s["x"], s["y"], c["n"])
    return s["y"]


def _prepare_matmul(c, seed):
    g, t = _gen(seed), QType[c["t"]]
    s = {"run": _run_matmul, "c": c, "t": t, "e": Enc()}
    s["W"] = synthetic.random_weights(t, c["rows"], c["cols"], g)
    x = torch.randn(c["n"], c["cols"], device="cuda", generator=g)
    s["x"] = x.half() if c["half"] else x
    s["y"] = torch.zeros(c["n"], c["rows"], device="cuda")
    need = q.matmul_scratch_bytes(t, c["rows"], c["cols"], c["n"], not c["half"])
    s["scratch"] = torch.zeros(max(need, 16), dtype=torch.uint8, device="cuda")
    return s


def _run_matmul(s):
    c = s["c"]
    if c["half"]:
        q.encode_matmul_h(s["e"], s["t"], s["W"], c["rows"], c["cols"], s["x"], s["y"], c["n"], False, 0, s["scratch"])
    else:
        q.encode_matmul(s["e"], s["t"], s["W"], c["rows"], c["cols"], s["x"], s["y"], c["n"], False, s["scratch"])
    return s["y"]


def _moe_weights(c, g):
    return moe_layer.MoeLayerWeights(c["dim"], c["inter"], c["experts"], QType[c["t_gate_up"]], QType[c["t_down"]],
                                     QType[c["t_shared"]]).randomize(g)


def _router_logits(c, n, g):
    """Logits [n][experts].  "bias": N(0, 1) plus a log-Zipf(1.1) popularity over a random order of the experts (a few take
    most tokens); "sample": the top-k of these is a draw without replacement from Zipf(0.8) popularities."""
    E = c["experts"]
    perm = torch.randperm(E, device="cuda", generator=g)
    rank = torch.empty(E, device="cuda")
    rank[perm] = torch.arange(1, E + 1, device="cuda", dtype=torch.float32)
    if c["routing"] == "bias":
        return torch.randn(n, E, device="cuda", generator=g) - 1.1 * torch.log(rank)
    u = torch.rand(n, E, device="cuda", generator=g).clamp_(1e-9, 1 - 1e-7)
    return -0.8 * torch.log(rank) - torch.log(-torch.log(u))


def _prepare_moe_prefill(c, seed):
    g = _gen(seed)
    n, k, E = c["n"], c["k"], c["experts"]
    lw = _moe_weights(c, g)
    a = q.MoePrefillArgs(c["dim"], c["inter"])
    a.t_gate_up, a.t_down, a.t_shared = lw.t_gate_up, lw.t_down, lw.t_shared
    a.n_tokens, a.k_per_token, a.has_shared, a.shared = n, k, True, lw.shared
    a.slots = [q.ExpertSlot(*lw.expert_views(e)) for e in range(E)]
    lists = arch.RouteLists(n, k, E)
    a.tok, a.wt, a.slot_of = lists.tok, lists.w, lists.slot_of
    a.X = torch.randn(n, c["dim"], device="cuda", generator=g)
    a.Y = torch.randn(n, c["dim"], device="cuda", generator=g)
    a.scratch = torch.empty(q.moe_prefill_scratch_bytes(n * k, n, E, c["dim"], c["inter"]), dtype=torch.uint8, device="cuda")
    return {"run": _run_moe_prefill, "c": c, "e": Enc(), "lw": lw, "a": a, "lists": lists, "logits": _router_logits(c, n, g),
            "ids": torch.zeros(n, k, dtype=torch.int32, device="cuda"), "w": torch.zeros(n, k, device="cuda")}


def _run_moe_prefill(s):
    c, a, lists = s["c"], s["a"], s["lists"]
    arch.encode_router_topk(s["e"], s["logits"], None, s["ids"], s["w"], c["n"], c["k"], arch.SCORE_SIGMOID, 1.0)
    arch.encode_route_lists(s["e"], s["ids"], s["w"], c["n"], lists)
    a.offs = lists.offsets.tolist()
    q.encode_moe_prefill(s["e"], a)
    return {"y": a.Y, "ids": s["ids"], "offsets": lists.offsets}


def _prepare_moe_decode(c, seed):
    g = _gen(seed)
    lw = _moe_weights(c, g)
    return {"run": _run_moe_decode, "e": Enc(), "lw": lw, "b": moe_layer.MoeLayerBufs(c["dim"], c["inter"], c["experts"], c["k"]),
            "x": torch.randn(c["dim"], device="cuda", generator=g), "y": torch.randn(c["dim"], device="cuda", generator=g)}


def _run_moe_decode(s):
    moe_layer.encode_moe_layer(s["e"], s["lw"], s["b"], s["x"], s["y"], arch.SCORE_SQRT_SOFTPLUS, arch.kRouteScale)
    return {"y": s["y"], "ids": s["b"].ids, "w": s["b"].w}


def _prepare_attend(c, seed):
    g = _gen(seed)
    sh = attn.Shape.reference() if c["shape"] == "reference" else attn.Shape.benchmark()
    n = c["kv_len"]
    st = attn.DecodeState(sh, n, _rope(n + 1))
    st.ckv.normal_(0, 1, generator=g)
    st.win.normal_(0, 1, generator=g)
    keys = torch.empty(st.ikey.shape, dtype=torch.float16, device="cuda").normal_(0, 1, generator=g)
    st.ikey.copy_(keys if sh.key_type == attn.KEY_F16 else keys.to(torch.float8_e4m3fn).view(torch.uint8))
    del keys
    rnd = lambda m: torch.randn(m, device="cuda", generator=g)
    s = {"run": _run_attend, "c": c, "e": Enc(), "st": st, "iq": rnd(sh.index_heads * sh.index_dim), "iw": rnd(sh.index_heads),
         "q": rnd(sh.heads * sh.D), "sinks": rnd(sh.heads), "out": torch.zeros(sh.heads, sh.D, device="cuda")}
    if c["cand"]:      # the layer before this one listed the candidate blocks, from an index query close to this layer's
        near = s["iq"] + 0.5 * rnd(s["iq"].numel())
        attn.encode_index_decode(s["e"], st, near, s["iw"], n - 1, n, cand_source=True)
    return s


def _run_attend(s):
    c, st, n = s["c"], s["st"], s["c"]["kv_len"]
    if c["cand"]:
        attn.encode_index_decode_list(s["e"], st, s["iq"], s["iw"], n - 1, n)
    else:
        attn.encode_index_decode(s["e"], st, s["iq"], s["iw"], n - 1, n)
    attn.encode_sparse(s["e"], st, s["q"], s["sinks"], s["out"], n - 1)
    return {"out": s["out"], "topk": st.topk}


def _prepare_sample(c, seed):
    g = _gen(seed)
    rows, V = c["rows"], c["vocab"]
    f = lambda *shape: torch.zeros(*shape, device="cuda")
    i = lambda *shape: torch.zeros(*shape, dtype=torch.int32, device="cuda")
    return {"run": _run_sample, "c": c, "e": Enc(), "x": 3 * torch.randn(rows, V, device="cuda", generator=g), "seed": seed,
            "scratch": arch.sample_scratch(rows), "v": f(rows, arch.SAMPLE_K), "i": i(rows, arch.SAMPLE_K), "lse": f(rows),
            "idx": i(rows), "val": f(rows), "out": f(rows, V) if c["what"] == "log_softmax" else None}


def _run_sample(s):
    c, e = s["c"], s["e"]
    rows, V, k = c["rows"], c["vocab"], c["k"]
    if c["what"] == "topk":
        arch.encode_sample_topk(e, s["x"], rows, V, k, 0.8, s["v"], s["i"], s["lse"], s["scratch"])
        return {"v": s["v"], "i": s["i"], "lse": s["lse"]}
    if c["what"] == "argmax":
        arch.encode_argmax_rows(e, s["x"], rows, V, s["idx"], s["val"], s["scratch"], 0.8, s["seed"])
        return {"idx": s["idx"], "val": s["val"]}
    arch.encode_log_softmax(e, s["x"], s["out"], rows, V)
    return s["out"]


def _prepare_mix(c, seed):
    g = _gen(seed)
    n, D, dev = c["n"], c["dim"], "cuda"
    rnd = lambda *shape, sd=1.0: torch.empty(*shape, device=dev).normal_(0, sd, generator=g)
    s = {"run": _run_mix, "c": c, "e": Enc(), "h": rnd(n, 4, D), "x_sub": rnd(n, D), "fn": [rnd(24, 4 * D, sd=0.02) for _ in range(2)],
         "scale": torch.tensor([0.7, 1.3, 0.9], device=dev), "base": rnd(24), "gain": 1 + rnd(D, sd=0.1),
         "mix0": rnd(n, 24).abs() + 0.05, "scratch": arch.hc_scratch(n)}
    for name in ("h1", "h2"):
        s[name] = torch.zeros(n, 4, D, device=dev)
    for name in ("x1", "x2"):
        s[name] = torch.zeros(n, D, device=dev)
    for name in ("mix1", "mix2"):
        s[name] = torch.zeros(n, 24, device=dev)
    if n == 1:
        sh = attn.Shape.reference()
        s["st"] = attn.DecodeState(sh, 1024, _rope(1153))
        s["c_kv"], s["c_gate"], s["c_norm"] = rnd(sh.D), rnd(sh.D), 1 + rnd(sh.D, sd=0.1)
        s["wk"], s["k_norm"] = rnd(sh.index_dim * sh.D, sd=0.05).to(torch.bfloat16), 1 + rnd(sh.index_dim, sd=0.1)
        s["part"] = rnd(2, c["ratio"], sh.D)
    return s


def _run_mix(s):
    c, e = s["c"], s["e"]
    arch.encode_hc_step(e, s["h"], s["h1"], s["x_sub"], s["mix0"], s["fn"][0], s["scale"], s["base"], s["mix1"], s["gain"], s["x1"],
                        c["dim"], s["scratch"], c["n"])
    arch.encode_hc_step(e, s["h1"], s["h2"], s["x_sub"], s["mix1"], s["fn"][1], s["scale"], s["base"], s["mix2"], s["gain"], s["x2"],
                        c["dim"], s["scratch"], c["n"])
    out = {"h": s["h2"], "x": [s["x1"], s["x2"]], "mix": [s["mix1"], s["mix2"]]}
    if c["n"] == 1:
        pos = 1001                      # the last token of its group at either ratio: a row is written
        attn.encode_compress(e, s["st"], s["c_kv"], s["c_gate"] if c["ratio"] > 1 else None, s["c_norm"], s["wk"], s["k_norm"],
                             s["part"], c["ratio"], pos)
        out["row"], out["key"], out["part"] = s["st"].ckv[pos // c["ratio"]], s["st"].ikey[pos // c["ratio"]], s["part"]
    return out


# ---------------------------------------------------------------------------------------------------- work / tolerance
def _moe_bytes(c, used):
    gu, dn = QType[c["t_gate_up"]], QType[c["t_down"]]
    expert = 2 * row_bytes(gu, c["dim"]) * c["inter"] + row_bytes(dn, c["inter"]) * c["dim"]
    sh = QType[c["t_shared"]]
    return used * expert + 2 * row_bytes(sh, c["dim"]) * c["inter"] + row_bytes(sh, c["inter"]) * c["dim"]


def _weights(t, rows, cols):
    be, _ = BLOCK.get(QType[t], (1, 0))
    assert cols % be == 0
    return row_bytes(QType[t], cols) * rows


def work(c):
    kind = c["kind"]
    if kind == "decode":
        cfg = dec_layer.DecConfig(n_layers=c["layers"], kv_len=c["kv_len"])
        lb = cfg.layer_bytes()
        rows = min(cfg.topk, cfg.kv_len) + min(cfg.window, cfg.kv_len)
        layer = lb["total"] - lb["kv_rows"] + rows * cfg.D * 2
        hD = cfg.heads * cfg.D
        mults = (cfg.dim * (cfg.q_lora + cfg.D) + cfg.q_lora * hD + cfg.o_a_rows * hD // cfg.o_groups + cfg.dim * cfg.o_a_rows
                 + cfg.index_heads * (cfg.dim + cfg.q_lora * cfg.index_dim) + cfg.kv_len * cfg.index_heads * cfg.index_dim
                 + 2 * rows * hD + cfg.n_experts * cfg.dim + 3 * (cfg.top_k + 1) * cfg.dim * cfg.inter)
        return {"bytes": layer * c["layers"] + cfg.head_bytes() + 4 * cfg.vocab, "flops": 2.0 * (mults * c["layers"] + cfg.vocab * cfg.dim)}
    if kind == "matvec":
        return {"bytes": _weights(c["t"], c["rows"], c["cols"]) + 4 * c["n"] * (c["rows"] + c["cols"]),
                "flops": 2.0 * c["n"] * c["rows"] * c["cols"]}
    if kind == "matmul":
        return {"bytes": _weights(c["t"], c["rows"], c["cols"]) + c["n"] * ((2 if c["half"] else 4) * c["cols"] + 4 * c["rows"]),
                "flops": 2.0 * c["n"] * c["rows"] * c["cols"]}
    if kind == "moe_prefill":
        n, k, E = c["n"], c["k"], c["experts"]
        p = [1.0 / (r + 1) ** (0.8 if c["routing"] == "sample" else 1.1) for r in range(E)]
        used = sum(1 - (1 - min(1.0, k * v / sum(p))) ** n for v in p)       # experts that get a token, about
        return {"bytes": _moe_bytes(c, used) + n * (12 * c["dim"] + 4 * E + 24 * k),
                "flops": 2.0 * 3 * c["dim"] * c["inter"] * n * (k + 1)}
    if kind == "moe_decode":
        return {"bytes": _moe_bytes(c, c["k"]) + 4 * c["experts"] * c["dim"] + 12 * c["dim"],
                "flops": 2.0 * (c["experts"] * c["dim"] + 3 * (c["k"] + 1) * c["dim"] * c["inter"])}
    if kind == "attend":
        sh = attn.Shape.reference() if c["shape"] == "reference" else attn.Shape.benchmark()
        n = min(c["kv_len"], sh.cand_blocks * sh.cand_bs) if c["cand"] else c["kv_len"]
        rows = min(sh.topk, c["kv_len"]) + min(sh.window, c["kv_len"])
        return {"bytes": n * sh.index_dim * (2 if sh.key_type == attn.KEY_F16 else 1) + rows * sh.D * 2 + 8 * sh.heads * sh.D,
                "flops": 2.0 * (n * sh.index_heads * sh.index_dim + 2 * rows * sh.heads * sh.D)}
    if kind == "sample":
        return {"bytes": (8 if c["what"] == "log_softmax" else 4) * c["rows"] * c["vocab"], "flops": 4.0 * c["rows"] * c["vocab"]}
    n, D = c["n"], c["dim"]
    return {"bytes": 2 * 4 * (24 * 4 * D + n * (8 * D + 2 * D)) + (2 * 128 * 512 if n == 1 else 0), "flops": 2.0 * 2 * n * 4 * D * (24 + 6)}


def tolerance(c):
    kind = c["kind"]
    if kind == "decode":
        # activations of every projection are rounded to 16 bits, index queries to 8 (FP8), rows are bf16: an earlier sum in
        # another order moves some of these roundings
        return {"rel": 2e-3, "max": 2e-2, "differ": 0.0}
    if kind == "matvec":
        return {"rel": 1e-4, "max": 1e-3}       # activations as 16-bit fixed point per 32 elements
    if kind == "matmul":
        return {"rel": 5e-4, "max": 5e-3}       # half operands, fp32 sums
    if kind == "moe_prefill":
        return {"rel": 1e-3, "max": 2e-2, "differ": 0.0}       # half operands, and a half intermediate
    if kind == "moe_decode":
        return {"rel": 1e-4, "max": 2e-3, "differ": 0.0}
    if kind == "attend":
        return {"rel": 1e-4, "max": 2e-3, "differ": 0.01}      # a near-tie at the selection's threshold
    if kind == "sample":
        return {"rel": 1e-5, "differ": 0.01}
    return {"rel": 1e-4, "max": 2e-3, "differ": 0.01}          # row and key are stored as f16
