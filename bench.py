#!/usr/bin/env python3
"""Benchmark of the per-token hot path: one full synthetic decode step at batch 1 with a 200K-token KV
-> decode tok/s.

  python bench.py --gpus 1 --steps 20 --warmup 3          this repository's CUDA path
  python bench.py --impl reference ...                    the reference's scalar CPU routines on the host cores
  torchrun ... bench.py --gpus N ...                      expert-parallel over N GPUs (one rank per GPU, NCCL)

Prints ONE JSON line (rank 0).  `value`: whole-job tok/s with the token's hidden state already in HBM (CUDA-graph
replays, CUDA events, max over ranks).  `e2e`: the same step driven from host buffers (H2D of the hidden state and D2H
of the sampled id inside the timed region).  `roofline`: the dominant kernel (MoE gate/up) timed live with CUDA events.
`cpu_baseline`: the CPU oracle / reference routines timed on a bounded sample of the same workload.
"""
import argparse
import json
import os
import subprocess
import sys
import tempfile
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)
sys.path.insert(0, os.path.join(ROOT, "tests"))

METRIC = "decode_tok_per_s_200k_ctx"
UNIT = "tok/s"
# DRAM bytes (read + write) of one moe_gu_kernel launch of the benchmark layer, all 8 routed experts resident:
# measured once with ncu (profiles/moe_gu_kernel_cfg3_ncu_full.txt); the algorithmic bytes are 44,040,192
NCU_GU_TRAFFIC_BYTES = 44_191_488     # dram__bytes_read.sum 44,190,976 + dram__bytes_write.sum 512


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--layers", type=int, default=43)
    ap.add_argument("--kv-len", type=int, default=200000)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--combine", default="peer", choices=["peer", "nccl"],
                    help="N > 1: how the ranks' partial MoE outputs are summed (peer-memory exchange, or an NCCL all-reduce)")
    ap.add_argument("--no-extras", action="store_true", help="skip the per-kernel roofline sweeps (cfg1/cfg2/cfg4)")
    return ap.parse_args()


def workload_config(a, world):
    return {"workload": "full synthetic decode step, batch 1, KV 200K: %d layers x (attention projections Q6_K, "
                        "64x128 FP8 indexer top-2048, sparse attention over 128+2048 bf16 rows of 576, 384-expert MoE "
                        "top-8 IQ1_S/IQ2_XXS + shared Q8_0) + Q6_K head 129280" % a.layers,
            "layers": a.layers, "kv_len": a.kv_len, "hidden": 4096, "experts": 384, "top_k": 8,
            "parallelism": "ep%d" % world,
            "l2": "inputs larger than L2: every step streams ~%.1f GB of distinct weights and caches" % (0.235 * a.layers + 0.43)}


# ------------------------------------------------------------------------------------------------ CPU sample
def cpu_token_seconds(a, use_ref=True, threads=None, row_div=1):
    """Time the CPU routines on a bounded sample of one token's work and scale to the whole token.  row_div > 1 times
    1 / row_div of every matrix's rows (and of the keys) and scales linearly: the single-thread run uses it to stay
    bounded.  Returns (seconds per token, dict describing the sample).  Imports nothing that loads the CUDA library."""
    import numpy as np
    import oracle_lib as ol
    import synth
    from macseek_b200.shapes import DecConfig
    c = DecConfig(n_layers=a.layers, kv_len=a.kv_len)
    orc = ol.Oracle()
    ref = ol.Ref.load(build=False) if use_ref else None
    T = threads or orc.threads
    rng = np.random.default_rng(0)

    def mv(t, rows, cols, groups=1):
        r = max(groups, (rows // row_div) // groups * groups)
        W = synth.random_weights(int(t), r, cols, rows + cols)
        x = synth.randn(cols * groups, 3)
        t0 = time.perf_counter()
        if ref is not None:
            ref.matvec(int(t), W, r, cols, x, groups, threads=T)
        else:
            orc.matvec(int(t), W, r, cols, x, groups, threads=T)
        return (time.perf_counter() - t0) * (rows / r)

    hD = c.heads * c.D
    layer = 0.0
    # attention projections
    layer += mv(c.t_attn, c.q_lora, c.dim) + mv(c.t_attn, c.D, c.dim) + mv(c.t_attn, hD, c.q_lora)
    layer += mv(c.t_index, c.index_heads, c.dim) + mv(c.t_index, c.index_heads * c.index_dim, c.q_lora)
    layer += mv(c.t_attn, c.o_a_rows, hD // c.o_groups, c.o_groups) + mv(c.t_attn, c.dim, c.o_a_rows)
    # MoE: router + 8 routed + shared
    Wr = (rng.standard_normal((c.n_experts, c.dim)) * 0.02).astype(np.float32)
    x = synth.randn(c.dim, 5)
    t0 = time.perf_counter()
    logits = Wr @ x
    orc.router(logits, np.zeros(c.n_experts, np.float32), c.top_k, c.score_fn, c.route_scale)
    layer += time.perf_counter() - t0
    for t, rows, cols, cnt in ((c.t_gate_up, c.inter, c.dim, 2 * c.top_k), (c.t_down, c.dim, c.inter, c.top_k),
                               (c.t_shared, c.inter, c.dim, 2), (c.t_shared, c.dim, c.inter, 1)):
        layer += mv(t, rows, cols) * cnt
    # indexer on a sample of the keys, exact top-k on full-length scores, sparse attention (full)
    n_keys = max(1000, min(c.kv_len, 20000) // row_div)
    keys = rng.standard_normal((n_keys, c.index_dim)).astype(np.float32)
    qi = rng.standard_normal((c.index_heads, c.index_dim)).astype(np.float32)
    wi = rng.standard_normal(c.index_heads).astype(np.float32)
    t0 = time.perf_counter()
    orc.index_scores(qi, wi, keys, threads=T)
    layer += (time.perf_counter() - t0) * (c.kv_len / n_keys)
    sc = rng.standard_normal(c.kv_len).astype(np.float32)
    t0 = time.perf_counter()
    orc.topk_sorted(sc, c.topk)
    layer += time.perf_counter() - t0
    rows = rng.standard_normal((c.window + c.topk, c.D)).astype(np.float32)
    qa = rng.standard_normal((c.heads, c.D)).astype(np.float32)
    tab = orc.rope_table(4, True)
    t0 = time.perf_counter()
    orc.sparse_attn(qa, tab[3], rows, np.zeros(c.heads, np.float32), threads=T)
    layer += time.perf_counter() - t0
    # head on a row sample
    n_head = 8192
    head = mv(c.t_head, n_head, c.dim) * (c.vocab / n_head)
    total = layer * c.n_layers + head
    frac = "" if row_div == 1 else " (1/%d of every matrix's rows and of the key sample, scaled)" % row_div
    return total, {"kind": "reference" if ref is not None else "port", "cores": T,
                   "sample": "one layer (projections, router, 8 routed + shared expert, sparse attention, top-k)%s "
                             "with the indexer on %d of %d keys and the head on %d of %d rows, scaled to %d layers + head; "
                             "%s" % (frac, n_keys, c.kv_len, max(1, n_head // row_div), c.vocab, c.n_layers,
                                     "matvec-shaped parts through the reference's own ref::dequant_row + double dot "
                                     "(oracle/_ref), router / indexer / attention at the benchmark's shapes through the C "
                                     "port because the reference fixes those shapes at compile time"
                                     if ref is not None else "C port of the reference routines (oracle/msb_oracle.c)")}


def cpu_baseline_dict(a):
    """The threaded figure (all host cores) with the single-thread-as-written figure beside it."""
    sec, info = cpu_token_seconds(a, use_ref=True)
    sec1, info1 = cpu_token_seconds(a, use_ref=True, threads=1, row_div=16)
    d = dict(info, value=1.0 / sec, unit=UNIT)
    d["single_thread"] = {"value": 1.0 / sec1, "unit": UNIT, "cores": 1, "sample": info1["sample"]}
    return d


def run_reference(a):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    import oracle_lib as ol
    ol.build_oracle()
    times = []
    info = None
    for i in range(a.warmup + a.steps):
        t, info = cpu_token_seconds(a, use_ref=True)
        if i >= a.warmup:
            times.append(t)
    sec = sum(times) / len(times)
    val = 1.0 / sec
    sec1, info1 = cpu_token_seconds(a, use_ref=True, threads=1, row_div=16)
    info = dict(info, single_thread={"value": 1.0 / sec1, "unit": UNIT, "cores": 1, "sample": info1["sample"]})
    line = {"impl": "reference", "metric": METRIC, "value": val, "unit": UNIT, "n_gpus": a.gpus, "steps": a.steps,
            "warmup": a.warmup, "ms_per_step": sec * 1e3, "higher_is_better": True, "scaling": "strong",
            "vs_baseline": None, "dtype": "f64 accumulate over f32 dequantised weights", "data": "synthetic",
            "config": workload_config(a, 1),
            "cpu_baseline": dict(info, value=val, unit=UNIT),
            "e2e": {"value": val, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
            "gpu_launches": 0}
    print(json.dumps(line))


# ------------------------------------------------------------------------------------------------ clocks
class ClockSampler:
    """SM clock and slowdown reasons of one GPU while the timed regions run: a thread that reads NVML every 10 ms
    (reading only; nothing is set), or -- without the NVML binding -- an `nvidia-smi -lms` child process."""
    Q = "index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown," \
        "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap"

    def __init__(self, index, pci_bus_id=None):
        self.index, self.pci, self.proc, self.path = index, pci_bus_id, None, None
        self.thread, self.stop_flag, self.samples, self.max_mhz, self.how = None, False, [], None, None

    def _nvml_loop(self, nv, h):
        import time
        bits = (("hw_slowdown", nv.nvmlClocksEventReasonHwSlowdown), ("hw_thermal_slowdown", nv.nvmlClocksEventReasonHwThermalSlowdown),
                ("sw_thermal_slowdown", nv.nvmlClocksEventReasonSwThermalSlowdown), ("sw_power_cap", nv.nvmlClocksEventReasonSwPowerCap))
        while not self.stop_flag:
            try:
                mhz = nv.nvmlDeviceGetClockInfo(h, nv.NVML_CLOCK_SM)
                mask = nv.nvmlDeviceGetCurrentClocksEventReasons(h)
                self.samples.append((float(mhz), [n for n, b in bits if mask & b]))
            except Exception:
                pass
            time.sleep(0.01)

    def start(self):
        try:
            import threading
            import pynvml as nv
            nv.nvmlInit()
            h = nv.nvmlDeviceGetHandleByPciBusId(self.pci.encode()) if self.pci else nv.nvmlDeviceGetHandleByIndex(self.index)
            self.max_mhz = float(nv.nvmlDeviceGetMaxClockInfo(h, nv.NVML_CLOCK_SM))
            self.thread = threading.Thread(target=self._nvml_loop, args=(nv, h), daemon=True)
            self.thread.start()
            self.how = "nvml thread, 10 ms"
            return
        except Exception:
            self.thread = None
        try:
            fd, self.path = tempfile.mkstemp(suffix=".csv")
            os.close(fd)
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), "--query-gpu=" + self.Q,
                                          "--format=csv,noheader,nounits", "-lms", "100"],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
            self.how = "nvidia-smi -lms 100"
        except Exception:
            self.proc = None

    def stop(self):
        out = {"sm_mhz": None, "sm_max_mhz": None, "reasons": []}
        if self.thread is not None:
            self.stop_flag = True
            self.thread.join(timeout=2)
            sm = sorted(v for v, _ in self.samples)
            if sm:
                reasons = sorted({r for _, rs in self.samples for r in rs})
                out = {"sm_mhz": sm[len(sm) // 2], "sm_max_mhz": self.max_mhz, "reasons": reasons, "samples": len(sm),
                       "how": self.how}
            return out
        if self.proc is None:
            return out
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        sm, mx, reasons = [], [], set()
        try:
            for ln in open(self.path):
                f = [v.strip() for v in ln.split(",")]
                if len(f) < 9:
                    continue
                try:
                    sm.append(float(f[1])); mx.append(float(f[2]))
                except ValueError:
                    continue
                for name, v in zip(("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"), f[5:9]):
                    if v.lower().startswith("active"):
                        reasons.add(name)
            os.unlink(self.path)
        except Exception:
            pass
        if sm:
            sm.sort()
            out = {"sm_mhz": sm[len(sm) // 2], "sm_max_mhz": max(mx), "reasons": sorted(reasons), "samples": len(sm),
                   "how": self.how}
        return out


# ------------------------------------------------------------------------------------------------ our arm
def run_ours(a):
    import torch
    import torch.distributed as dist
    from macseek_b200 import quant as q
    from macseek_b200.core import Enc
    from macseek_b200.dec_layer import DecConfig, SyntheticModel

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    group = None
    if world > 1:
        dist.init_process_group("nccl", device_id=dev)
        group = dist.group.WORLD
    cfg = DecConfig(n_layers=a.layers, kv_len=a.kv_len)
    model = SyntheticModel(cfg, seed=1234, device=dev, ep_rank=rank, ep_world=world, group=group, combine=a.combine)
    b = model.bufs
    gen = torch.Generator(device=dev)
    gen.manual_seed(99)
    h_in = torch.empty(cfg.dim, dtype=torch.float32, device=dev).normal_(0, 1, generator=gen)
    h_host = h_in.cpu().pin_memory()
    id_host = torch.zeros(1, dtype=torch.int32).pin_memory()

    stream = torch.cuda.Stream(device=dev)
    with torch.cuda.stream(stream):
        e = Enc(stream)
        for _ in range(max(a.warmup, 3)):                      # eager warm-up: first-use set-up, NCCL channels
            b.h.copy_(h_in)
            launches = model.forward_token(e)
        e.wait()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            b.h.copy_(h_in)
            model.forward_token(Enc(torch.cuda.current_stream()))
        for _ in range(a.warmup):
            graph.replay()
        stream.synchronize()

        def barrier():
            if world > 1:
                dist.barrier()
            torch.cuda.synchronize()

        # ---- value: device-resident input, K graph replays
        try:
            pr = torch.cuda.get_device_properties(dev)
            pci = "%08x:%02x:%02x.0" % (pr.pci_domain_id, pr.pci_bus_id, pr.pci_device_id)
        except Exception:
            pci = None
        sampler = ClockSampler(local, pci)
        barrier()
        sampler.start()
        ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        ev0.record(stream)
        for _ in range(a.steps):
            graph.replay()
        ev1.record(stream)
        barrier()
        ms = ev0.elapsed_time(ev1)
        # ---- e2e: host hidden state in, sampled id out, every step
        barrier()
        ev2, ev3 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        ev2.record(stream)
        for _ in range(a.steps):
            h_in.copy_(h_host, non_blocking=True)
            graph.replay()
            id_host.copy_(b.next_id, non_blocking=True)
            stream.synchronize()
        ev3.record(stream)
        barrier()
        ms_e2e = ev2.elapsed_time(ev3)
        clocks = sampler.stop()

        # ---- roofline of the dominant kernel (MoE gate/up of all experts), timed alone, one launch per layer.  Each
        # layer's launch uses the ids its own router produced for this token (logged in one eager pass), so that the
        # byte count is the sum over layers of the experts actually resident here.
        ids_log = torch.zeros(cfg.n_layers, cfg.top_k, dtype=torch.int32, device=dev)
        model.ids_log = ids_log
        b.h.copy_(h_in)
        model.forward_token(e)
        e.wait()
        model.ids_log = None
        ids_host = ids_log.cpu().tolist()
        lw0 = model.layers[0].moe
        s_lo, s_hi = model.s_lo, model.s_hi
        shared_gu = 2 * q.row_bytes(cfg.t_shared, cfg.dim) * (s_hi - s_lo)
        shared_d = q.row_bytes(cfg.t_shared, s_hi - s_lo) * cfg.dim
        n_local_layers = [sum(1 for i in ids_host[l] if lw0.expert_lo <= i < lw0.expert_hi) for l in range(cfg.n_layers)]
        reps = max(1, 40 // cfg.n_layers)
        n_gu = reps * cfg.n_layers
        gu_bytes = sum(n * 2 * lw0.gu_bytes + shared_gu for n in n_local_layers) / cfg.n_layers
        d_bytes = sum(n * lw0.d_bytes + shared_d for n in n_local_layers) / cfg.n_layers

        def moe_graph(part):
            g = torch.cuda.CUDAGraph()
            y_tmp = torch.zeros(cfg.dim, dtype=torch.float32, device=dev)
            with torch.cuda.graph(g, stream=stream):
                for _ in range(reps):
                    for l in range(cfg.n_layers):
                        w = model.layers[l].moe
                        args = q.MoeDecodeArgs(cfg.dim, cfg.inter)
                        args.t_gate_up, args.t_down, args.t_shared = cfg.t_gate_up, cfg.t_down, cfg.t_shared
                        args.n_routed, args.has_shared, args.shared = cfg.top_k, True, w.shared
                        args.weights, args.x, args.y, args.scratch = b.moe.w, b.x, y_tmp, b.moe.moe_scratch
                        ec = Enc(torch.cuda.current_stream())
                        if world == 1:
                            q.encode_moe_decode_ids(ec, args, w.table, ids_log[l], w.expert_lo, w.expert_hi, part)
                        else:
                            # the expert-parallel form has no "part" argument: time both launches, gate/up = pair - down
                            q.encode_moe_decode_ep(ec, args, w.table, ids_log[l], w.expert_lo, w.expert_hi, s_lo, s_hi, None)
            g.replay()
            stream.synchronize()
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0.record(stream)
            g.replay()
            t1.record(stream)
            stream.synchronize()
            return g, t0.elapsed_time(t1) * 1e3 / n_gu

        if world == 1:
            ggraph, gu_us = moe_graph(q.MoePart.GuAll)
            dgraph, d_us = moe_graph(q.MoePart.DownAll)
            pair_us = gu_us + d_us
        else:
            ggraph, pair_us = moe_graph(q.MoePart.All)
            dgraph = None
            gu_us = d_us = None
        # the output head (Q6_K 129280 x dim) alone: the one launch of the step that is purely a weight stream
        hgraph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(hgraph, stream=stream):
            for _ in range(4):
                q.encode_matvec(Enc(torch.cuda.current_stream()), cfg.t_head, model.w_head, cfg.vocab, cfg.dim, b.x,
                                b.logits, False, 1)
        hgraph.replay()
        stream.synchronize()
        ev6, ev7 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        ev6.record(stream)
        hgraph.replay()
        ev7.record(stream)
        stream.synchronize()
        head_us = ev6.elapsed_time(ev7) * 1e3 / 4
        # ---- expert parallel: the N-rank step must compute what one GPU computes.  A 2-layer model with ALL experts
        # and the same model split over the ranks (experts are seeded by global id) decode the same token.
        ep_check = None
        if world > 1:
            ccfg = DecConfig(n_layers=2, kv_len=8192)
            full = SyntheticModel(ccfg, seed=77, device=dev)
            part = SyntheticModel(ccfg, seed=77, device=dev, ep_rank=rank, ep_world=world, group=group, combine=a.combine,
                                  comm=model.comm)
            gen2 = torch.Generator(device=dev)
            gen2.manual_seed(5)
            hc = torch.empty(cfg.dim, dtype=torch.float32, device=dev).normal_(0, 1, generator=gen2)
            full.bufs.h.copy_(hc)
            full.forward_token(e)
            part.bufs.h.copy_(hc)
            part.forward_token(e)
            e.wait()
            ref_l, got_l = full.bufs.logits, part.bufs.logits
            rel = float((got_l - ref_l).abs().max() / ref_l.abs().max())
            same_id = int(full.bufs.next_id.item()) == int(part.bufs.next_id.item())
            chk = torch.stack([got_l.view(torch.int32).to(torch.int64).sum(), part.bufs.next_id.to(torch.int64)[0]])
            allchk = [torch.zeros_like(chk) for _ in range(world)]
            dist.all_gather(allchk, chk)
            ranks_identical = all(torch.equal(c, allchk[0]) for c in allchk)
            ep_check = {"ep_matches_n1": bool(same_id and rel <= 1e-3), "next_id_equal": same_id, "max_rel_logit_diff": rel,
                        "ranks_bit_identical": bool(ranks_identical), "model": "2 layers, all experts vs split over ranks"}
            del full, part
        extras = {}
        if world == 1 and not a.no_extras:
            import kernel_bench as kb
            T = q.QType
            sweep = [kb.matvec_case(T.IQ1_S, 4096, 4096, 1, quiet=True)]                         # cfg1
            for t in (T.Q8_0, T.Q6_K, T.Q5_K, T.IQ4_NL, T.IQ2_XXS):                               # cfg2
                for rows, cols in ((4096, 4096), (16384, 4096), (4096, 16384)):
                    for n in (1, 4):
                        sweep.append(kb.matvec_case(t, rows, cols, n, quiet=True))
            extras["matvec"] = sweep
            extras["prefill"] = kb.moe_prefill_case(4096, quiet=True)
        if world > 1 and not a.no_extras:
            # cfg4's prefill layer expert-parallel: tokens and experts sharded over the ranks, all-to-all dispatch and
            # combine, every rank's result checked against the single-GPU kernels on the same tokens
            import kernel_bench as kb
            try:
                extras["prefill_ep"] = kb.moe_prefill_ep_case(4096, check=True, quiet=True)
            except Exception as ex:
                extras["prefill_ep"] = {"error": str(ex)[:200]}
        st = __import__("macseek_b200._lib", fromlist=["x"]).device_status()
        if st:
            raise RuntimeError("device-side failure word %d" % st)

    # max over ranks
    t = torch.tensor([ms, ms_e2e], dtype=torch.float64, device=dev)
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    ms, ms_e2e = t.tolist()
    if rank == 0:
        peaks = {}
        try:
            peaks = json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))
        except Exception:
            pass
        peak = float(peaks.get("hbm_gbs", 6650.0))
        peak_src = "measured (MEASURED_PEAKS.json hbm_gbs)" if "hbm_gbs" in peaks else "fallback 6650 GB/s"
        tf_peak = float(peaks.get("bf16_tflops", 1590.0))
        if world == 1:
            r_kernel = "moe_gu_kernel (gate/up + SwiGLU of the 8 routed experts + shared expert)"
            r_us, r_bytes = gu_us, gu_bytes
        else:
            r_kernel = "moe_gu_kernel + moe_down_kernel pair on the experts resident on rank 0 and its slice of the shared expert"
            r_us, r_bytes = pair_us, gu_bytes + d_bytes
        achieved = r_bytes / r_us / 1e3
        lb = cfg.layer_bytes(1.0 / world)
        token_bytes = lb["total"] * cfg.n_layers + cfg.head_bytes()
        line = {"metric": METRIC, "value": a.steps / (ms / 1e3), "unit": UNIT, "n_gpus": world, "steps": a.steps,
                "warmup": a.warmup, "ms_per_step": ms / a.steps, "higher_is_better": True, "scaling": "strong",
                "vs_baseline": None, "dtype": "u8 codes x int16 fixed-point activations (dp4a), f32 accumulate; fp8 tcgen05 (indexer) and bf16 mma (attention)",
                "data": "synthetic", "config": dict(workload_config(a, world), combine=(a.combine if world > 1 else "none")),
                "e2e": {"value": a.steps / (ms_e2e / 1e3), "unit": UNIT, "h2d_bytes_per_step": cfg.dim * 4,
                        "d2h_bytes_per_step": 4},
                "gpu_launches": launches * a.steps,
                "clocks": clocks,
                "roofline": {"bound": "hbm", "kernel": r_kernel,
                             "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                             "peak_source": peak_src, "us_per_launch": r_us, "bytes_per_launch": r_bytes,
                             "local_experts_per_layer": {"min": min(n_local_layers), "mean": sum(n_local_layers) / len(n_local_layers),
                                                         "max": max(n_local_layers)},
                             # dram__bytes_read.sum + dram__bytes_write.sum of one launch with all 8 routed
                             # experts resident, from the ncu capture summarised under profiles/
                             "traffic": NCU_GU_TRAFFIC_BYTES if world == 1 else None},
                "roofline_head": {"bound": "hbm", "kernel": "matvec_kernel<Q6_K> output head %d x %d" % (cfg.vocab, cfg.dim),
                                  "achieved": cfg.head_bytes() / head_us / 1e3, "peak": peak, "unit": "GB/s",
                                  "frac": cfg.head_bytes() / head_us / 1e3 / peak, "us_per_launch": head_us,
                                  "bytes_per_launch": cfg.head_bytes()},
                "step_bytes": {"per_token_this_rank": token_bytes, "gbs_whole_step": token_bytes / (ms / a.steps) / 1e6,
                               "moe_this_rank": lb["moe"], "replicated": lb["total"] - lb["moe"]}}
        if world == 1:
            line["roofline_moe_down"] = {"bound": "hbm", "kernel": "moe_down_kernel (8 routed IQ2_XXS + shared Q8_0, accumulated into y)",
                                         "achieved": d_bytes / d_us / 1e3, "peak": peak, "unit": "GB/s",
                                         "frac": d_bytes / d_us / 1e3 / peak, "us_per_launch": d_us, "bytes_per_launch": d_bytes}
        if ep_check is not None:
            line["ep_check"] = ep_check
            line["ep_matches_n1"] = ep_check["ep_matches_n1"]
        if "matvec" in extras:
            # cfg1 and the cfg2 sweep: CUDA-graph replays of 20 launches rotating over a pool of weight copies >= 512 MB
            line["roofline_matvec"] = [dict(m, frac=m["gbs"] / peak, unit="GB/s") for m in extras["matvec"]]
        if "prefill" in extras:
            pf = extras["prefill"]
            line["roofline_prefill"] = {"bound": "tensor", "kernel": "msb_moe_prefill (moep_ts_kernel and moep_gemm_kernel for gate/up and down, gather, combine), cfg4: "
                                        "4096 tokens, top-8 of 384, N(0,1) logits + log-Zipf(1.1) bias", "achieved": pf["tflops"],
                                        "peak": tf_peak, "unit": "TFLOP/s", "frac": pf["tflops"] / tf_peak,
                                        "peak_source": "MEASURED_PEAKS.json bf16_tflops (burst); half operands",
                                        "ms_per_layer": pf["ms"], "flop": pf["flop"], "experts_hit": pf["experts_hit"],
                                        "tokens_per_expert": pf["tokens_per_expert"]}
        if "prefill_ep" in extras:
            line["prefill_ep"] = extras["prefill_ep"]
        if world == 1 and not a.no_cpu_baseline:
            try:
                line["cpu_baseline"] = cpu_baseline_dict(a)
            except Exception as ex:      # the oracle is test infrastructure: never let it break the GPU number
                line["cpu_baseline"] = {"value": None, "unit": UNIT, "error": str(ex)[:200]}
        print(json.dumps(line), flush=True)
    if world > 1:
        # Tear down in dependency order: the captured graphs hold NCCL kernels, so they go before the communicator
        # (destroying the process group while such graphs are alive blocks forever).  Every rank is idle here.
        torch.cuda.synchronize()
        dist.barrier()
        torch.cuda.synchronize()
        del graph, ggraph, hgraph, dgraph
        torch.cuda.synchronize()
        sys.stdout.flush()
        sys.stderr.flush()
        # the communicator itself is released with the process: its destructor waits on a watchdog thread that can
        # outlive the work, and a benchmark that has printed its line must not hang at exit
        os._exit(0)


def main():
    a = parse()
    if a.impl == "reference":
        run_reference(a)
    else:
        run_ours(a)


if __name__ == "__main__":
    main()
