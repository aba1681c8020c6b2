#!/usr/bin/env python
"""Benchmark of the hot path: compressed-KV decode attention, Llama-3.1-8B layer shape,
32-layer sweep at context 32768, batch 8 (one "step" = one decode step of all 32 layers).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--budget 96] [--impl reference]

Prints ONE JSON line (rank 0).  `value` = microseconds per layer-step with the cache
resident in HBM (CUDA-graph replay of the 32 layer-steps); `e2e` = the same through the
public API with the step's queries copied from pinned host memory and the outputs read back
inside the timed region.  Under torchrun every rank owns its own batch rows (units are
independent: no data-path collective), so per-GPU work is fixed ("weak").  The line also carries
two blocks measured in the same run: `splitkv` (one 131072-token sequence cut over the N ranks, the
exchange inside the merge kernel; T(1) on rank 0's GPU alongside) and `encode_c4` (32768 tokens x 8
KV heads of fp32 keys: tier-1 and tier-2 codes from one pass, both page sets assembled from them);
`--no-side` skips both.

`--impl reference` times the CPU restatement of the reference's torch path
(oracle/oracle.py) on a bounded sample of the same workload with all host threads.
"""
from __future__ import annotations

import argparse
import importlib
import json
import os
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

import torch  # noqa: E402

CFG = dict(B=8, Hq=32, Hkv=8, dh=128, ctx=32768, layers=32, page_size=16)
METRIC, UNIT = "decode_attn_us_per_layer_step", "us"
# measured DRAM bytes / algorithmic bytes of the decode kernel (profiles/decode_splitk_ctx16k_ncu.txt)
DRAM_TRAFFIC_RATIO = 1.052


def algorithmic_bytes(lists, tiers, dh: int) -> float:
    """Bytes one layer-step must move: per retained token K-page bytes / N + V (2*dh) +
    position (4), plus 8 bytes of block/bits table per page; queries, outputs and codebooks
    counted once."""
    N = lists.page_size
    tot = 0.0
    cnt = lists.page_count.long()
    for s, t in enumerate(tiers.tiers):
        sel = lists.page_slot == s
        G = dh // t.g
        c = cnt[sel]
        tot += float((8 + 4 * G + (c * G * t.b_theta + 7) // 8 + c * G).sum())
        tot += float(c.sum()) * (2 * dh + 4)
    tot += lists.n_pages * 8
    tot += lists.B * CFG["Hq"] * dh * 2 * 2 + lists.Hkv * sum(dh * (1 << t.b_theta) * 4 for t in tiers.tiers)
    return tot


class ClockSampler(threading.Thread):
    """Samples SM clock and throttle reasons of one GPU with nvidia-smi while running."""

    def __init__(self, index: int):
        super().__init__(daemon=True)
        self.index, self.rows, self._stop_evt = index, [], threading.Event()

    def run(self):
        if self._run_nvml():
            return
        q = ("clocks.sm,clocks.max.sm,clocks_event_reasons.hw_slowdown,"
             "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
             "clocks_event_reasons.sw_power_cap")
        while not self._stop_evt.is_set():
            try:
                out = subprocess.run(["nvidia-smi", f"--query-gpu={q}", "--format=csv,noheader,nounits",
                                      "-i", str(self.index)], capture_output=True, text=True, timeout=5)
                if out.returncode == 0:
                    self.rows.append([x.strip() for x in out.stdout.strip().split(",")])
            except Exception:
                pass
            self._stop_evt.wait(0.1)

    def _run_nvml(self) -> bool:
        """Read-only NVML polling every 20 ms (a nvidia-smi process per sample takes > 100 ms, too
        coarse for a sub-second timed region).  Returns False if NVML is unusable."""
        try:
            import pynvml
            pynvml.nvmlInit()
            # NVML enumerates physical GPUs; honour CUDA_VISIBLE_DEVICES when it lists indices
            vis = os.environ.get("CUDA_VISIBLE_DEVICES", "")
            ids = [v for v in vis.split(",") if v.strip().isdigit()]
            phys = int(ids[self.index]) if self.index < len(ids) else self.index
            h = pynvml.nvmlDeviceGetHandleByIndex(phys)
            mx = pynvml.nvmlDeviceGetMaxClockInfo(h, pynvml.NVML_CLOCK_SM)
            bits = [("hw_slowdown", pynvml.nvmlClocksEventReasonHwSlowdown),
                    ("hw_thermal_slowdown", pynvml.nvmlClocksEventReasonHwThermalSlowdown),
                    ("sw_thermal_slowdown", pynvml.nvmlClocksEventReasonSwThermalSlowdown),
                    ("sw_power_cap", pynvml.nvmlClocksEventReasonSwPowerCap)]
            get_reasons = getattr(pynvml, "nvmlDeviceGetCurrentClocksEventReasons", None) or \
                pynvml.nvmlDeviceGetCurrentClocksThrottleReasons
            get_reasons(h)
        except Exception:
            return False
        while not self._stop_evt.is_set():
            try:
                sm = pynvml.nvmlDeviceGetClockInfo(h, pynvml.NVML_CLOCK_SM)
                r = get_reasons(h)
                self.rows.append([str(sm), str(mx)] + ["Active" if r & b else "Not Active" for _, b in bits])
            except Exception:
                pass
            self._stop_evt.wait(0.02)
        return True

    def stop(self) -> dict:
        self._stop_evt.set()
        self.join(timeout=6)
        sm = sorted(int(r[0]) for r in self.rows if r and r[0].isdigit())
        mx = [int(r[1]) for r in self.rows if len(r) > 1 and r[1].isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = [n for i, n in enumerate(names)
                   if any(len(r) > 2 + i and r[2 + i].lower().startswith("active") for r in self.rows)]
        return {"sm_mhz": sm[len(sm) // 2] if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(sm)}


class CpuReference:
    """The oracle's restatement of the reference torch decode path
    (_compressed_head_attention_batched) on `n_units` (batch row, KV head) units of the
    benchmark workload, all host threads."""

    def __init__(self, budget: float, n_units: int, threads: int):
        sys.path.insert(0, os.path.join(ROOT, "oracle"))
        import oracle as orc
        pkg = importlib.import_module("spherical-kv_b200")
        torch.set_num_threads(threads)
        self.orc, self.n_units, self.threads = orc, n_units, threads
        dh, ctx, Hq, Hkv = CFG["dh"], CFG["ctx"], CFG["Hq"], CFG["Hkv"]
        self.grp = Hq // Hkv
        specs = pkg.REFERENCE_TIERS[:2]
        fr = pkg.synth.budget_fractions(budget)
        K, V, self.Q, _ = pkg.synth.make_kvq(1, self.grp * n_units, n_units, dh, ctx, seed=0)
        cbs = pkg.synth.make_codebooks(n_units, dh, specs, seed=1)
        assign = pkg.synth.make_tier_assign(1, n_units, ctx, fr, seed=2)
        self.cos, self.sin = orc.rope_tables(ctx + 8, dh)
        self.units = []
        for h in range(n_units):
            tl = []
            for s, t in enumerate(specs):
                pos = torch.nonzero(assign[0, h] == t.tier_id).flatten()
                if pos.numel() == 0:
                    continue
                r, th = orc.encode(K[0, pos, h].contiguous(), cbs[s][h])
                tl.append(dict(r=torch.from_numpy(r), theta=torch.from_numpy(th), positions=pos,
                               V=V[0, pos, h].half().float(), cb=cbs[s][h]))
            self.units.append(tl)
        self.total_units = CFG["B"] * Hkv
        self.desc = (f"{n_units} of {self.total_units} (batch row, KV head) units at ctx {ctx} per step, "
                     f"scaled linearly to the full layer-step")
        self.K, self.V, self.cbs, self.assign, self.specs = K, V, cbs, assign, specs
        self.last_out = None

    def gpu_same_input_diff(self, dev) -> float:
        """The units this arm evaluates, decoded by the CUDA path from the same seeded keys, values,
        queries and codebooks (uploaded bits): max-abs difference of the attention outputs."""
        pkg = importlib.import_module("spherical-kv_b200")
        dh, ctx = CFG["dh"], CFG["ctx"]
        tiers = pkg.TierSet(dh, self.specs)
        lists = pkg.build_page_lists(self.assign.to(dev), tiers, CFG["page_size"], shuffle_seed=0)
        cache = pkg.encode_pages(self.K[0].to(dev), self.V[0].to(dev), lists,
                                 tiers.pack_codebooks(self.cbs).to(dev), tiers)
        rope = pkg.rope_table(ctx + 8, dh, device=dev)
        out = pkg.decode_paged(self.Q.to(dev), cache, rope).float().cpu()[0]
        if self.last_out is None:
            self.step_us()
        return float((out - self.last_out).abs().max())

    def step_us(self) -> float:
        """One pass over the sample; microseconds per full layer-step (scaled)."""
        t0 = time.perf_counter()
        outs = []
        for h, tl in enumerate(self.units):
            outs.append(self.orc.decode_unit(self.Q[0, h * self.grp:(h + 1) * self.grp], tl, self.cos, self.sin,
                                             torch.float32)[1])
        dt = time.perf_counter() - t0
        self.last_out = torch.cat(outs, 0)
        return dt / self.n_units * self.total_units * 1e6


def run_reference(args) -> None:
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    threads = os.cpu_count() or 1
    ref = CpuReference(args.budget, n_units=2, threads=threads)
    for _ in range(max(1, args.warmup)):
        ref.step_us()
    steps = max(1, args.steps)
    t0 = time.perf_counter()
    vals = [ref.step_us() for _ in range(steps)]
    v = sum(vals) / len(vals)
    line = {"impl": "reference", "metric": METRIC, "value": v, "unit": UNIT, "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": v * CFG["layers"] / 1e3,
            "higher_is_better": False, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic", "config": workload_config(args),
            "cpu_baseline": {"value": v, "unit": UNIT, "cores": threads, "kind": "port",
                             "sample": ref.desc},
            "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def workload_config(args) -> dict:
    return {"workload": f"Llama-3.1-8B decode attention, 32-layer sweep, ctx {CFG['ctx']}, batch "
                        f"{CFG['B']} per GPU, K budget {args.budget:g} bits/token-head, 16-token pages, "
                        f"bf16 Q/V/out, int8 radii",
            "B_per_gpu": CFG["B"], "Hq": CFG["Hq"], "Hkv": CFG["Hkv"], "dh": CFG["dh"], "ctx": CFG["ctx"],
            "layers": CFG["layers"], "page_size": CFG["page_size"], "budget_bits": args.budget,
            "l2_policy": "32 distinct layer caches (>= 8 GB) cycled per step: inputs larger than L2",
            "sharding": "batch rows per GPU, no collective",
            "page_importance_ema": bool(getattr(args, "ema", False))}


def run_side_workload(args) -> None:
    """Secondary measurements (not the headline line): split-KV decode of one long sequence
    over the ranks and encode / page-build throughput (config 4)."""
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl", device_id=dev)
    pkg = importlib.import_module("spherical-kv_b200")
    Hq, Hkv, dh, N = CFG["Hq"], CFG["Hkv"], CFG["dh"], CFG["page_size"]
    specs = pkg.REFERENCE_TIERS[:2]
    tiers = pkg.TierSet(dh, specs)
    gen = torch.Generator(device=dev).manual_seed(77)
    scale = torch.exp(0.5 * torch.randn(dh, generator=gen, device=dev))

    def ev_time(fn, steps):
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier(); torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(steps):
            fn()
        e1.record()
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1)
        if world > 1:
            t = torch.tensor([ms], device=dev)
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            ms = float(t.item())
        return ms / steps

    if args.workload == "splitkv":
        ctx = 131072 if args.ctx == 32768 else args.ctx
        n_seq = 8  # distinct sequences cycled so that a step never finds its pages in L2
        rope = pkg.rope_table(ctx + 8, dh, device=dev)
        decs, qs = [], []
        for i in range(n_seq):
            assign = pkg.synth.make_tier_assign(1, Hkv, ctx, {1: 0.2, 2: 0.6}, seed=500 + i).to(dev)
            lists = pkg.build_page_lists(assign, tiers, N, shuffle_seed=i)
            K = (torch.randn(ctx, Hkv, dh, generator=gen, device=dev) * scale).bfloat16()
            V = (torch.randn(ctx, Hkv, dh, generator=gen, device=dev) * scale).bfloat16()
            cb = tiers.pack_codebooks([c.to(dev) for c in pkg.synth.make_codebooks(Hkv, dh, specs, seed=i)])
            cache = pkg.encode_pages(K, V, lists, cb, tiers, v_dtype=torch.bfloat16)
            decs.append(pkg.split_kv.SplitKVDecoder(pkg.split_kv.shard_cache(cache, rank, world), 1, Hq,
                                                    out_dtype=torch.bfloat16))
            qs.append((torch.randn(1, Hq, dh, generator=gen, device=dev) * scale).bfloat16())
            if i == 0:
                alg = algorithmic_bytes(lists, tiers, dh) - 1 * Hq * dh * 4 + Hq * dh * 4
        def step():
            for d, q in zip(decs, qs):
                d.decode(q, rope)
        for _ in range(args.warmup):
            step()
        # one CUDA graph for the whole step (decode kernels, all-gathers, merges): the exchange is
        # latency-bound, so launch gaps matter; fall back to plain launches if capture is refused
        graphed = False
        try:
            if world > 1:
                # ranks must issue identical collective sequences; a capture that fails on one
                # rank only would leave the others waiting, so multi-rank runs use plain launches
                raise RuntimeError("multi-rank: plain launches")
            side = torch.cuda.Stream(device=dev)
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                step()
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=side):
                    step()
            torch.cuda.current_stream().wait_stream(side)
            torch.cuda.synchronize()
            run = g.replay
            graphed = True
        except Exception as exc:  # noqa: BLE001
            run = step
        for _ in range(args.warmup):
            run()
        ms = ev_time(run, args.steps) / n_seq
        if rank == 0:
            print(json.dumps({"metric": "splitkv_decode_us_per_step", "value": ms * 1e3, "unit": "us",
                              "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
                              "higher_is_better": False, "scaling": "strong", "data": "synthetic",
                              "config": {"workload": f"split-KV decode, B1 Hq32 Hkv8 dh128 ctx {ctx}, 20/60/20, "
                                                     f"pages sharded contiguously over {world} GPU(s), all-gather + "
                                                     f"log-sum-exp merge; {n_seq} sequences cycled (L2)"},
                              "cuda_graph": graphed, "algorithmic_bytes_total": alg,
                              "achieved_hbm_gbs_all_gpus": alg / (ms * 1e-3) / 1e9}), flush=True)
    elif args.workload == "encode":
        ctx, layers = args.ctx, min(args.layers, 8)
        assign1 = torch.full((1, Hkv, ctx), 1, dtype=torch.uint8, device=dev)
        assign2 = torch.full((1, Hkv, ctx), 2, dtype=torch.uint8, device=dev)
        l1 = pkg.build_page_lists(assign1, tiers, N)
        l2 = pkg.build_page_lists(assign2, tiers, N)
        Ks = [(torch.randn(ctx, Hkv, dh, generator=gen, device=dev) * scale) for _ in range(layers)]
        for Kt in Ks:   # 1 % of the channels are x20 outliers
            Kt[..., torch.randperm(dh, generator=torch.Generator().manual_seed(3))[:max(1, dh // 100)].to(dev)] *= 20
        cb = tiers.pack_codebooks([c.to(dev) for c in pkg.synth.make_codebooks(Hkv, dh, specs, seed=9)])
        c1 = pkg.encode_pages(Ks[0], Ks[0], l1, cb, tiers, v_dtype=torch.bfloat16)
        c2 = pkg.encode_pages(Ks[0], None, l2, cb, tiers, v_dtype=torch.bfloat16)
        def step():
            for Kt in Ks:   # every token-head is matched against both codebooks (64 + 16 centroids)
                pkg.encode_pages(Kt, Kt, l1, cb, tiers, out=c1)
                pkg.encode_pages(Kt, None, l2, cb, tiers, out=c2)
        for _ in range(args.warmup):
            step()
        ms = ev_time(step, args.steps)
        th = layers * ctx * Hkv
        rd = th * dh * 4 * 3          # K read twice (once per tier), V once, fp32
        wr = layers * (l1.pool_bytes + l2.pool_bytes + l1.n_pages * N * dh * 2)
        if rank == 0:
            print(json.dumps({"metric": "encode_token_heads_per_s", "value": th / (ms * 1e-3), "unit": "token-heads/s",
                              "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms,
                              "higher_is_better": True, "data": "synthetic",
                              "config": {"workload": f"spherical encode + page build, {ctx} tokens x {layers} layers x "
                                                     f"{Hkv} KV heads x dh {dh}, fp32 K with 1% x20 outlier channels, "
                                                     f"tier-1 (C=64) and tier-2 (C=16) pages for every token"},
                              "gmac_per_s": th * (dh // 16) * 16 * 80 / (ms * 1e-3) / 1e9,
                              "hbm_gbs": (rd + wr) / (ms * 1e-3) / 1e9}), flush=True)
    elif args.workload == "recode":
        # all-tier code cache in one pass over K, then re-paging from it, against the per-tier route
        ctx, layers = args.ctx, min(args.layers, 4)
        specs3 = pkg.REFERENCE_TIERS
        tiers3 = pkg.TierSet(dh, specs3)
        cb3 = tiers3.pack_codebooks([c.to(dev) for c in pkg.synth.make_codebooks(Hkv, dh, specs3, seed=9)])
        Ks = [(torch.randn(ctx, Hkv, dh, generator=gen, device=dev) * scale) for _ in range(layers)]
        Vs = [k.bfloat16() for k in Ks]
        per_tier = [pkg.build_page_lists(torch.full((1, Hkv, ctx), t.tier_id, dtype=torch.uint8, device=dev),
                                         tiers3, N) for t in specs3]
        mixed = pkg.build_page_lists(pkg.synth.make_tier_assign(1, Hkv, ctx, {1: 0.2, 2: 0.5, 3: 0.3}, seed=1,
                                                                per_head=True).to(dev), tiers3, N)
        codes = pkg.encode_codes(Ks[0], cb3, tiers3)
        outs = [pkg.encode_pages(Ks[0], None, l, cb3, tiers3) for l in per_tier]
        direct = pkg.encode_pages(Ks[0], Vs[0], mixed, cb3, tiers3, v_dtype=torch.bfloat16)
        again = pkg.pages_from_codes(codes, Vs[0], mixed, cb3, v_dtype=torch.bfloat16)
        same = bool(torch.equal(direct.k_pages, again.k_pages) and torch.equal(direct.v_pool, again.v_pool))

        def one_pass():
            for Kt in Ks:
                pkg.encode_codes(Kt, cb3, tiers3)

        def three_passes():
            for Kt in Ks:
                for l, o in zip(per_tier, outs):
                    pkg.encode_pages(Kt, None, l, cb3, tiers3, out=o)

        def repage():
            for Vt in Vs:
                pkg.pages_from_codes(codes, Vt, mixed, cb3, out=again)

        def reencode():
            for Kt, Vt in zip(Ks, Vs):
                pkg.encode_pages(Kt, Vt, mixed, cb3, tiers3, out=direct)

        res = {}
        for name, fn in (("codes_one_pass", one_pass), ("encode_three_tiers", three_passes),
                         ("repage_from_codes", repage), ("reencode_from_keys", reencode)):
            for _ in range(args.warmup):
                fn()
            res[name] = ev_time(fn, args.steps)
        th = layers * ctx * Hkv
        if rank == 0:
            print(json.dumps({"metric": "all_tier_codes_token_heads_per_s", "value": th / (res["codes_one_pass"] * 1e-3),
                              "unit": "token-heads/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
                              "ms_per_step": res["codes_one_pass"], "higher_is_better": True, "data": "synthetic",
                              "config": {"workload": f"codes of tiers 1/2/3 for {ctx} tokens x {layers} layers x {Hkv} KV "
                                                     f"heads x dh {dh} in one pass over fp32 K; re-paging a 20/50/30 "
                                                     f"tier mix from the cache ({N}-token pages, bf16 V)"},
                              "ms": res, "speedup_vs_three_encodes": res["encode_three_tiers"] / res["codes_one_pass"],
                              "repage_speedup_vs_reencode": res["reencode_from_keys"] / res["repage_from_codes"],
                              "repage_bytes_identical": same,
                              "gmac_per_s": th * dh * (64 + 16 + 8) / (res["codes_one_pass"] * 1e-3) / 1e9}), flush=True)
    elif args.workload == "kmeans":
        import torch.nn.functional as F
        res = []
        for Np, d, K in ((4_000_000, 16, 64), (4_000_000, 16, 16), (2_000_000, 32, 8)):
            U = F.normalize(torch.randn(Np, d, generator=gen, device=dev), dim=1)
            Cn = F.normalize(torch.randn(K, d, generator=gen, device=dev), dim=1)

            def torch_step():
                sims = U @ Cn.T
                a_ = sims.argmax(1)
                torch.zeros_like(Cn).index_add_(0, a_, U)
                torch.bincount(a_, minlength=K)

            for _ in range(args.warmup):
                pkg.kmeans_assign(U, Cn, want_sim=False); torch_step()
            t_k = ev_time(lambda: pkg.kmeans_assign(U, Cn, want_sim=False), args.steps)
            t_t = ev_time(torch_step, args.steps)
            res.append({"N": Np, "d": d, "K": K, "kernel_us": t_k * 1e3, "torch_ops_us": t_t * 1e3,
                        "points_per_s": Np / (t_k * 1e-3), "tmac_per_s": Np * K * d / (t_k * 1e-3) / 1e12,
                        "read_gbs": Np * d * 4 / (t_k * 1e-3) / 1e9})
        if rank == 0:
            print(json.dumps({"metric": "kmeans_assign_points_per_s", "value": res[0]["points_per_s"], "unit": "points/s",
                              "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "higher_is_better": True,
                              "data": "synthetic",
                              "config": {"workload": "spherical k-means assignment + accumulation step (codebook "
                                                     "training inner loop) on random unit vectors; torch_ops = the "
                                                     "same step as matmul + argmax + index_add_ + bincount"},
                              "cases": res}), flush=True)
    else:  # pool: device-resident LayerPool
        import time as _time
        sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "spherical-kv_b200", "dropin"))
        import sphkv_lut
        from types import SimpleNamespace
        ctx, Np = min(args.ctx, 32768), 16
        tobj = [SimpleNamespace(tier_id=0, g=dh, G=1, b_theta=0)] + [
            SimpleNamespace(tier_id=t.tier_id, g=t.g, G=dh // t.g, b_theta=t.b_theta) for t in pkg.REFERENCE_TIERS]
        idx_map = sphkv_lut.make_tier_idx_map(tobj)
        cpu_gen = torch.Generator().manual_seed(5)
        per_head, cbs = {}, {}
        for h in range(Hkv):
            ent = []
            for t, n in ((tobj[1], ctx // 4), (tobj[2], ctx // 2), (tobj[3], ctx // 4)):
                ent.append((None, None, t.b_theta, n, torch.randn(n, dh, generator=cpu_gen).half().to(dev),
                            (torch.rand(n, t.G, generator=cpu_gen).to(dev) * 3,
                             torch.randint(0, 2 ** t.b_theta, (n, t.G), generator=cpu_gen).to(dev))))
            per_head[(0, h)] = ent
            for t in tobj[1:]:
                c = torch.randn(t.G, 2 ** t.b_theta, t.g, generator=cpu_gen)
                cbs[(0, h, t.tier_id)] = c / c.norm(dim=-1, keepdim=True)
        pipe = SimpleNamespace(per_head_pages=per_head, codebooks=cbs)
        cap = 64 * Hkv
        torch.cuda.synchronize()
        t0 = _time.perf_counter()
        pool = sphkv_lut.LayerPool(pipe, 0, Np, 8, 64, cap, dev, tobj, idx_map, Hq, Hkv, Hq // Hkv, dh)
        torch.cuda.synchronize()
        build_ms = (_time.perf_counter() - t0) * 1e3
        q = torch.randn(Hq, dh, device=dev); k = torch.randn(Hkv, dh, device=dev); v = torch.randn(Hkv, dh, device=dev)
        sm = dh ** -0.5
        pool.append_and_compute(q, k, v, tobj, sm)
        torch.cuda.synchronize()
        side = torch.cuda.Stream(device=dev)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.stream(side):
            with torch.cuda.graph(g, stream=side):
                pool.append_and_compute(q, k, v, tobj, sm)
        torch.cuda.synchronize()
        n_steps = min(200, (cap // Hkv - 2) * Np // 2)
        graph_us = ev_time(g.replay, n_steps) * 1e3
        plain_us = ev_time(lambda: pool.append_and_compute(q, k, v, tobj, sm), n_steps) * 1e3
        pool.check_overflow()
        # same-box GPU comparison: the reference's own CUDA kernels (compiled from the reference tree
        # into oracle/_ref/ by oracle/build_ref.py) on the same data at 128-token pages, the only
        # page size their launch geometry supports; skipped when the module is not there
        ref_cmp = None
        sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "oracle"))
        import build_ref
        ref_mod = build_ref.load_module()
        if ref_mod is not None:
            pool128 = sphkv_lut.LayerPool(pipe, 0, 128, 8, 64, 8 * Hkv, dev, tobj, idx_map, Hq, Hkv, Hq // Hkv, dh)
            out_r = torch.zeros(Hq, dh, device=dev)
            part_r = torch.zeros(Hq, pool128.max_blocks, dh + 2, device=dev)
            dargs = (q, pool128.cb_flat, pool128.tier_G_gpu, pool128.tier_g_gpu, pool128.theta_codes,
                     pool128.radius_codes, pool128.r_scales, pool128.v_pool, pool128.block_table_gpu,
                     pool128.bits_table_gpu, pool128.ctx_lens_gpu)
            tail = (Hq, Hkv, Hq // Hkv, len(idx_map), pool128.max_blocks, 128, dh, 8, 64, pool128.g_max, sm, ctx)
            import fused_decode as ours
            ref_fn = lambda: ref_mod.forward(*dargs, out_r, part_r, *tail)  # noqa: E731
            our_fn = lambda: ours.sphkv_decode(*dargs, pool128._out_buf, pool128._partial_scratch, *tail)  # noqa: E731
            for _ in range(3):
                ref_fn(); our_fn()
            torch.cuda.synchronize()
            diff = float((out_r - pool128._out_buf).abs().max().item())
            ref_cmp = {"page_size": 128, "reference_cuda_decode_us": ev_time(ref_fn, 50) * 1e3,
                       "this_library_decode_us": ev_time(our_fn, 50) * 1e3, "max_abs_diff": diff}
        if rank == 0:
            print(json.dumps({"metric": "layerpool_step_us", "value": graph_us, "unit": "us", "n_gpus": world,
                              "steps": n_steps, "warmup": 1, "higher_is_better": False, "data": "synthetic",
                              "config": {"workload": f"LayerPool decode step (append with on-device page roll-over + "
                                                     f"pool decode), 1 sequence, Hq{Hq} Hkv{Hkv} dh{dh}, ctx {ctx}, "
                                                     f"{Np}-token pages, tiers 25/50/25; replayed from one CUDA graph"},
                              "plain_launch_us": plain_us, "pool_pages": int(pool.num_pages_used),
                              "bulk_construction_ms": build_ms,
                              "same_box_reference_kernel": ref_cmp}), flush=True)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()



def _graph_time(fn, steps, warmup, dev, world):
    """Records `fn` into a CUDA graph on a side stream, replays it `steps` times between events;
    milliseconds per replay, max over ranks."""
    import torch.distributed as dist
    st = torch.cuda.Stream(device=dev)
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        fn(); fn()
        st.synchronize()
        if world > 1:
            dist.barrier()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            fn()
        for _ in range(warmup):
            g.replay()
        st.synchronize()
        if world > 1:
            dist.barrier()
            torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(st)
        for _ in range(steps):
            g.replay()
        e1.record(st)
        st.synchronize()
        ms = e0.elapsed_time(e1) / steps
    torch.cuda.current_stream().wait_stream(st)
    if world > 1:
        t = torch.tensor([ms], device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = float(t.item())
    return ms


def splitkv_block(args, pkg, dev, rank, world):
    """BASELINE config 5 on the ranks of this run: one 131072-token sequence (batch 1, 20/60/20),
    its pages cut contiguously over the GPUs, partial (max, sum, acc) rows exchanged by peer stores
    inside the merge kernel.  T1 is measured in the same run (every rank decodes the whole sequence
    alone, same launch mode), so the efficiency T1 / (n * Tn) compares like with like."""
    Hq, Hkv, dh, N = CFG["Hq"], CFG["Hkv"], CFG["dh"], CFG["page_size"]
    ctx, n_seq = 131072, 4   # distinct sequences cycled: a step never finds its pages in L2
    specs = pkg.REFERENCE_TIERS[:2]
    tiers = pkg.TierSet(dh, specs)
    gen = torch.Generator(device=dev).manual_seed(4242)   # the same sequences on every rank
    scale = torch.exp(0.5 * torch.randn(dh, generator=gen, device=dev))
    rope = pkg.rope_table(ctx + 8, dh, device=dev)
    fulls, shards, qs, alg = [], [], [], None
    for i in range(n_seq):
        assign = pkg.synth.make_tier_assign(1, Hkv, ctx, {1: 0.2, 2: 0.6}, seed=500 + i).to(dev)
        lists = pkg.build_page_lists(assign, tiers, N, shuffle_seed=i)
        K = (torch.randn(ctx, Hkv, dh, generator=gen, device=dev) * scale).bfloat16()
        V = (torch.randn(ctx, Hkv, dh, generator=gen, device=dev) * scale).bfloat16()
        cb = tiers.pack_codebooks([c.to(dev) for c in pkg.synth.make_codebooks(Hkv, dh, specs, seed=i)])
        cache = pkg.encode_pages(K, V, lists, cb, tiers, v_dtype=torch.bfloat16)
        fulls.append(cache)
        shards.append(pkg.split_kv.shard_cache(cache, rank, world))
        qs.append((torch.randn(1, Hq, dh, generator=gen, device=dev) * scale).bfloat16())
        if alg is None:
            alg = algorithmic_bytes(lists, tiers, dh) - CFG["B"] * Hq * dh * 4 + Hq * dh * 4
        del K, V
    out_full = [torch.empty(1, Hq, dh, dtype=torch.bfloat16, device=dev) for _ in range(n_seq)]
    out_split = [torch.empty(1, Hq, dh, dtype=torch.bfloat16, device=dev) for _ in range(n_seq)]

    def full_step():
        for c, q, o in zip(fulls, qs, out_full):
            pkg.decode_paged(q, c, rope, out=o)

    t1_us = _graph_time(full_step, args.steps, args.warmup, dev, world) * 1e3 / n_seq
    blk = {"workload": f"split-KV decode, B1 Hq{Hq} Hkv{Hkv} dh{dh} ctx {ctx}, 20/60/20, pages cut contiguously "
                       f"over {world} GPU(s); {n_seq} sequences cycled (inputs larger than L2); CUDA-graph replay",
           "n_gpus": world, "t1_us_per_step": t1_us, "algorithmic_bytes": alg,
           "t1_hbm_gbs": alg / (t1_us * 1e-6) / 1e9}
    if world == 1:
        blk.update({"us_per_step": t1_us, "efficiency": 1.0, "exchange": "none (one GPU)"})
        return blk
    try:
        ex = pkg.split_kv.PeerExchange(1, Hq, Hkv, dh, device=dev)
    except Exception as exc:  # noqa: BLE001  (raised on every rank alike: see PeerExchange)
        blk["error"] = f"peer exchange unavailable: {exc}"
        return blk

    def split_step():
        for c, q, o in zip(shards, qs, out_split):
            pkg.decode_paged(q, c, rope, out=o, exchange=ex)

    tn_us = _graph_time(split_step, args.steps, args.warmup, dev, world) * 1e3 / n_seq
    # the same shards decoded without the exchange (partial rows only): what a rank spends on its own
    parts = [torch.empty(1, Hq, dh + 2, device=dev) for _ in range(n_seq)]

    def local_step():
        for c, q, pt in zip(shards, qs, parts):
            pkg.decode_paged(q, c, rope, out_partial=pt, want_out=False)

    local_us = _graph_time(local_step, args.steps, args.warmup, dev, world) * 1e3 / n_seq
    torch.cuda.synchronize()
    diff = max(float((a.float() - b.float()).abs().max()) for a, b in zip(out_split, out_full))
    status = sum(int(c.status.item()) for c in shards)
    st = torch.tensor([diff, float(status)], device=dev)
    import torch.distributed as dist
    dist.all_reduce(st, op=dist.ReduceOp.MAX)
    blk.update({"us_per_step": tn_us, "efficiency": t1_us / (world * tn_us),
                "local_us_per_step": local_us, "exchange_us_per_step": tn_us - local_us,
                "exchange": "peer stores of 64-bit (step, value) words + bounded wait inside the merge kernel "
                            "(no fence, flag or collective)",
                "bytes_sent_per_rank_per_step": (world - 1) * Hq * (dh + 2) * 8,
                "merged_vs_single_pass_max_abs": float(st[0].item()), "kernel_status": int(st[1].item()),
                "achieved_hbm_gbs_all_gpus": alg / (tn_us * 1e-6) / 1e9})
    ex.close()
    return blk


def encode_c4_block(args, pkg, dev):
    """BASELINE config 4 shape, a few layers at a time: 32768 tokens x 8 KV heads x dh 128 of fp32
    keys with 1 % of the channels scaled by 20; every token-head gets its tier-1 and its tier-2 codes
    from ONE pass over the keys, then both sets of bit-packed pages are assembled from the codes."""
    Hkv, dh, N, ctx, layers = CFG["Hkv"], CFG["dh"], CFG["page_size"], 32768, 4
    specs = pkg.REFERENCE_TIERS[:2]
    tiers = pkg.TierSet(dh, specs)
    gen = torch.Generator(device=dev).manual_seed(99)
    scale = torch.exp(0.5 * torch.randn(dh, generator=gen, device=dev))
    scale[torch.randperm(dh, generator=torch.Generator().manual_seed(3))[:max(1, dh // 100)].to(dev)] *= 20
    Ks = [torch.randn(ctx, Hkv, dh, generator=gen, device=dev) * scale for _ in range(layers)]
    cb = tiers.pack_codebooks([c.to(dev) for c in pkg.synth.make_codebooks(Hkv, dh, specs, seed=9)])
    l1 = pkg.build_page_lists(torch.full((1, Hkv, ctx), 1, dtype=torch.uint8, device=dev), tiers, N)
    l2 = pkg.build_page_lists(torch.full((1, Hkv, ctx), 2, dtype=torch.uint8, device=dev), tiers, N)
    codes = pkg.encode_codes(Ks[0], cb, tiers)
    c1 = pkg.pages_from_codes(codes, None, l1, cb)
    c2 = pkg.pages_from_codes(codes, None, l2, cb)
    # bit-exactness of this route at this shape: the pages equal a direct encode of the keys
    d1 = pkg.encode_pages(Ks[0], None, l1, cb, tiers)
    d2 = pkg.encode_pages(Ks[0], None, l2, cb, tiers)
    same = bool(torch.equal(c1.k_pages, d1.k_pages) and torch.equal(c2.k_pages, d2.k_pages))

    def step():
        for Kt in Ks:
            cd = pkg.encode_codes(Kt, cb, tiers)
            pkg.pages_from_codes(cd, None, l1, cb, out=c1)
            pkg.pages_from_codes(cd, None, l2, cb, out=c2)

    for _ in range(max(3, args.warmup)):
        step()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    reps = max(3, min(args.steps, 10))
    e0.record()
    for _ in range(reps):
        step()
    e1.record()
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / reps
    th = layers * ctx * Hkv
    macs = th * dh * (64 + 16)
    rd = th * dh * 4
    wr = layers * (l1.pool_bytes + l2.pool_bytes)
    return {"workload": f"{ctx} tokens x {layers} layers x {Hkv} KV heads x dh {dh}, fp32 keys with 1% x20 outlier "
                        f"channels; tier-1 (64 centroids) and tier-2 (16) codes in one pass over the keys, both page sets "
                        f"assembled from the codes ({N}-token pages)",
            "ms_per_32_layers": ms / layers * 32, "token_heads_per_s": th / (ms * 1e-3),
            "tmac_per_s": macs / (ms * 1e-3) / 1e12,
            "hbm_gbs": (rd + wr) / (ms * 1e-3) / 1e9, "pages_identical_to_direct_encode": same}


def main() -> None:
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--budget", type=float, default=96.0, help="average K bits per token-head")
    ap.add_argument("--impl", default="b200", choices=["b200", "reference"])
    ap.add_argument("--layers", type=int, default=CFG["layers"])
    ap.add_argument("--ctx", type=int, default=CFG["ctx"])
    ap.add_argument("--batch", type=int, default=CFG["B"], help="batch rows per GPU")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-side", action="store_true", help="skip the split-KV and encode blocks of the line")
    ap.add_argument("--ema", action="store_true",
                    help="also update the page-importance EMA in the decode epilogue (per-tile statistics + "
                         "omega blend inside the merge kernel); off for the headline line")
    ap.add_argument("--workload", default="decode", choices=["decode", "splitkv", "encode", "recode", "kmeans", "pool"],
                    help="decode: the headline line (default); splitkv: one 131072-token sequence "
                         "split over the ranks; encode: prefill compression throughput")
    args = ap.parse_args()
    CFG["layers"], CFG["ctx"], CFG["B"] = args.layers, args.ctx, args.batch
    if args.impl == "reference":
        run_reference(args)
        return
    args.warmup = max(args.warmup, 3)
    if args.workload != "decode":
        run_side_workload(args)
        return

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl", device_id=dev)

    pkg = importlib.import_module("spherical-kv_b200")
    B, Hq, Hkv, dh, ctx, NL, N = (CFG[k] for k in ("B", "Hq", "Hkv", "dh", "ctx", "layers", "page_size"))
    specs = pkg.REFERENCE_TIERS[:2]
    tiers = pkg.TierSet(dh, specs)
    fr = pkg.synth.budget_fractions(args.budget)
    rope = pkg.rope_table(ctx + 8, dh, device=dev)

    # ---- build the 32 layer caches with the encode kernel (seeded, generated on the GPU) ----
    gen = torch.Generator(device=dev).manual_seed(1234 + rank)
    scale = torch.exp(0.5 * torch.randn(dh, generator=gen, device=dev))
    caches, enc_ms, alg_bytes, tok_heads = [], [], None, None
    for layer in range(NL):
        assign = pkg.synth.make_tier_assign(B, Hkv, ctx, fr, seed=100 + layer).to(dev)
        lists = pkg.build_page_lists(assign, tiers, N, shuffle_seed=layer)
        K = (torch.randn(B * ctx, Hkv, dh, generator=gen, device=dev) * scale).bfloat16()
        V = (torch.randn(B * ctx, Hkv, dh, generator=gen, device=dev) * scale).bfloat16()
        cb = tiers.pack_codebooks([c.to(dev) for c in pkg.synth.make_codebooks(Hkv, dh, specs, seed=layer)])
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        cache = pkg.encode_pages(K, V, lists, cb, tiers, v_dtype=torch.bfloat16)
        e1.record()
        torch.cuda.synchronize()
        enc_ms.append(e0.elapsed_time(e1))
        if alg_bytes is None:
            alg_bytes = algorithmic_bytes(lists, tiers, dh)
            tok_heads = int(lists.page_count.sum().item())
        cache.scratch = pkg.decode_scratch(cache)
        caches.append(cache)
        del K, V, assign

    q_host = (torch.randn(NL, B, Hq, dh) * scale.cpu()).bfloat16().pin_memory()
    q_dev = q_host.to(dev)
    out_dev = torch.empty(NL, B, Hq, dh, dtype=torch.bfloat16, device=dev)
    out_host = torch.empty(NL, B, Hq, dh, dtype=torch.bfloat16).pin_memory()

    # size-independent self-check at full size: the result must not depend on how the blocks are
    # split over CTAs (148 vs 37 vs 5 CTAs walk very different tile sequences per warp)
    ref_out = pkg.decode_paged(q_dev[0], caches[0], rope).float()
    self_check = 0.0
    for n_alt in (37, 5):
        alt = pkg.PagedCache(tiers=caches[0].tiers, lists=caches[0].lists, codebooks=caches[0].codebooks,
                             k_pages=caches[0].k_pages, v_pool=caches[0].v_pool, radius_fmt=caches[0].radius_fmt)
        alt_out = pkg.decode_paged(q_dev[0], alt, rope, n_ctas=n_alt).float()
        self_check = max(self_check, float((alt_out - ref_out).abs().max().item()))
    torch.cuda.synchronize()

    if args.ema:
        tile_ml = [torch.empty(B, Hq, c.lists.max_blocks, N // 16, 2, device=dev) for c in caches]
        omegas = [torch.ones(B * Hkv, c.lists.max_blocks, device=dev) for c in caches]

    def sweep():
        for layer in range(NL):
            if args.ema:
                pkg.decode_paged(q_dev[layer], caches[layer], rope, out=out_dev[layer], page_ml=tile_ml[layer],
                                 omega=omegas[layer], ema_beta=0.9)
            else:
                pkg.decode_paged(q_dev[layer], caches[layer], rope, out=out_dev[layer])

    stream = torch.cuda.Stream(device=dev)
    with torch.cuda.stream(stream):
        sweep()
        sweep()
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            sweep()
        for _ in range(args.warmup):
            graph.replay()
        stream.synchronize()

        def barrier():
            torch.cuda.synchronize()
            if world > 1:
                dist.barrier()
                torch.cuda.synchronize()

        def timed(fn, steps):
            barrier()
            sampler = ClockSampler(local)
            sampler.start()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            for _ in range(steps):
                fn()
            e1.record(stream)
            barrier()
            ms = e0.elapsed_time(e1)
            clocks = sampler.stop()
            if world > 1:
                t = torch.tensor([ms], device=dev)
                dist.all_reduce(t, op=dist.ReduceOp.MAX)
                ms = float(t.item())
            return ms, clocks

        # device-resident: the graph of 32 layer-steps.  Clock samples need some wall time, so
        # run at least ~0.5 s worth of steps but report exactly `steps`.
        ms, clocks = timed(graph.replay, args.steps)

        def e2e_step():
            q_dev.copy_(q_host, non_blocking=True)
            sweep()
            out_host.copy_(out_dev, non_blocking=True)

        for _ in range(args.warmup):
            e2e_step()
        ms_e2e, _ = timed(e2e_step, args.steps)

    ms_per_step = ms / args.steps
    us_layer = ms_per_step * 1e3 / NL
    us_layer_e2e = ms_e2e / args.steps * 1e3 / NL
    peaks_path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(peaks_path):
        peak, peak_src = float(json.load(open(peaks_path))["hbm_gbs"]), "measured"
    else:
        peak, peak_src = 6650.0, "fallback"
    achieved = alg_bytes / (us_layer * 1e-6) / 1e9
    status = sum(int(c.status.item()) for c in caches)

    enc_tail = enc_ms[1:] if len(enc_ms) > 1 else enc_ms   # first launch pays one-time set-up
    enc_avg = sum(enc_tail) / len(enc_tail)
    if rank == 0:
        line = {
            "metric": METRIC, "value": us_layer, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms_per_step, "higher_is_better": False,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": workload_config(args),
            "clocks": clocks,
            "e2e": {"value": us_layer_e2e, "unit": UNIT, "h2d_bytes_per_step": q_host.numel() * 2,
                    "d2h_bytes_per_step": out_host.numel() * 2},
            "gpu_launches": 2 * NL * args.steps * 2,  # decode + merge kernel per layer-step, graph leg and e2e leg
            "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                         "frac": achieved / peak, "traffic": alg_bytes * DRAM_TRAFFIC_RATIO, "peak_source": peak_src,
                         "traffic_source": "ncu dram__bytes_read+write of one decode launch on a ctx-16384 case "
                                           "(282.8 MB for 268.7 MB algorithmic), scaled by token-heads",
                         "algorithmic_bytes_per_launch": alg_bytes,
                         "note": "duration = one layer-step (decode + merge kernels) from CUDA "
                                 "events over the timed region; frac_of_8TBs = %.3f" % (achieved / 8000.0)},
            "achieved_hbm_gbs_all_gpus": achieved * world,
            "token_heads_per_layer_step": tok_heads,
            "encode": {"ms_per_layer": enc_avg, "token_heads_per_s": tok_heads / (enc_avg * 1e-3)},
            "kernel_status": status, "split_invariance_max_abs": self_check,
        }
        if not args.no_cpu_baseline and world == 1:
            threads = os.cpu_count() or 1
            ref = CpuReference(args.budget, n_units=2, threads=threads)
            ref.step_us()
            v = min(ref.step_us() for _ in range(3))
            line["cpu_baseline"] = {"value": v, "unit": UNIT, "cores": threads, "kind": "port",
                                    "sample": ref.desc + ", best of 3",
                                    "same_units_gpu_vs_cpu_max_abs": ref.gpu_same_input_diff(dev),
                                    "same_units_note": "the CUDA path decoded the very units timed here (same seeded "
                                                       "keys, values, queries, codebooks); it reads int8-radius pages, "
                                                       "the reference torch path its raw fp32 radii"}
    # ---- side measurements carried in the same line: split-KV (config 5) at this run's GPU count and
    #      encode / page build (config 4); both after the headline timing, on every rank ----
    del caches, graph
    torch.cuda.empty_cache()
    splitkv = None if args.no_side else splitkv_block(args, pkg, dev, rank, world)
    encode_c4 = None
    if not args.no_side and rank == 0:
        try:
            encode_c4 = encode_c4_block(args, pkg, dev)
        except Exception as exc:  # noqa: BLE001  (a side block must not cost the headline line)
            encode_c4 = {"error": str(exc)}
    if rank == 0:
        if splitkv is not None:
            line["splitkv"] = splitkv
        if encode_c4 is not None:
            line["encode_c4"] = encode_c4
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
