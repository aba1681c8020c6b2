"""Timed workloads of the Spherical-KV hot path, through the package's public entry points.

Every case is one call (or the two calls that always go together) of a program that serves or
builds a compressed KV cache:

    decode   decode_paged: one decode-attention step of one layer over the bit-packed pages
    prefill  build_page_lists + encode_pages: a prompt's keys and values become pages
    codes    encode_codes: the code cache of every tier, one pass over the keys
    retier   build_page_lists + pages_from_codes: new tiers for a prompt that is already encoded
    pool     sphkv_encode_append + sphkv_decode: a step over the LayerPool format
    ragged   fused_decode_ragged: logits over the byte pages of one tier
    kmeans   kmeans_assign: one iteration of codebook training

Keys, values and queries are seeded Gaussians with a lognormal(0, 0.5) scale per channel (the
configurations of the benchmark), keys before RoPE where the path rotates them; codebooks are
normalised Gaussians; every token draws its tier at random (the rest of the fractions is dropped).
"""
from __future__ import annotations

import importlib
import math
import os
import sys

import torch

pkg = importlib.import_module("spherical-kv_b200")
_DROPIN = os.path.join(os.path.dirname(os.path.abspath(pkg.__file__)), "dropin")
if _DROPIN not in sys.path:
    sys.path.insert(0, _DROPIN)
import fused_decode  # noqa: E402  (the drop-in module of the package)

DEV = "cuda"
TIERS = pkg.REFERENCE_TIERS  # (g, bits): (16, 6), (16, 4), (32, 3)
DT = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
SIZE = {"f32": 4, "bf16": 2, "f16": 2}


def _decode(name, B, Hq, Hkv, dh, ctx, page, t1, t2, t3, per_head, q, v, radius, importance, uneven):
    return dict(name=name, kind="decode", B=B, Hq=Hq, Hkv=Hkv, dh=dh, ctx=ctx, page=page, t1=t1, t2=t2, t3=t3,
                per_head=per_head, q=q, v=v, radius=radius, importance=importance, uneven=uneven)


def _prefill(name, kind, B, Hkv, dh, ctx, page, t1, t2, t3, per_head, k, v, radius):
    return dict(name=name, kind=kind, B=B, Hkv=Hkv, dh=dh, ctx=ctx, page=page, t1=t1, t2=t2, t3=t3,
                per_head=per_head, k=k, v=v, radius=radius)


def listed():
    return [
        # decode attention, the serving loop: one layer of one step.  A 1B-class head shape with one
        # short sequence (latency), an 8B-class batch at 8K, the benchmark's 32K batch (the largest), and
        # one 128K sequence (the grid has to be filled from a single row)
        _decode("decode_b1_2k_dh64", 1, 32, 8, 64, 2048, 16, 0.5, 0.5, 0.0, False, "f32", "f16", "f16", False, False),
        _decode("decode_b16_8k", 16, 32, 8, 128, 8192, 16, 0.3, 0.6, 0.0, False, "bf16", "bf16", "i8", False, False),
        _decode("decode_b8_32k", 8, 32, 8, 128, 32768, 16, 0.31, 0.62, 0.0, False, "bf16", "bf16", "i8", False, False),
        _decode("decode_b1_128k", 1, 32, 8, 128, 131072, 16, 0.2, 0.6, 0.0, True, "bf16", "bf16", "i8", False, False),
        # the reference pipeline's own setting: 128-token pages, all three tiers, tiers chosen per head, fp16
        # values, and the page-importance update that its re-tiering reads; rows of different, odd lengths
        _decode("decode_b3_6k_page128", 3, 32, 8, 128, 6001, 128, 0.2, 0.5, 0.2, True, "f32", "f16", "i8", True, True),
        # prompts coming in: a short odd one (launches and host work count) and a long one in fp32
        _prefill("prefill_777", "prefill", 1, 8, 128, 777, 16, 0.3, 0.6, 0.0, True, "bf16", "bf16", "i8"),
        _prefill("prefill_32k", "prefill", 1, 8, 128, 32768, 16, 0.3, 0.6, 0.0, False, "f32", "bf16", "i8"),
        # all tiers encoded ahead (fp32 keys), and a later change of the tiers of a prompt
        _prefill("codes_32k", "codes", 1, 8, 128, 32768, 16, 1.0, 1.0, 1.0, False, "f32", "bf16", "i8"),
        _prefill("retier_8k", "retier", 1, 8, 128, 8190, 128, 0.2, 0.5, 0.3, True, "bf16", "f16", "i8"),
        # the drop-in operators that the reference's pipeline calls in its decode loop
        dict(name="pool_step_4k", kind="pool", Hq=32, Hkv=8, dh=128, ctx=4000, page=128),
        dict(name="ragged_4k", kind="ragged", Hq=32, Hkv=8, dh=128, ctx=4097, page=128, tier=2, keep=0.6),
        # codebook training
        dict(name="kmeans_4m", kind="kmeans", points=4000000, d=16, K=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mix(rng):
    keep = rng.uniform(0.4, 1.0)
    t1 = round(keep * rng.uniform(0.15, 0.5), 3)
    t3 = round(keep * rng.choice([0.0, 0.0, rng.uniform(0.1, 0.3)]), 3)
    return t1, round(keep - t1 - t3, 3), t3


def draw(rng):
    kind = rng.choice(["decode"] * 5 + ["prefill"] * 2 + ["codes", "retier", "pool", "ragged", "kmeans"])
    Hq, Hkv = rng.choice([(32, 8), (32, 8), (16, 2), (16, 8), (8, 8)])
    dh = rng.choice([64, 128, 128])
    page = rng.choice([16, 16, 32, 64, 128])
    t1, t2, t3 = _mix(rng)
    v = rng.choice(["bf16", "f16"])
    radius = rng.choice(["i8", "i8", "i8", "f16"])
    per_head = rng.random() < 0.5
    if kind == "decode":
        B = rng.choice([1, 1, 2, 3, 5, 8, 16])
        ctx = _log(rng, 256, min(131072, 2000000 // (B * Hkv)))
        c = _decode("", B, Hq, Hkv, dh, ctx, page, t1, t2, t3, per_head, rng.choice(["bf16", "f32", "f16"]), v, radius,
                    rng.random() < 0.25, rng.random() < 0.4)
    elif kind in ("prefill", "codes", "retier"):
        B = rng.choice([1, 1, 2, 3])
        ctx = _log(rng, 64, 32768 // B)
        c = _prefill("", kind, B, Hkv, dh, ctx, page, t1, t2, t3, per_head, rng.choice(["f32", "bf16", "f16"]), v, radius)
    elif kind == "pool":
        c = dict(kind=kind, Hq=Hq, Hkv=Hkv, dh=dh, ctx=_log(rng, 256, 32768), page=rng.choice([16, 128]))
    elif kind == "ragged":
        c = dict(kind=kind, Hq=Hq, Hkv=Hkv, dh=dh, ctx=_log(rng, 256, 16384), page=rng.choice([16, 128]),
                 tier=rng.choice([1, 2, 3]), keep=round(rng.uniform(0.2, 0.9), 3))
    else:
        d, K = rng.choice([(16, 64), (16, 16), (32, 8), (16, 8)])
        c = dict(kind=kind, points=_log(rng, 4096, 4000000), d=d, K=K)
    c.pop("name", None)
    return c


# ---- inputs ------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _scaled(g, scale, *shape):
    return torch.randn(*shape, scale.numel(), generator=g, device=DEV) * scale


def _scale(g, dh):
    return torch.exp(0.5 * torch.randn(dh, generator=g, device=DEV))


def _codebooks(g, Hkv, dh, specs):
    out = []
    for t in specs:
        c = torch.randn(Hkv, dh // t.g, 1 << t.b_theta, t.g, generator=g, device=DEV)
        out.append(c / c.norm(dim=-1, keepdim=True))
    return out


def _counts(c):
    """Tokens of every (batch row, KV head) in tiers 1, 2, 3: [B][Hkv][3].  An uneven batch has rows of
    different lengths (down to a quarter); tiers chosen per head keep 70 .. 100 % of the mix by head."""
    out = []
    for b in range(c["B"]):
        length = _length(c, b)
        row = []
        for h in range(c["Hkv"]):
            keep = 1.0 - 0.3 * ((5 * h + 3 * b) % 8) / 7 if c["per_head"] else 1.0
            row.append([int(length * c["t%d" % tid] * keep) for tid in (1, 2, 3)])
        out.append(row)
    return out


def _length(c, b):
    return c["ctx"] if not c.get("uneven") else max(16, int(c["ctx"] * (1.0 - 0.75 * b / max(1, c["B"] - 1))))


def _assign(g, c):
    """Tier of every token, u8 [B, Hkv, ctx]; 0 = dropped (or past the end of a shorter row).  How many
    tokens a tier holds follows from the case, which ones is random."""
    u = torch.rand(c["B"], c["Hkv"] if c["per_head"] else 1, c["ctx"], generator=g, device=DEV)
    for b in range(c["B"]):
        u[b, :, _length(c, b):] = 2.0
    rank = u.argsort(-1).argsort(-1).expand(c["B"], c["Hkv"], c["ctx"])
    ends = torch.tensor(_counts(c), device=DEV).cumsum(-1)
    a = torch.zeros(rank.shape, dtype=torch.uint8, device=DEV)
    for tid in (3, 2, 1):
        a[rank < ends[..., tid - 1:tid]] = tid
    return a


def _specs(c):
    return [t for t in TIERS if c["t%d" % t.tier_id] > 0]


def _fmt(c):
    return pkg.RADIUS_F16 if c["radius"] == "f16" else pkg.RADIUS_I8


def _prepare_decode(c, g):
    B, Hkv, dh, ctx = c["B"], c["Hkv"], c["dh"], c["ctx"]
    specs = _specs(c)
    tiers = pkg.TierSet(dh, specs)
    scale = _scale(g, dh)
    K = torch.empty(B * ctx, Hkv, dh, dtype=torch.bfloat16, device=DEV)
    V = torch.empty_like(K)
    for b in range(B):
        K[b * ctx:(b + 1) * ctx] = _scaled(g, scale, ctx, Hkv)
        V[b * ctx:(b + 1) * ctx] = _scaled(g, scale, ctx, Hkv)
    lists = pkg.build_page_lists(_assign(g, c), tiers, c["page"], radius_fmt=_fmt(c),
                                 shuffle_seed=int(torch.randint(1 << 30, (1,), generator=g, device=DEV)))
    cache = pkg.encode_pages(K, V, lists, tiers.pack_codebooks(_codebooks(g, Hkv, dh, specs)), tiers,
                             radius_fmt=_fmt(c), v_dtype=DT[c["v"]])
    s = dict(cache=cache, q=_scaled(g, scale, B, c["Hq"]).to(DT[c["q"]]), rope=pkg.rope_table(ctx + 8, dh, device=DEV))
    if c["importance"]:
        s["omega"] = torch.rand(B * Hkv, lists.max_blocks, generator=g, device=DEV)
    return s


def _prepare_prefill(c, g):
    B, Hkv, dh, ctx = c["B"], c["Hkv"], c["dh"], c["ctx"]
    specs = TIERS if c["kind"] == "codes" else _specs(c)
    tiers = pkg.TierSet(dh, specs)
    scale = _scale(g, dh)
    K = _scaled(g, scale, B * ctx, Hkv).to(DT[c["k"]])
    s = dict(tiers=tiers, cb=tiers.pack_codebooks(_codebooks(g, Hkv, dh, specs)), assign=None)
    if c["kind"] != "retier":
        s["K"] = K
    if c["kind"] != "codes":
        s["V"] = _scaled(g, scale, B * ctx, Hkv).to(DT[c["k"]])
        s["assign"] = _assign(g, c)
    if c["kind"] == "retier":
        s["codes"] = pkg.encode_codes(K, s["cb"], tiers)
    return s


def _prepare_pool(c, g):
    """A LayerPool of one sequence: a quarter / half / quarter of every head's tokens in tiers 1 / 2 / 3,
    one page of every head open for the step's token."""
    Hkv, dh, N = c["Hkv"], c["dh"], c["page"]
    tiers = pkg.TierSet(dh, TIERS)
    n = [-(-c["ctx"] * f // (4 * N)) for f in (1, 2, 1)]          # pages of each tier per head
    per_head = sum(n)
    P = Hkv * per_head + 4
    slot_of = torch.cat([torch.full((k,), i, dtype=torch.int32) for i, k in enumerate(n)]).to(DEV)
    order = torch.randperm(P, generator=g, device=DEV)[:Hkv * per_head].reshape(Hkv, per_head)
    theta = torch.zeros(P, N, tiers.G_max, dtype=torch.uint8, device=DEV)
    radius = torch.zeros_like(theta)
    scales = torch.zeros(P, tiers.G_max, device=DEV)
    for i, t in enumerate(TIERS):
        pages = order[:, slot_of == i].reshape(-1)
        G = dh // t.g
        r = torch.rand(pages.numel(), N, G, generator=g, device=DEV) * 0.8 + 0.2
        scales[pages, :G] = r.amax(1) * math.sqrt(t.g)
        theta[pages, :, :G] = torch.randint(1 << t.b_theta, (pages.numel(), N, G), generator=g, device=DEV).to(torch.uint8)
        radius[pages, :, :G] = (r / r.amax(1, keepdim=True) * 255).round().to(torch.uint8)
    max_blocks = per_head + 2
    table = torch.full((Hkv, max_blocks), -1, dtype=torch.int32, device=DEV)
    table[:, :per_head] = order.to(torch.int32)
    bits = torch.zeros_like(table)
    bits[:, :per_head] = slot_of
    cbs = _codebooks(g, Hkv, dh, TIERS)
    scale = _scale(g, dh)
    return dict(
        q=_scaled(g, scale, c["Hq"]), k=_scaled(g, scale, Hkv), v=_scaled(g, scale, Hkv),
        cb=tiers.pack_codebooks(cbs), append_cb=cbs[0].contiguous(),
        tier_G=torch.tensor([dh // t.g for t in TIERS], dtype=torch.int32, device=DEV),
        tier_g=torch.tensor([t.g for t in TIERS], dtype=torch.int32, device=DEV),
        theta=theta, radius=radius, scales=scales, v_pool=_scaled(g, scale, P, N).half(),
        table=table, bits=bits, ctx=torch.full((Hkv,), per_head * N, dtype=torch.int32, device=DEV),
        pids=order[:, 0].contiguous(), out=torch.zeros(c["Hq"], dh, device=DEV),
        part=torch.zeros(c["Hq"], max_blocks, dh + 2, device=DEV), tiers=tiers, max_blocks=max_blocks)


def _prepare_ragged(c, g):
    Hkv, dh, ctx = c["Hkv"], c["dh"], c["ctx"]
    t = TIERS[c["tier"] - 1]
    tiers = pkg.TierSet(dh, [t])
    scale = _scale(g, dh)
    u = torch.rand(1, Hkv, ctx, generator=g, device=DEV)
    keep = u.argsort(-1).argsort(-1) < max(1, int(ctx * c["keep"]))
    lists = pkg.build_page_lists(keep.to(torch.uint8) * t.tier_id, tiers, c["page"], page_align=4)
    cbs = _codebooks(g, Hkv, dh, [t])
    cache = pkg.encode_pages(_scaled(g, scale, ctx, Hkv), None, lists, tiers.pack_codebooks(cbs), tiers)
    ang = torch.arange(ctx, device=DEV).float()[:, None] * pkg.hf_inv_freq(dh).to(DEV)[None]
    ang = torch.cat([ang, ang], 1)
    return dict(pages=cache.k_pages, lists=lists, positions=lists.positions.reshape(-1), cos=ang.cos(), sin=ang.sin(),
                q=_scaled(g, scale, c["Hq"]), cb=cbs[0].reshape(Hkv * (dh // t.g), 1 << t.b_theta, t.g).contiguous(), t=t)


def _prepare_kmeans(c, g):
    unit = lambda n: torch.nn.functional.normalize(torch.randn(n, c["d"], generator=g, device=DEV), dim=1)  # noqa: E731
    return dict(U=unit(c["points"]), centers=unit(c["K"]))


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    make = {"decode": _prepare_decode, "prefill": _prepare_prefill, "codes": _prepare_prefill, "retier": _prepare_prefill,
            "pool": _prepare_pool, "ragged": _prepare_ragged, "kmeans": _prepare_kmeans}[kind]
    s = make(case, g)
    s["case"] = dict(case)
    return s


# ---- one pass ----------------------------------------------------------------------------------
def _lists_out(L):
    return {k: getattr(L, k) for k in ("positions", "src_index", "page_head", "page_slot", "page_count", "ptable",
                                       "block_table", "bits_table", "num_blocks", "bundles")}


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "decode":
        if c["importance"]:
            out = pkg.decode_paged(s["q"], s["cache"], s["rope"], omega=s["omega"])
            return {"out": out, "omega": s["omega"]}
        return pkg.decode_paged(s["q"], s["cache"], s["rope"])
    if kind == "codes":
        codes = pkg.encode_codes(s["K"], s["cb"], s["tiers"])
        return {"r": codes.r, "theta": codes.theta}
    if kind in ("prefill", "retier"):
        lists = pkg.build_page_lists(s["assign"], s["tiers"], c["page"], radius_fmt=_fmt(c))
        if kind == "prefill":
            cache = pkg.encode_pages(s["K"], s["V"], lists, s["cb"], s["tiers"], radius_fmt=_fmt(c), v_dtype=DT[c["v"]])
        else:
            cache = pkg.pages_from_codes(s["codes"], s["V"], lists, s["cb"], radius_fmt=_fmt(c), v_dtype=DT[c["v"]])
        return dict(_lists_out(lists), k_pages=cache.k_pages, v_pool=cache.v_pool)
    if kind == "pool":
        t, T = TIERS[0], s["tiers"]
        fused_decode.sphkv_encode_append(s["k"], s["v"], s["append_cb"], s["theta"], s["radius"], s["scales"], s["v_pool"],
                                         s["pids"], c["page"] - 3, c["dh"] // t.g, t.g, 1 << t.b_theta, T.G_max, c["dh"],
                                         c["page"], 0)
        fused_decode.sphkv_decode(s["q"], s["cb"], s["tier_G"], s["tier_g"], s["theta"], s["radius"], s["scales"],
                                  s["v_pool"], s["table"], s["bits"], s["ctx"], s["out"], s["part"], c["Hq"], c["Hkv"],
                                  c["Hq"] // c["Hkv"], len(TIERS), s["max_blocks"], c["page"], c["dh"], T.G_max, T.C_max,
                                  T.g_max, 1.0 / math.sqrt(c["dh"]), c["ctx"])
        return {k: s[k] for k in ("out", "part", "theta", "radius", "scales", "v_pool")}
    if kind == "ragged":
        L, t = s["lists"], s["t"]
        return fused_decode.fused_decode_ragged(s["pages"], L.ptable, L.page_head, s["positions"], s["cos"], s["sin"], s["q"],
                                                c["Hq"] // c["Hkv"], c["Hkv"], s["cb"], c["dh"], c["dh"] // t.g, t.g,
                                                t.b_theta, c["page"])
    assigns, best, sums, counts = pkg.kmeans_assign(s["U"], s["centers"])
    return {"assigns": assigns, "best": best, "sums": sums, "counts": counts}


# ---- what a pass cannot do without ---------------------------------------------------------------
def _page_bytes(c, dh, rb):
    """Tokens per tier, pages, K page bytes, multiply-adds of the centroid search."""
    per_tier, pages, nbytes, macs = [], 0, 0, 0
    for t in TIERS:
        G = dh // t.g
        ns = [row[t.tier_id - 1] for heads in _counts(c) for row in heads]
        p = sum(-(-n // c["page"]) for n in ns)
        per_tier.append(sum(ns))
        pages += p
        nbytes += p * (8 + 4 * G) + sum(-(-n * G * t.b_theta // 8) + n * G * rb for n in ns)
        macs += sum(ns) * dh * (1 << t.b_theta)
    return per_tier, pages, nbytes, macs


def work(case):
    c, kind = case, case["kind"]
    if kind == "kmeans":
        n, d, K = c["points"], c["d"], c["K"]
        return {"bytes": n * (4 * d + 8) + 8 * K * d, "flops": 2.0 * n * d * K}
    dh = c["dh"]
    if kind == "pool":
        tokens = c["Hkv"] * c["ctx"]
        blocks = c["ctx"] / c["page"]
        grp = c["Hq"] // c["Hkv"]
        # codes and scales, fp16 values, the per-page partial rows that the call returns, codebooks
        b = tokens * (2 * 7 + 2 * dh) + c["Hkv"] * blocks * 40 + c["Hq"] * blocks * (dh + 2) * 4 + c["Hkv"] * dh * 88 * 4
        return {"bytes": b, "flops": tokens * grp * (16 + 2 * dh) + c["Hq"] * dh * 88 * 2}
    if kind == "ragged":
        t = TIERS[c["tier"] - 1]
        G = dh // t.g
        n = c["Hkv"] * c["ctx"] * c["keep"]
        slots = c["Hkv"] * math.ceil(c["ctx"] * c["keep"] / c["page"]) * c["page"]
        b = n * (G * t.b_theta / 8 + G) + slots * 4 + c["ctx"] * dh * 8 + c["Hq"] * slots * 4 + c["Hkv"] * dh * (4 << t.b_theta)
        # the query is rotated, normalised per group and matched for every token and query head
        return {"bytes": b, "flops": n * (c["Hq"] // c["Hkv"]) * dh * 7}
    heads = c["B"] * c["Hkv"]
    rb = 2 if c["radius"] == "f16" else 1
    if kind == "codes":
        n = heads * c["ctx"]
        return {"bytes": n * (dh * SIZE[c["k"]] + 5 * (2 * (dh // 16) + dh // 32)) + c["Hkv"] * dh * 88 * 4,
                "flops": 2.0 * n * dh * (64 + 16 + 8 + 1)}
    per_tier, pages, nbytes, macs = _page_bytes(c, dh, rb)
    kept = sum(per_tier)
    if kind == "decode":
        grp = c["Hq"] // c["Hkv"]
        b = nbytes + kept * (2 * dh + 4) + pages * (8 + 12) + c["ctx"] * dh * 4
        b += c["B"] * c["Hq"] * dh * 2 * SIZE[c["q"]] + c["Hkv"] * sum(dh * (4 << t.b_theta) for t in _specs(c))
        if c["importance"]:
            b += pages * 8
        return {"bytes": b, "flops": kept * dh * (4 * grp + 4)}
    # prefill / retier: tier of every token, tables and lists, pages out, values in and out
    lists = heads * c["ctx"] + pages * (12 + 3 * 4 + 2 * 4 + 4) + pages * c["page"] * 8
    b = lists + nbytes + kept * dh * SIZE[c["k"]] + pages * c["page"] * dh * 2
    if kind == "prefill":
        return {"bytes": b + kept * dh * SIZE[c["k"]], "flops": 2.0 * macs}
    code_bytes = sum(n * (dh // t.g) * 5 for n, t in zip(per_tier, TIERS))
    return {"bytes": b + code_bytes, "flops": 0.0}


def tolerance(case):
    kind = case["kind"]
    if kind in ("prefill", "codes", "retier"):
        return "exact"  # codes, bytes and tables are whole numbers; radii follow one fixed fp32 order
    if kind == "decode":
        # keys enter the tensor cores with 16 mantissa bits, the softmax weights with 11 (fp16 values) or 16
        # (bf16 values); a 16-bit output adds its own rounding
        return {"rel": 2e-3} if case["q"] == "f32" else {"rel": 1e-2}
    return {"rel": 2e-5}  # fp32 sums in another order; codes, assignments and counts have to be equal
