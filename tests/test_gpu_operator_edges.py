"""GPU: the reference-signature operators at the edges of their dispatch -- warps per page of the pool
decode, rows-across-lanes ragged logits -- against the CPU restatements."""
import math
import os
import sys

import numpy as np
import pytest
import torch

from test_gpu_compat import dev, make_pool
from util import ROOT, load_oracle, load_pkg

pkg = load_pkg()
orc = load_oracle()
synth = pkg.synth
pytestmark = pytest.mark.gpu
DEV = "cuda:0"
sys.path.insert(0, os.path.join(ROOT, "spherical-kv_b200", "dropin"))


# page sizes that split over 1, 2, 4, 8 warps and one that does not split evenly; 1, 3 and 8 query heads
@pytest.mark.parametrize("page_size,dh,grp", [(16, 64, 3), (32, 128, 8), (64, 128, 1), (128, 64, 4), (24, 128, 4), (40, 64, 4)])
def test_pool_decode_page_splits(page_size, dh, grp):
    import fused_decode
    Hkv = 2
    Hq = Hkv * grp
    pool = make_pool(Hkv, grp, dh, [page_size * 11 + 1, 3], page_size, seed=page_size)
    G_max, C_max, g_max, max_blocks = pool["dims"]
    q = torch.randn(Hq, dh, generator=torch.Generator().manual_seed(5))
    sm = 1.0 / math.sqrt(dh)
    want, want_part = orc.pool_decode(q, pool["cb_flat"], pool["tier_G"], pool["tier_g"], pool["theta"], pool["radius"],
                                      pool["scales"], pool["v"], pool["block_table"], pool["bits_table"], sm)
    d = dev(pool)
    out, part = torch.zeros(Hq, dh, device=DEV), torch.full((Hq, max_blocks, dh + 2), 7.0, device=DEV)
    fused_decode.sphkv_decode(q.to(DEV), d["cb_flat"], d["tier_G"], d["tier_g"], d["theta"], d["radius"], d["scales"],
                              d["v"], d["block_table"], d["bits_table"], d["ctx_lens"], out, part, Hq, Hkv, grp, 3,
                              max_blocks, page_size, dh, G_max, C_max, g_max, sm, int(pool["ctx_lens"].max()))
    assert (out.cpu() - want).abs().max().item() <= 2e-4
    gp, live = part.cpu(), torch.isfinite(want_part[:, :, 0])
    assert torch.equal(torch.isfinite(gp[:, :, 0]), live) and (gp[:, :, 1:][~live] == 0).all()
    # fp32 sums of at most page_size terms in another order: a few ulps of the sum of magnitudes
    assert (gp[live] - want_part[live]).abs().max().item() <= 1e-4 * want_part[live].abs().max().item()


@pytest.mark.parametrize("dh,page_size,tier,grp", [(64, 16, 0, 4), (64, 128, 2, 1), (128, 32, 1, 8), (128, 48, 2, 5)])
def test_ragged_logits_shapes(dh, page_size, tier, grp):
    import fused_decode
    t = pkg.REFERENCE_TIERS[tier]
    Hkv, ctx = 3, 150
    Hq, G = Hkv * grp, dh // t.g
    tiers = pkg.TierSet(dh, [t])
    K, V, Q, _ = synth.make_kvq(1, Hq, Hkv, dh, ctx, seed=2)
    cbs = synth.make_codebooks(Hkv, dh, [t], seed=3)
    assign = synth.make_tier_assign(1, Hkv, ctx, {t.tier_id: 0.6}, seed=4, per_head=True)
    lists = pkg.build_page_lists(assign, tiers, page_size, page_align=4)
    pages = np.zeros(lists.pool_bytes + 16, np.uint8)
    want = torch.zeros(Hq, lists.n_pages * page_size)
    cos, sin = orc.rope_tables(ctx + 4, dh)
    for ph in range(lists.n_pages):
        c, h = int(lists.page_count[ph]), int(lists.page_head[ph])
        rows = lists.src_index[ph, :c].long()
        r, th = orc.encode(K.reshape(ctx, Hkv, dh)[rows, h].contiguous(), cbs[0][h])
        page, _, _ = orc.build_page(r, th, t.b_theta, t.tier_id, 0)
        po = int(lists.ptable[ph, 0])
        pages[po:po + page.size] = page
        _, _, _, th2, r2 = orc.parse_page(pages, *(int(x) for x in lists.ptable[ph]), G, t.b_theta, 0)
        want[h * grp:(h + 1) * grp, ph * page_size:ph * page_size + c] = orc.backrot_logits(
            Q[0, h * grp:(h + 1) * grp], torch.from_numpy(r2), torch.from_numpy(th2), lists.positions[ph, :c].long(),
            cbs[0][h], cos, sin)
    got = fused_decode.fused_decode_ragged(
        torch.from_numpy(pages).to(DEV), lists.ptable.to(DEV), lists.page_head.to(DEV),
        lists.positions.reshape(-1).to(DEV), cos.to(DEV), sin.to(DEV), Q[0].to(DEV), grp, Hkv,
        torch.cat([cbs[0][h] for h in range(Hkv)], 0).to(DEV), dh, G, t.g, t.b_theta, page_size).cpu()
    assert (got - want).abs().max().item() <= 2e-4
    assert torch.equal(got == 0, want == 0)


# CTAs that take several rounds of pages, restaging their rows between them: a warp per page (16-token pages) and eight
# warps per page; holes, a last round that is partly empty, and a second pool so that what the first call left in
# shared memory cannot match
@pytest.mark.parametrize("page_size,grp", [(16, 2), (128, 1)])
@pytest.mark.parametrize("rounds", [1, 2, 3, 4])
def test_pool_decode_rounds(page_size, grp, rounds):
    import fused_decode
    Hkv, dh = 8, 128
    tiers = pkg.TierSet(dh, pkg.REFERENCE_TIERS)
    at_once = 8 if page_size == 16 else 1
    max_blocks = -(-rounds * at_once * 2 * pkg._lib.load().sphkv_sm_count() // Hkv) + 3
    for seed in (1, 2):
        g = torch.Generator().manual_seed(10 * rounds + seed)
        cbs = synth.make_codebooks(Hkv, dh, pkg.REFERENCE_TIERS, seed=seed)
        P = 150                                              # pages may repeat in the lists: they are only read
        bits = torch.randint(0, 3, (Hkv, max_blocks), generator=g, dtype=torch.int32)
        table = torch.randint(0, P // 3, (Hkv, max_blocks), generator=g, dtype=torch.int32) * 3 + bits
        table[torch.rand(Hkv, max_blocks, generator=g) < 0.05] = -1
        C = torch.tensor([1 << t.b_theta for t in pkg.REFERENCE_TIERS])[torch.arange(P) % 3]
        theta = (torch.rand(P, page_size, tiers.G_max, generator=g) * C[:, None, None]).to(torch.uint8)
        radius = torch.randint(0, 256, theta.shape, generator=g).to(torch.uint8)
        scales = torch.rand(P, tiers.G_max, generator=g) + 0.5
        v = torch.randn(P, page_size, dh, generator=g).half()
        tier_G = torch.tensor([dh // t.g for t in pkg.REFERENCE_TIERS], dtype=torch.int32)
        tier_g = torch.tensor([t.g for t in pkg.REFERENCE_TIERS], dtype=torch.int32)
        cb = tiers.pack_codebooks(cbs)
        Hq, sm = Hkv * grp, 1.0 / math.sqrt(dh)
        q = torch.randn(Hq, dh, generator=g)
        want, want_part = orc.pool_decode(q, cb, tier_G, tier_g, theta, radius, scales, v, table, bits, sm)
        out, part = torch.zeros(Hq, dh, device=DEV), torch.full((Hq, max_blocks, dh + 2), 7.0, device=DEV)
        ctx = torch.full((Hkv,), max_blocks * page_size, dtype=torch.int32, device=DEV)
        fused_decode.sphkv_decode(q.to(DEV), cb.to(DEV), tier_G.to(DEV), tier_g.to(DEV), theta.to(DEV), radius.to(DEV),
                                  scales.to(DEV), v.to(DEV), table.to(DEV), bits.to(DEV), ctx, out, part, Hq, Hkv, grp, 3,
                                  max_blocks, page_size, dh, tiers.G_max, tiers.C_max, tiers.g_max, sm, max_blocks * page_size)
        gp, live = part.cpu(), torch.isfinite(want_part[:, :, 0])
        assert torch.equal(torch.isfinite(gp[:, :, 0]), live) and (gp[:, :, 1:][~live] == 0).all()
        # fp32 sums of at most page_size terms in another order: a few ulps of the sum of magnitudes
        assert (gp[live] - want_part[live]).abs().max().item() <= 1e-4 * want_part[live].abs().max().item()
        assert (out.cpu() - want).abs().max().item() <= 2e-4


def random_pool(seed, Hkv, dh, page_size, max_blocks, g, C, n_tiers=1, P=20):
    """A LayerPool of one group size and C centroids per group, random codes and a hole per head."""
    gen = torch.Generator().manual_seed(seed)
    G = dh // g
    cb = torch.nn.functional.normalize(torch.randn(Hkv, n_tiers, G, C, g, generator=gen), dim=-1)
    table = torch.randint(0, P, (Hkv, max_blocks), generator=gen, dtype=torch.int32)
    table[:, 1] = -1
    return dict(cb=cb, table=table, bits=torch.randint(0, n_tiers, (Hkv, max_blocks), generator=gen, dtype=torch.int32),
                theta=torch.randint(0, C, (P, page_size, G), generator=gen).to(torch.uint8),
                radius=torch.randint(1, 256, (P, page_size, G), generator=gen).to(torch.uint8),
                scales=torch.rand(P, G, generator=gen) + 0.5, v=torch.randn(P, page_size, dh, generator=gen).half(),
                tier_G=torch.full((n_tiers,), G, dtype=torch.int32), tier_g=torch.full((n_tiers,), g, dtype=torch.int32))


def run_pool(pool, q, grp):
    import fused_decode
    Hkv, max_blocks = pool["table"].shape
    _, n_tiers, G, C, g = pool["cb"].shape
    Hq, dh = q.shape
    page_size, sm = pool["theta"].shape[1], 1.0 / math.sqrt(dh)
    out, part = torch.zeros(Hq, dh, device=DEV), torch.full((Hq, max_blocks, dh + 2), 7.0, device=DEV)
    d = {k: x.to(DEV) for k, x in pool.items()}
    fused_decode.sphkv_decode(q.to(DEV), d["cb"], d["tier_G"], d["tier_g"], d["theta"], d["radius"], d["scales"], d["v"],
                              d["table"], d["bits"], torch.full((Hkv,), max_blocks * page_size, dtype=torch.int32, device=DEV),
                              out, part, Hq, Hkv, grp, n_tiers, max_blocks, page_size, dh, G, C, g, sm, max_blocks * page_size)
    want, want_part = orc.pool_decode(q, pool["cb"], pool["tier_G"], pool["tier_g"], pool["theta"], pool["radius"],
                                      pool["scales"], pool["v"], pool["table"], pool["bits"], sm)
    return out.cpu(), part.cpu(), want, want_part


# tables of an odd number of floats in front of the pieces that are stored eight bytes at a time
@pytest.mark.parametrize("page_size", [16, 32, 128])
@pytest.mark.parametrize("dh,g,C,n_tiers,grp", [(48, 16, 5, 1, 1), (48, 16, 7, 3, 3), (80, 16, 3, 1, 5)])
def test_pool_decode_odd_table_sizes(page_size, dh, g, C, n_tiers, grp):
    pool = random_pool(dh + C, 2, dh, page_size, 7, g, C, n_tiers)
    q = torch.randn(2 * grp, dh, generator=torch.Generator().manual_seed(1))
    out, part, want, want_part = run_pool(pool, q, grp)
    live = torch.isfinite(want_part[:, :, 0])
    assert (out - want).abs().max().item() <= 2e-4
    # fp32 sums of at most page_size terms in another order: a few ulps of the sum of magnitudes
    assert (part[live] - want_part[live]).abs().max().item() <= 1e-4 * want_part[live].abs().max().item()


# a warp's 16 tokens all at -inf, and single tokens at -inf, beside finite logits in the same page
@pytest.mark.parametrize("page_size", [32, 128])
def test_pool_decode_tokens_at_minus_infinity(page_size):
    pool = random_pool(3, 2, 64, page_size, 5, 16, 2)
    pool["cb"][..., 0, 0], pool["cb"][..., 1, 0] = -1000.0, 1e-36   # times 3e38 / 255: overflows, and about one
    pool["scales"][:, 0], pool["scales"][:, 1:], pool["radius"][:] = 3e38, 0.0, 1
    pool["theta"][:] = 1
    pool["theta"][:, :16] = 0
    pool["theta"][:, 20] = 0
    q = torch.zeros(2, 64)
    q[:, 0] = 1.0
    out, part, want, want_part = run_pool(pool, q, 1)
    live = torch.isfinite(want_part[:, :, 0])
    assert torch.isfinite(want).all() and live.sum() == 8
    assert (out - want).abs().max().item() <= 2e-4
    assert (part[live] - want_part[live]).abs().max().item() <= 1e-4 * want_part[live].abs().max().item()


# group sizes beside the reference's 16 and 32: tables built in 16-byte pieces, and element by element
@pytest.mark.parametrize("dh,g,C", [(128, 8, 64), (128, 64, 64), (120, 10, 16), (128, 4, 16)])
def test_pool_decode_other_group_sizes(dh, g, C):
    pool = random_pool(g, 2, dh, 32, 9, g, C, 2)
    q = torch.randn(8, dh, generator=torch.Generator().manual_seed(1))
    out, part, want, want_part = run_pool(pool, q, 4)
    live = torch.isfinite(want_part[:, :, 0])
    assert (out - want).abs().max().item() <= 2e-4
    assert (part[live] - want_part[live]).abs().max().item() <= 1e-4 * want_part[live].abs().max().item()


def test_pool_decode_of_more_pages_than_a_grid_has_rows():
    """128-token pages, one page per CTA at a time: four rounds of them leave more CTAs than a grid's second dimension"""
    mb = 4 * 65535 + 1000
    pool = random_pool(7, 1, 16, 128, mb, 16, 4)
    live = torch.tensor([0, 5, 4 * 65535 - 1, 4 * 65535, mb - 1])
    table = torch.full((1, mb), -1, dtype=torch.int32)
    table[0, live] = torch.arange(5, dtype=torch.int32)
    pool["table"] = table
    q = torch.randn(1, 16, generator=torch.Generator().manual_seed(1))
    out, part, want, want_part = run_pool(pool, q, 1)
    assert (out - want).abs().max().item() <= 2e-4
    assert torch.equal(torch.isfinite(part[0, :, 0]), table[0] >= 0)
    assert (part[0, live] - want_part[0, live]).abs().max().item() <= 1e-4 * want_part[0, live].abs().max().item()
