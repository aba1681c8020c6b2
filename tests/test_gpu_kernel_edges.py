"""GPU: edges of the dispatch rules and tiles of the decode, encode and k-means kernels."""
import pytest
import torch

from test_gpu_decode import DEV, build, check_against_oracle
from util import load_pkg

pkg = load_pkg()
synth = pkg.synth
pytestmark = pytest.mark.gpu
T1, T2, T3 = pkg.REFERENCE_TIERS


# tiles per segment around the 24 of a round of three teams and the 8 of a macro tile; blocks dealt by unit (few
# units) and by range (more units than CTAs divide evenly, uneven rows); a tier whose theta stream holds
# fewer than eight bits per token (dh 64, tier 3)
@pytest.mark.parametrize("B,Hkv,dh,ctx,page,specs,fr", [
    (1, 1, 128, 16, 16, (T1,), {1: 1.0}),
    (1, 2, 128, 129, 16, (T1,), {1: 1.0}),
    (1, 1, 64, 385, 16, (T2, T3), {2: 0.5, 3: 0.5}),
    (1, 3, 64, 4000, 64, (T1, T3), {1: 0.3, 3: 0.6}),
    (19, 8, 64, 150, 32, (T1, T2), {1: 0.4, 2: 0.4}),
    (5, 8, 128, 700, 16, (T1, T2, T3), {1: 0.2, 2: 0.3, 3: 0.3}),
])
@pytest.mark.parametrize("radius_fmt", [0, 1])
def test_decode_segment_shapes(B, Hkv, dh, ctx, page, specs, fr, radius_fmt):
    cache, cbs, K, V, Q, _ = build(B, 2 * Hkv, Hkv, dh, ctx, page, specs, fr, radius_fmt=radius_fmt, seed=ctx)
    check_against_oracle(cache, cbs, Q, ctx, dh)


# batch x KV heads and tier sets at which one, two or three teams and one or two copies of a codebook just fit shared memory
@pytest.mark.parametrize("B,Hkv,dh,ctx,bits", [
    (16, 8, 128, 150, (6, 6, 6, 6)), (16, 8, 128, 100, (6, 6, 6)), (75, 2, 128, 100, (6, 6, 5, 2)), (80, 8, 128, 40, (6, 4)),
    (24, 8, 128, 90, (6, 6, 6, 6)), (64, 8, 64, 70, (6, 6, 6, 6))])
def test_decode_where_teams_and_copies_just_fit(B, Hkv, dh, ctx, bits):
    specs = [pkg.TierSpec(i + 1, 16, b) for i, b in enumerate(bits)]
    cache, cbs, K, V, Q, _ = build(B, 2 * Hkv, Hkv, dh, ctx, 16, specs, {t.tier_id: 0.9 / len(bits) for t in specs}, seed=ctx)
    check_against_oracle(cache, cbs, Q, ctx, dh)


def test_decode_many_partial_rows_and_idle_ctas():
    """more than 32 partial rows per unit (the merge's general path), and CTAs without a block"""
    cache, cbs, K, V, Q, _ = build(1, 4, 1, 128, 2300, 16, (T1, T2), {1: 0.3, 2: 0.6}, seed=3)
    for n_ctas in (40, 131, 400):
        cache.scratch = None
        check_against_oracle(cache, cbs, Q, 2300, 128, n_ctas=n_ctas)


@pytest.mark.parametrize("page", [16, 64])
def test_decode_pool_off_a_16_byte_boundary(page):
    """byte pool and positions at 4-byte alignment take word copies; the result does not change"""
    cache, cbs, K, V, Q, _ = build(2, 8, 2, 128, 500, page, (T1, T2), {1: 0.4, 2: 0.4}, seed=5)
    rope = pkg.rope_table(512, 128, device=DEV)
    want = pkg.decode_paged(Q.to(DEV), cache, rope).clone()
    flat = torch.zeros(cache.k_pages.numel() + 16, dtype=torch.uint8, device=DEV)
    flat[4:4 + cache.k_pages.numel()] = cache.k_pages
    L = cache.lists
    pos = torch.zeros(L.positions.numel() + 4, dtype=torch.int32, device=DEV)
    pos[1:1 + L.positions.numel()] = L.positions.reshape(-1)
    L.positions = pos[1:1 + L.positions.numel()].view(L.positions.shape)
    cache.k_pages = flat[4:4 + cache.k_pages.numel()]
    assert torch.equal(pkg.decode_paged(Q.to(DEV), cache, rope), want)
    pkg.check_status(cache)


@pytest.mark.parametrize("page", [16, 128])
def test_decode_honours_the_header_count(page):
    """a page whose header counts fewer tokens than its theta stream has room for"""
    cache, cbs, K, V, Q, _ = build(1, 8, 2, 128, 400, page, (T1, T2), {1: 0.4, 2: 0.5}, seed=9)
    L = cache.lists
    rope = pkg.rope_table(512, 128, device=DEV)
    fewer = torch.clamp(L.page_count - 5, min=1)
    slot = torch.arange(page, device=DEV)
    held, L.positions = L.positions, torch.where(slot[None] < fewer[:, None], L.positions, torch.full_like(L.positions, -1))
    want = pkg.decode_paged(Q.to(DEV), cache, rope).clone()
    L.positions = held
    cache.k_pages[L.ptable[:, 0].long() + 1] = fewer.to(torch.uint8)
    assert torch.equal(pkg.decode_paged(Q.to(DEV), cache, rope), want)


# the chains' kernel with one, two and four tokens per thread, staged and direct loads (16 centroids always take it, 40 up to 4700
# rows of 8 heads), and the tensor-core kernel (80 centroids)
@pytest.mark.parametrize("bits", [(4,), (5, 3), (6, 4)])
@pytest.mark.parametrize("T,Hkv,dh", [(2047, 8, 128), (4097, 8, 128), (9001, 8, 128), (6001, 8, 64)])
@pytest.mark.parametrize("dtype,shift", [(torch.float32, 0), (torch.bfloat16, 0), (torch.float32, 1)])
def test_codes_do_not_depend_on_tokens_per_thread(bits, T, Hkv, dh, dtype, shift):
    """large inputs equal the codes of 64-row slices of them (one token per thread)"""
    specs = tuple(pkg.pages.TierSpec(i + 1, 32 if b == 3 else 16, b) for i, b in enumerate(bits))
    tiers = pkg.TierSet(dh, specs)
    cb = tiers.pack_codebooks(synth.make_codebooks(Hkv, dh, specs, seed=T)).to(DEV)
    flat = torch.randn(T * Hkv * dh + 8, generator=torch.Generator(device=DEV).manual_seed(T), device=DEV).to(dtype)
    K = flat[shift:shift + T * Hkv * dh].view(T, Hkv, dh)
    got = pkg.encode_codes(K, cb, tiers)
    for t0 in (0, 64 * (T // 128), T - 64):
        part = pkg.encode_codes(K[t0:t0 + 64], cb, tiers)
        for s in range(len(specs)):
            assert torch.equal(got.r[s][:, t0:t0 + 64].view(torch.int32), part.r[s].view(torch.int32))
            assert torch.equal(got.theta[s][:, t0:t0 + 64], part.theta[s])


@pytest.mark.parametrize("dh,dtype", [(128, torch.float32), (64, torch.float16), (128, torch.bfloat16)])
def test_encode_pages_of_keys_off_a_16_byte_boundary(dh, dtype):
    Hkv, T, tiers = 3, 900, pkg.TierSet(dh, pkg.REFERENCE_TIERS)
    cb = tiers.pack_codebooks(synth.make_codebooks(Hkv, dh, pkg.REFERENCE_TIERS, seed=2)).to(DEV)
    assign = synth.make_tier_assign(1, Hkv, T, {1: 0.3, 2: 0.3, 3: 0.3}, seed=1, per_head=True).to(DEV)
    lists = pkg.build_page_lists(assign, tiers, 32)
    K = torch.randn(T, Hkv, dh, generator=torch.Generator(device=DEV).manual_seed(4), device=DEV).to(dtype)
    flat = torch.zeros(K.numel() + 8, dtype=dtype, device=DEV)
    off = flat[1:1 + K.numel()].view(K.shape)
    off.copy_(K)
    a, b = pkg.encode_pages(K, K, lists, cb, tiers), pkg.encode_pages(off, off, lists, cb, tiers)
    c = pkg.encode_pages(K, K, lists, cb, tiers, use_scratch=False)
    for other in (b, c):
        assert torch.equal(a.k_pages, other.k_pages) and torch.equal(a.v_pool, other.v_pool)


@pytest.mark.parametrize("N", [1, 31, 1025, 70001])
@pytest.mark.parametrize("d,K", [(8, 256), (16, 64), (16, 200), (32, 8), (32, 170)])
def test_kmeans_sums_and_counts(N, d, K):
    g = torch.Generator(device=DEV).manual_seed(N)
    U = torch.nn.functional.normalize(torch.randn(N, d, generator=g, device=DEV), dim=1)
    C = torch.nn.functional.normalize(torch.randn(K, d, generator=g, device=DEV), dim=1)
    assigns, best, sums, counts = pkg.kmeans_assign(U, C)
    sims = U.double() @ C.double().T
    # the winner of the fp32 chain is within its rounding (16 or 32 terms of magnitude below 1) of the exact maximum
    picked = sims.gather(1, assigns.long()[:, None])[:, 0]
    assert (sims.max(1).values - picked).max().item() <= 4 * d * 2.0 ** -24
    assert (best.double() - picked).abs().max().item() <= 2 * d * 2.0 ** -24
    assert torch.equal(counts.long(), torch.bincount(assigns.long(), minlength=K))
    want = torch.zeros(K, d, dtype=torch.float64, device=DEV).index_add_(0, assigns.long(), U.double())
    # every one of the n_k additions rounds by at most 2^-24 of sum |u|, and independently: four standard deviations.
    # (n_k * 2^-22, without the magnitudes, was passed by up to 1.5 times in a quarter of the runs with d 8, K 256; the
    # largest error seen is 9 * 2^-24 * sum |u|, of 4 * sqrt(490) = 89 allowed there; a lost row is far beyond)
    mag = torch.zeros(K, d, dtype=torch.float64, device=DEV).index_add_(0, assigns.long(), U.double().abs())
    bound = 4 * counts.double().clamp(min=1).sqrt()[:, None] * 2.0 ** -24 * mag
    assert ((sums.double() - want).abs() <= bound).all()


# both sides of the rules that choose the tensor-core search (148 SMs): centroids, rounds of the chains' blocks; batches of 128
@pytest.mark.parametrize("N,d,K", [(129, 8, 47), (129, 8, 48), (113664, 8, 48), (113665, 8, 48), (75777, 8, 225), (75777, 8, 224),
                                   (385, 16, 31), (385, 16, 32), (113665, 16, 32), (151553, 16, 32), (50000, 16, 256),
                                   (56832, 32, 8), (56833, 32, 8), (75777, 32, 8), (60000, 32, 9), (3000, 32, 17), (3000, 32, 128)])
def test_kmeans_search_rules(N, d, K):
    test_kmeans_sums_and_counts(N, d, K)


@pytest.mark.parametrize("d,K", [(8, 64), (16, 64), (32, 8), (32, 20)])
def test_kmeans_ties_and_special_points(d, K):
    """equal centroids, points between two centroids, zeros and norms out of range: the fp32 chains' first maximum"""
    g = torch.Generator(device=DEV).manual_seed(d)
    C = torch.nn.functional.normalize(torch.randn(K, d, generator=g, device=DEV), dim=1)
    C[K - 1] = C[1]
    C[3] = 0
    U = C[torch.randint(K, (999,), generator=g, device=DEV)] + C[torch.randint(K, (999,), generator=g, device=DEV)]
    U[::7] = 0
    U[1::7] *= 1e-30
    U[2::7] *= 1e15
    sims = torch.zeros(999, K, dtype=torch.float64, device=DEV)
    for i in range(d):  # an fma rounds the exact product and sum once
        sims = (U[:, i:i + 1].double() * C[:, i].double() + sims).float().double()
    assigns, best, _, counts = pkg.kmeans_assign(U, C)
    want = sims.max(1).values
    # (a 64-bit product and sum rounds a second time, in one of 2^29 cases differently from the fma)
    assert (sims.gather(1, assigns.long()[:, None])[:, 0] == want).sum() >= 997 and (best.double() == want).sum() >= 997
    assert (assigns.long() == (sims == want[:, None]).int().argmax(1)).sum() >= 997
    assert torch.equal(counts.long(), torch.bincount(assigns.long(), minlength=K))


@pytest.mark.parametrize("d,K,N", [(32, 8, 70000), (16, 40, 140000), (8, 60, 200000), (8, 256, 200000)])
def test_kmeans_kernels_agree_bit_for_bit(d, K, N):
    """the chains take these numbers of points, the tensor-core search their first 30000: ties, narrow cones, zeros and all"""
    g = torch.Generator(device=DEV).manual_seed(K)
    U = torch.randn(N, d, generator=g, device=DEV)
    U[1::4] = 1 + 0.02 * U[1::4]
    C = U[torch.randint(N, (K,), generator=g, device=DEV)].clone()
    C[::9] = C[5]
    n = U[2::4].shape[0]
    U[2::4] = C[torch.randint(K, (n,), generator=g, device=DEV)] + C[torch.randint(K, (n,), generator=g, device=DEV)]
    U[3::64] = 0
    U[7::64, 3] = float("nan")
    U[11::64, d - 1] = float("inf")
    U[4096:4160] = 0
    few, all_ = pkg.kmeans_assign(U[:30000], C), pkg.kmeans_assign(U, C)
    assert torch.equal(few[0], all_[0][:30000])
    assert torch.equal(few[1].view(torch.int32), all_[1][:30000].view(torch.int32))


# the column loop (sixteen at a time) and the whole rows, with most points open and a few columns each
@pytest.mark.parametrize("d,K", [(8, 48), (8, 200), (16, 64), (16, 100), (16, 256), (32, 8), (32, 16), (32, 64), (32, 72)])
def test_kmeans_narrow_cones(d, K):
    g = torch.Generator(device=DEV).manual_seed(d * K)
    U = 1 + 0.02 * torch.randn(1500, d, generator=g, device=DEV)
    C = 1 + 0.02 * torch.randn(K, d, generator=g, device=DEV)
    C[K // 2] = C[1]
    sims = torch.zeros(1500, K, dtype=torch.float64, device=DEV)
    for i in range(d):  # an fma rounds the exact product and sum once
        sims = (U[:, i:i + 1].double() * C[:, i].double() + sims).float().double()
    assigns, best, _, _ = pkg.kmeans_assign(U, C)
    # (a 64-bit product and sum rounds a second time, in one of 2^29 cases differently from the fma)
    assert (assigns.long() == (sims == sims.max(1).values[:, None]).int().argmax(1)).sum() >= 1498
    assert (best.double() == sims.max(1).values).sum() >= 1498


# both kernels: the chains (few centroids) and the tensor-core search
@pytest.mark.parametrize("d,K", [(8, 47), (8, 64), (16, 16), (16, 64), (16, 200), (32, 8), (32, 64), (32, 128)])
def test_kmeans_points_that_are_not_finite(d, K):
    """sums that are NaN never win; a point that has no other gets cluster 0 and a similarity of -inf"""
    g = torch.Generator(device=DEV).manual_seed(d + K)
    U = torch.randn(300, d, generator=g, device=DEV)
    C = torch.randn(K, d, generator=g, device=DEV)
    C[::3, 2] = 0  # inf * 0 is NaN: such a point has sums of both kinds
    U[::4, 1] = float("nan")
    U[1::4, 2] = float("inf")
    U[2::8, 2] = -float("inf")
    U[2::16, 5] = float("inf")
    sims = torch.zeros(300, K, dtype=torch.float64, device=DEV)
    for i in range(d):  # an fma rounds the exact product and sum once
        sims = (U[:, i:i + 1].double() * C[:, i].double() + sims).float().double()
    want = torch.where(sims.isnan(), -torch.inf, sims)
    assigns, best, _, counts = pkg.kmeans_assign(U, C)
    first = (want == want.max(1).values[:, None]).int().argmax(1)
    assert torch.equal(best.double(), want.max(1).values) and torch.equal(assigns.long(), first)
    assert torch.equal(counts.long(), torch.bincount(first, minlength=K))


# the largest codebooks of 32-dim points: eight, then seven sets of sums per CTA
@pytest.mark.parametrize("K", [172, 173, 179])
def test_kmeans_largest_codebooks(K):
    test_kmeans_sums_and_counts(5001, 32, K)


def test_kmeans_refuses_what_it_refused():
    U, C = torch.zeros(8, 32, device=DEV), torch.zeros(180, 32, device=DEV)
    with pytest.raises(pkg.SphKVError, match="K=180 x d=32"):
        pkg.kmeans_assign(U, C)


# 8-dim points: four, two and one set of sums per warp
@pytest.mark.parametrize("K", [98, 99, 190, 191])
def test_kmeans_sets_of_sums(K):
    test_kmeans_sums_and_counts(9001, 8, K)


@pytest.mark.parametrize("page", [16, 64])
def test_importance_update_with_statistics_off_an_8_byte_boundary(page):
    cache, cbs, K, V, Q, _ = build(2, 8, 2, 128, 500, page, (T1, T2), {1: 0.4, 2: 0.4}, seed=5)
    L, rope, q = cache.lists, pkg.rope_table(512, 128, device=DEV), Q.to(DEV)
    n = 2 * 8 * L.max_blocks * (page // 16) * 2
    got = []
    for shift in (0, 1):
        ml = torch.zeros(n + 1, device=DEV)[shift:shift + n].view(2, 8, L.max_blocks, page // 16, 2)
        omega = torch.full((4, L.max_blocks), 0.5, device=DEV)
        got.append((pkg.decode_paged(q, cache, rope, page_ml=ml, omega=omega).clone(), omega, ml.clone()))
    for a, b in zip(*got):
        assert torch.equal(a, b)
    pkg.check_status(cache)


# Rows are staged beside the codebook tensor while they fit: up to C_max 422, 390 and 326 for bundles in quarters, in halves and
# whole.  With such tensors an SM takes one CTA, and bundles are cut up to 0.2 and 0.4 of them per SM (`share`).
@pytest.mark.parametrize("share,sizes", [(0.1, (64, 326, 327, 422, 423, 430)), (0.3, (64, 390, 391)), (0.6, (64, 326, 327))])
def test_encode_with_a_wide_codebook_tensor(share, sizes):
    """codebook tensors of any C_max that the encoder takes"""
    Hkv, dh = 2, 128
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    T = int(128 * (share * sms - 2) / (0.8 * Hkv))
    K = torch.randn(T, Hkv, dh, generator=torch.Generator(device=DEV).manual_seed(4), device=DEV)
    assign = synth.make_tier_assign(1, Hkv, T, {1: 0.5, 2: 0.3}, seed=1, per_head=True).to(DEV)
    cbs = synth.make_codebooks(Hkv, dh, (T1, T2), seed=2)
    got = []
    for c_max in sizes:
        tiers = pkg.TierSet(dh, (T1, T2))
        tiers.C_max = c_max
        lists = pkg.build_page_lists(assign, tiers, 16)
        assert share - 0.1 < lists.bundles.shape[0] / sms < share + 0.1
        got.append(pkg.encode_pages(K, K, lists, tiers.pack_codebooks(cbs).to(DEV), tiers))
    for other in got[1:]:
        assert torch.equal(other.k_pages, got[0].k_pages) and torch.equal(other.v_pool, got[0].v_pool)
    fused = pkg.encode_pages(K, K, lists, got[0].codebooks, got[0].tiers, use_scratch=False)
    assert torch.equal(fused.k_pages, got[0].k_pages)


def test_a_refused_size_does_not_fail_the_next_call():
    Hkv, T, dh = 2, 300, 128
    K = torch.randn(T, Hkv, dh, generator=torch.Generator(device=DEV).manual_seed(4), device=DEV)
    tiers, wide = pkg.TierSet(dh, (T1, T2)), pkg.TierSet(dh, (T1, T2))
    wide.C_max = 460
    cbs = synth.make_codebooks(Hkv, dh, (T1, T2), seed=2)
    lists = pkg.build_page_lists(torch.ones(1, Hkv, T, dtype=torch.uint8, device=DEV), tiers, 16)
    want = pkg.encode_pages(K, K, lists, tiers.pack_codebooks(cbs).to(DEV), tiers)
    with pytest.raises(pkg.SphKVError, match="shared memory"):
        pkg.encode_pages(K, K, lists, wide.pack_codebooks(cbs).to(DEV), wide)
    pkg.kmeans_assign(K.view(-1, 16), K.view(-1, 16)[:8].contiguous())
    got = pkg.encode_pages(K, K, lists, tiers.pack_codebooks(cbs).to(DEV), tiers)
    assert torch.equal(got.k_pages, want.k_pages)


def test_importance_update_keeps_no_workspace_that_copies_would_share():
    """a cache and its dataclasses.replace() share their `extra`: nothing that a step writes may live there"""
    import dataclasses
    cache, cbs, K, V, Q, _ = build(1, 8, 2, 128, 400, 16, (T1, T2), {1: 0.4, 2: 0.4}, seed=5)
    rope = pkg.rope_table(512, 128, device=DEV)
    before = {k for k, v in cache.extra.items() if isinstance(v, torch.Tensor)}
    pkg.decode_paged(Q.to(DEV), cache, rope, omega=torch.zeros(2, cache.lists.max_blocks, device=DEV))
    other = dataclasses.replace(cache, scratch=None, status=None)
    pkg.decode_paged(Q.to(DEV), other, rope, omega=torch.zeros(2, cache.lists.max_blocks, device=DEV))
    assert other.extra is cache.extra and other.scratch.data_ptr() != cache.scratch.data_ptr()
    assert {k for k, v in cache.extra.items() if isinstance(v, torch.Tensor)} == before


def padded_pages(cache, lead, pad):
    """The same pages with `lead` bytes from a page to its theta stream (0: as it is) and the stream padded to `pad`."""
    L, tiers, rb = cache.lists, cache.tiers, 2 if cache.radius_fmt == 1 else 1
    old, pt = cache.k_pages.cpu(), L.ptable.cpu().tolist()
    slots, counts = L.page_slot.cpu().tolist(), L.page_count.cpu().tolist()
    pieces, table, at = [], [], 0
    for (po, to, ro), s, n in zip(pt, slots, counts):
        G = tiers.G(s)
        to2 = at + (lead or to - po)
        ro2 = to2 + -(-(ro - to) // pad) * pad
        end = ro2 + n * G * rb
        page = torch.full((-(-(end - at) // 16) * 16,), 0xEE, dtype=torch.uint8)
        page[:8 + 4 * G] = old[po:po + 8 + 4 * G]
        page[to2 - at:to2 - at + ro - to] = old[to:ro]
        page[ro2 - at:end - at] = old[ro:ro + n * G * rb]
        pieces.append(page)
        table.append((at, to2, ro2))
        at += page.numel()
    cache.k_pages = torch.cat(pieces + [torch.zeros(16, dtype=torch.uint8)]).to(DEV)
    L.ptable = torch.tensor(table, dtype=torch.int32, device=DEV)


# page, radius format, lead, padding: pointer tables whose sections do not lie back to back
@pytest.mark.parametrize("page,fmt,lead,pad", [(64, 0, 64, 16), (32, 0, 44, 1), (128, 1, 1020, 256), (16, 1, 64, 16), (16, 0, 0, 16)])
def test_decode_of_padded_sections(page, fmt, lead, pad):
    cache, cbs, K, V, Q, _ = build(2, 8, 2, 128, 500, page, (T1, T2, T3), {1: 0.3, 2: 0.3, 3: 0.2}, radius_fmt=fmt, seed=5)
    rope = pkg.rope_table(512, 128, device=DEV)
    want = pkg.decode_paged(Q.to(DEV), cache, rope).clone()
    padded_pages(cache, lead, pad)
    assert torch.equal(pkg.decode_paged(Q.to(DEV), cache, rope), want)
    pkg.check_status(cache)
