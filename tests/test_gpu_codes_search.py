"""GPU: the code cache's tensor-core search against the fused encoder, whose searches are the fp32 fma chains themselves.
Bytes have to be equal: for keys where the sums do not decide (ties, near ties, zeros, norms out of range), for tiers with
a kernel of their own and without, in one pass and in several."""
import pytest
import torch

from util import load_pkg

pkg = load_pkg()
pytestmark = pytest.mark.gpu
DEV = "cuda:0"
REF = pkg.REFERENCE_TIERS
T = pkg.pages.TierSpec
SETS = {
    "reference": REF,
    "first two": REF[:2],
    "32 dims": (T(3, 32, 3),),
    "small and odd": (T(1, 16, 1), T(2, 32, 2), T(3, 16, 5), T(4, 32, 6)),
    "two passes": (T(1, 16, 6), T(2, 16, 5), T(3, 32, 6)),
    "four passes, rows not staged": (T(1, 16, 6), T(2, 16, 6), T(3, 16, 6), T(4, 16, 6)),
    "16 centroids": (T(1, 16, 4),),
    "40 centroids": (T(1, 16, 5), T(2, 32, 3)),
    "48 centroids": (T(1, 16, 5), T(2, 16, 4)),
    "64 centroids": (T(1, 16, 6),),
}


def keys(kind, rows, hkv, dh, cbs, g):
    k = torch.randn(rows, hkv, dh, generator=g, device=DEV)
    if kind == "near ties":  # the mean of two centroids of the first slot, and a little more of one of them
        c = cbs[0]
        G, C, gs = c.shape[1:]
        i, j = (torch.randint(C, (rows, hkv, G, 1, 1), generator=g, device=DEV) for _ in range(2))
        pick = lambda n: torch.take_along_dim(c[None].expand(rows, -1, -1, -1, -1), n, 3)[:, :, :, 0]  # noqa: E731
        eps = torch.randint(-3, 4, (rows, hkv, G, 1), generator=g, device=DEV) * 2.0 ** -23
        k = (pick(i) * (1 + eps) + pick(j)).reshape(rows, hkv, dh)
    elif kind == "worst mantissas":  # where a value is farthest from its bf16 pair; sums around 0, relative to the norms
        k = (1 + 2.0 ** -8 - 2.0 ** -16 + 2.0 ** -17) * torch.randint(0, 2, k.shape, generator=g, device=DEV).float().mul(2).sub(1)
        k *= 2.0 ** torch.randint(-2, 3, (rows, hkv, 1), generator=g, device=DEV).float()
    elif kind == "cone":  # most lanes of a warp open, each with a few columns
        k = 1 + 0.03 * k
    elif kind == "padding":  # whole warps of zeros
        k[rows // 3:] = 0
    elif kind == "zeros":
        k[::3] = 0
        k[1::3, :, ::2] = 0
    elif kind == "scales":  # from underflow to overflow of the squares
        k *= 10.0 ** torch.randint(-38, 38, (rows, 1, 1), generator=g, device=DEV).float()
    elif kind == "not finite":
        k[::5, :, 3] = float("inf")
        k[1::5, :, 17] = float("nan")
        k[2::5, :, 40] = -float("inf")
    return k


@pytest.mark.parametrize("kind", ["random", "near ties", "worst mantissas", "cone", "padding", "zeros", "scales", "not finite"])
@pytest.mark.parametrize("tiers", SETS)
@pytest.mark.parametrize("dh,rows,dtype", [(128, 129, torch.float32), (64, 300, torch.float32), (128, 127, torch.bfloat16),
                                           (64, 128, torch.float16)])
def test_codes_equal_the_chains(kind, tiers, dh, rows, dtype):
    specs, hkv = SETS[tiers], 2
    g = torch.Generator(device=DEV).manual_seed(rows + dh)
    cbs = []
    for t in specs:
        c = torch.randn(hkv, dh // t.g, t.codebook_size, t.g, generator=g, device=DEV)
        if kind == "cone":
            c = 1 + 0.03 * c
        cbs.append(c / c.norm(dim=-1, keepdim=True))
    if kind == "worst mantissas":
        for c in cbs:
            c[:] = (1 + 2.0 ** -8 - 2.0 ** -16 + 2.0 ** -17) * torch.randint(0, 2, c.shape, generator=g, device=DEV).float().mul(2).sub(1)
            c[:, :, 1::2] = -c[:, :, ::2] * (1 + 2.0 ** -7 * torch.randint(0, 2, c[:, :, ::2].shape, generator=g, device=DEV))
    cbs[0][:, 0, -1] = cbs[0][:, 0, 0]  # two equal centroids, and one of zeros
    cbs[0][:, 1, 0] = 0
    if kind == "padding":
        cbs[-1][:, :, 0, 0] = float("inf")  # its sum with zeros is NaN: the next centroid is the first maximum
    ts = pkg.TierSet(dh, specs)
    cb = ts.pack_codebooks(cbs)
    K = keys(kind, rows, hkv, dh, cbs, g).to(dtype)
    codes = pkg.encode_codes(K, cb, ts)
    for t in specs:
        lists = pkg.build_page_lists(torch.full((1, hkv, rows), t.tier_id, dtype=torch.uint8, device=DEV), ts, 16)
        want = pkg.encode_pages(K, None, lists, cb, ts, use_scratch=False)
        got = pkg.pages_from_codes(codes, None, lists, cb)
        assert torch.equal(got.k_pages, want.k_pages)


def compare_with_chains(tiers, K, dh, hkv, seed):
    """every code of K against the fused encoder's pages, every radius against the fma chain's root"""
    specs = SETS[tiers]
    ts = pkg.TierSet(dh, specs)
    cb = ts.pack_codebooks(pkg.synth.make_codebooks(hkv, dh, specs, seed=seed)).to(DEV)
    codes = pkg.encode_codes(K, cb, ts)
    rows = K.shape[0]
    for s, t in enumerate(specs):
        lists = pkg.build_page_lists(torch.full((1, hkv, rows), t.tier_id, dtype=torch.uint8, device=DEV), ts, 64)
        want = pkg.encode_pages(K, None, lists, cb, ts, use_scratch=False)
        assert torch.equal(pkg.pages_from_codes(codes, None, lists, cb).k_pages, want.k_pages)
        k = K.double().reshape(rows, hkv, dh // t.g, t.g).transpose(0, 1)
        n = torch.zeros(k.shape[:3], dtype=torch.float64, device=DEV)
        for d in range(t.g):  # an fma rounds the exact product and sum once
            n = (k[..., d] * k[..., d] + n).float().double()
        # (a 64-bit product and sum rounds a second time, in one of 2^29 cases differently from the fma)
        assert (codes.r[s].view(torch.int32) != n.float().sqrt().view(torch.int32)).sum() <= 2


# more than 148 blocks of 128 rows: blocks in a row, blocks of two heads in one CTA, a last block that is not full
@pytest.mark.parametrize("tiers", SETS)
@pytest.mark.parametrize("dh,dtype,shift", [(128, torch.float32, 0), (64, torch.bfloat16, 0), (128, torch.float16, 1), (64, torch.float32, 1)])
def test_long_inputs_cross_blocks_and_heads(tiers, dh, dtype, shift):
    rows, hkv = 9001, 8
    g = torch.Generator(device=DEV).manual_seed(dh + shift)
    flat = torch.randn(rows * hkv * dh + 8, generator=g, device=DEV).to(dtype)
    compare_with_chains(tiers, flat[shift:shift + rows * hkv * dh].view(rows, hkv, dh), dh, hkv, seed=rows)


# both sides of the lines of the dispatch (148 blocks): one round of the chains with one, two, four tokens per thread
@pytest.mark.parametrize("tiers,edge", [("64 centroids", 18 * 64), ("48 centroids", 18 * 128), ("40 centroids", 18 * 256), ("reference", 18 * 64)])
@pytest.mark.parametrize("past", [0, 1])
@pytest.mark.parametrize("shift", [0, 1])
def test_lines_of_the_dispatch(tiers, edge, past, shift):
    rows, hkv, dh = edge + past, 8, 128
    g = torch.Generator(device=DEV).manual_seed(edge)
    flat = torch.randn(rows * hkv * dh + 8, generator=g, device=DEV)
    compare_with_chains(tiers, flat[shift:shift + rows * hkv * dh].view(rows, hkv, dh), dh, hkv, seed=edge)


def test_padding_costs_no_more_than_keys():
    """whole warps of undecided searches: 11 times the time of random keys when every lane walked all centroids"""
    g = torch.Generator(device=DEV).manual_seed(1)
    ts = pkg.TierSet(128, REF)
    cb = ts.pack_codebooks(pkg.synth.make_codebooks(8, 128, REF, seed=2)).to(DEV)
    K = torch.randn(16384, 8, 128, generator=g, device=DEV)

    def us(k):
        events = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        times = []
        for _ in range(8):
            events[0].record()
            pkg.encode_codes(k, cb, ts)
            events[1].record()
            events[1].synchronize()
            times.append(events[0].elapsed_time(events[1]))
        return min(times)
    assert us(torch.zeros_like(K)) <= 4 * us(K)
