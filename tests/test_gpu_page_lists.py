"""GPU: page lists built by the library equal the array-operation construction on host tensors."""
import pytest
import torch

from util import load_pkg

pkg = load_pkg()
pytestmark = pytest.mark.gpu
TABLES = ("positions", "src_index", "page_head", "page_slot", "page_count", "ptable", "block_table", "bits_table",
          "num_blocks", "bundles")


# one token; one short of / exactly / one past a 2048-token chunk; a length that is no multiple of the vector width
@pytest.mark.parametrize("B,Hkv,T", [(1, 1, 1), (2, 3, 2047), (1, 2, 2048), (1, 5, 2049), (3, 8, 6001), (1, 600, 70)])
@pytest.mark.parametrize("page_size,radius_fmt,align", [(16, 0, 16), (128, 1, 4)])
@pytest.mark.parametrize("shuffle,extra,dtype", [(None, 0, torch.uint8), (5, 3, torch.int32), (None, 1, torch.int64)])
def test_page_lists_on_device_equal_host_construction(B, Hkv, T, page_size, radius_fmt, align, shuffle, extra, dtype):
    tiers = pkg.TierSet(128, pkg.REFERENCE_TIERS)
    assign = pkg.synth.make_tier_assign(B, Hkv, T, {1: 0.3, 2: 0.4, 3: 0.1}, seed=T, per_head=True)
    assign[0, 0, 0] = 2                      # at least one token
    if Hkv > 1:
        assign[:, -1] = 0                    # a head without any
    assign[-1, 0, T // 2:] = 1
    args = dict(radius_fmt=radius_fmt, page_align=align, shuffle_seed=shuffle, extra_blocks=extra)
    want = pkg.build_page_lists(assign, tiers, page_size, **args)
    got = pkg.build_page_lists(assign.to(dtype).to("cuda:0"), tiers, page_size, **args)
    for name in ("n_pages", "page_size", "max_blocks", "pool_bytes", "B", "Hkv"):
        assert getattr(got, name) == getattr(want, name), name
    for name in TABLES:
        assert torch.equal(getattr(got, name).cpu(), getattr(want, name)), name


# runs (heads x tiers) that one warp, several, all of a block take, and more than it keeps counts of in shared memory
@pytest.mark.parametrize("Hkv,T", [(5, 100), (11, 2049), (341, 64), (342, 64), (700, 40)])
def test_totals_of_each_call_and_tables_equal_host_construction(Hkv, T):
    tiers = pkg.TierSet(128, pkg.REFERENCE_TIERS)
    assign = pkg.synth.make_tier_assign(1, Hkv, T, {1: 0.3, 2: 0.4, 3: 0.1}, seed=T, per_head=True)
    assign[0, Hkv // 2] = 0
    want = pkg.build_page_lists(assign, tiers, 32)
    for _ in range(3):  # the totals of one call are not taken for the next one's
        got = pkg.build_page_lists(assign.to("cuda:0"), tiers, 32)
        assert (got.n_pages, got.max_blocks, got.pool_bytes) == (want.n_pages, want.max_blocks, want.pool_bytes)
        for name in TABLES:
            assert torch.equal(getattr(got, name).cpu(), getattr(want, name)), name
        assign[0, 0, : T // 2] = 0
        want = pkg.build_page_lists(assign, tiers, 32)


# 2^18 pages of 2^30 bytes and of the largest alignment, one page too many for 32-bit offsets, one that just fits
@pytest.mark.parametrize("pages,align,fits", [(1 << 18, 1 << 30, False), (1 << 18, (1 << 31) - 4, False), (2, 1 << 30, False),
                                              (1, (1 << 31) - 64, True)])
def test_pools_past_32_bit_offsets_are_refused(pages, align, fits):
    tiers = pkg.TierSet(128, pkg.REFERENCE_TIERS[:1])
    assign = torch.ones(1, 1, 16 * pages, dtype=torch.uint8, device="cuda:0")
    for _ in range(2):  # the totals' words carry an odd and an even call number
        if fits:
            assert pkg.build_page_lists(assign, tiers, 16, page_align=align).pool_bytes == align + 16
        else:
            with pytest.raises(ValueError, match="pointer-table offsets"):
                pkg.build_page_lists(assign, tiers, 16, page_align=align)


def test_page_lists_reject_empty_assignment():
    with pytest.raises(ValueError, match="no retained tokens"):
        pkg.build_page_lists(torch.zeros(1, 2, 50, dtype=torch.uint8, device="cuda:0"), pkg.TierSet(128), 16)
