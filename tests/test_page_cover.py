"""A V pool is left unfilled only for lists whose bundles are known to hold every page."""
import copy
import dataclasses

import pytest
import torch

from util import load_pkg

pkg = load_pkg()


def lists(device="cpu"):
    return pkg.build_page_lists(torch.ones(1, 2, 40, dtype=torch.uint8, device=device), pkg.TierSet(64), 16)


def narrowed(L):
    L.bundles = L.bundles[:1].contiguous()
    return L


def written(L):
    L.bundles[0, 0] = -1
    return L


def more_pages(L):
    L.n_pages += 1
    return L


CHANGES = [narrowed, written, more_pages, lambda L: dataclasses.replace(L, bundles=L.bundles[:1].contiguous()),
           lambda L: pkg.PageLists(**{k: (v.clone() if isinstance(v, torch.Tensor) else v) for k, v in L.__dict__.items()}),
           lambda L: dataclasses.replace(L, covers_pool=True)]


def test_built_lists_cover_their_pool():
    L = lists()
    assert L.encode_fills_pool()
    assert copy.copy(L).encode_fills_pool()
    assert pkg.PageLists(**L.__dict__).encode_fills_pool()
    assert pkg.shard_block_lists(L, 0, 2).encode_fills_pool()
    with torch.inference_mode():
        assert not lists().encode_fills_pool()


@pytest.mark.parametrize("change", CHANGES)
def test_changed_lists_do_not(change):
    assert not change(lists()).encode_fills_pool()


@pytest.mark.gpu
@pytest.mark.parametrize("change", CHANGES[:4])
def test_pages_outside_the_bundles_are_zero(change):
    dev = "cuda:0"
    L = change(lists(dev))
    tiers = pkg.TierSet(64)
    K = torch.randn(40, 2, 64, device=dev)
    cb = tiers.pack_codebooks(pkg.synth.make_codebooks(2, 64, pkg.REFERENCE_TIERS[:2], seed=1)).to(dev)
    held = set(L.bundles.flatten().tolist())
    if change is more_pages:  # the tables of the added page
        L.src_index = torch.cat([L.src_index, torch.full_like(L.src_index[:1], -1)])
        L.ptable = torch.cat([L.ptable, L.ptable[:1]])
        L.page_head, L.page_slot = (torch.cat([x, x[:1]]) for x in (L.page_head, L.page_slot))
    for _ in range(3):
        poison = [torch.full((n,), float("nan"), device=dev) for n in (1 << 10, 1 << 12, 1 << 14, 1 << 16)]
        del poison
        v = pkg.encode_pages(K, K, L, cb, tiers).v_pool
        for page in range(L.n_pages):
            if page not in held:
                assert (v[page] == 0).all()
        assert not v.isnan().any()
