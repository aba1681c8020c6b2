"""A cache that has been decoded is still plain data: it can be copied, replaced, pickled and saved, and a decode of the
copy works on the copy's tensors."""
import copy
import dataclasses
import io
import pickle

import pytest
import torch

from util import load_pkg

pkg = load_pkg()
ops = __import__("importlib").import_module("spherical-kv_b200.ops")


def decoded_cache():
    """tensors on the host: what the parameter struct is made from; nothing is launched"""
    tiers = pkg.TierSet(64)
    lists = pkg.build_page_lists(torch.ones(1, 2, 40, dtype=torch.uint8), tiers, 16)
    cache = pkg.PagedCache(tiers=tiers, lists=lists, codebooks=torch.zeros(2, 2, 4, 64, 16),
                           k_pages=torch.zeros(lists.pool_bytes, dtype=torch.uint8),
                           v_pool=torch.zeros(lists.n_pages, 16, 64, dtype=torch.float16))
    template(cache)
    return cache


def template(cache, Hq=8, n_ctas=4):
    return ops._decode_template(pkg._lib.load(), cache, 1, Hq, 64, n_ctas, torch.device("cpu"))


def saved(cache):
    f = io.BytesIO()
    torch.save(cache, f)
    f.seek(0)
    return torch.load(f, weights_only=False)


@pytest.mark.parametrize("make", [copy.copy, copy.deepcopy, dataclasses.replace, lambda c: pickle.loads(pickle.dumps(c)), saved,
                                  lambda c: pkg.PagedCache(**c.__dict__)])
def test_copies_of_a_decoded_cache(make):
    cache = decoded_cache()
    other = make(cache)
    p = template(other)
    assert (p.k_pages, p.v_pool, p.status) == (other.k_pages.data_ptr(), other.v_pool.data_ptr(), other.status.data_ptr())
    assert (p.ptable, p.scratch) == (other.lists.ptable.data_ptr(), other.scratch.data_ptr())
    q = template(cache)
    assert (q.k_pages, q.ptable) == (cache.k_pages.data_ptr(), cache.lists.ptable.data_ptr())
    dataclasses.asdict(other)


def test_the_kept_struct_follows_what_it_was_made_from():
    cache = decoded_cache()
    assert bytes(template(cache)) == bytes(template(cache))
    cache.tiers = pkg.TierSet(64, pkg.REFERENCE_TIERS)      # another set, whatever its id
    assert template(cache).tiers.n_slots == 3
    cache.tiers.C_max = 80
    assert template(cache).tiers.C_max == 80
    cache.lists.positions = cache.lists.positions.clone()
    assert template(cache).positions == cache.lists.positions.data_ptr()
    cache.radius_fmt = pkg.RADIUS_F16
    assert template(cache).radius_fmt == pkg.RADIUS_F16
    assert template(cache, Hq=4).Hq == 4
    cache.tiers = pkg.TierSet(128)
    with pytest.raises(AssertionError):
        template(cache)


def test_a_tier_set_saved_without_the_struct_loads():
    tiers = pkg.TierSet(64)
    tiers.to_c()
    assert "_c" not in tiers.__getstate__()
    old = pkg.TierSet.__new__(pkg.TierSet)
    old.__dict__.update(tiers.__getstate__())
    assert bytes(old.to_c()) == bytes(tiers.to_c())
