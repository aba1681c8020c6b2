"""The page tables' allocation: shapes, addresses and room of every table, no two of them overlapping."""
import ctypes as C

import pytest
import torch

from util import load_pkg

pkg = load_pkg()


@pytest.mark.parametrize("P,N,U,mb,nb", [(1, 16, 1, 1, 1), (63, 128, 3, 22, 63), (64, 16, 64, 1, 8), (65, 32, 600, 7, 33)])
def test_tables_lie_side_by_side_on_256_byte_boundaries(P, N, U, mb, nb):
    ptrs = (C.c_void_p * 10)()
    tables = pkg._lib.host_tables().make(C.addressof(ptrs), -1, P, N, U, mb, nb)
    shapes = [(P, N), (P, N), (P,), (P,), (P,), (P, 3), (U, mb), (U, mb), (U,), (nb, 8)]
    assert [tuple(t.shape) for t in tables] == shapes
    assert all(t.dtype == torch.int32 and t.is_contiguous() for t in tables)
    assert [t.data_ptr() for t in tables] == list(ptrs)
    assert all((t.data_ptr() - tables[0].data_ptr()) % 256 == 0 for t in tables)
    for i, t in enumerate(tables):
        t.fill_(i)
    assert all(bool((t == i).all()) for i, t in enumerate(tables))


def test_the_module_is_named_after_what_it_was_built_against(monkeypatch):
    import sys
    path = pkg._lib.host_path()
    assert sys.implementation.cache_tag in path and torch.__version__ in path
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    monkeypatch.setattr(pkg._lib, "_host", None)
    assert pkg._lib.host_path() != path
    with pytest.raises(pkg.SphKVError, match="is missing"):
        pkg._lib.host_tables()


@pytest.mark.parametrize("bf16,zero_v,scratch", [(1, 1, 64), (0, 1, 0), (1, 0, 1), (0, 0, 4096)])
def test_pools_and_their_addresses(bf16, zero_v, scratch):
    k, v, s, *at = pkg._lib.host_tables().pools(-1, 1000, 5, 32, 64, bf16, zero_v, scratch)
    assert (k.dtype, tuple(k.shape)) == (torch.uint8, (1000,)) and not bool(k.any())
    assert (v.dtype, tuple(v.shape)) == (torch.bfloat16 if bf16 else torch.float16, (5, 32, 64))
    assert not zero_v or not bool(v.any())
    assert (s is None) if not scratch else (s.dtype, s.numel()) == (torch.uint8, scratch)
    assert at == [k.data_ptr(), v.data_ptr(), 0 if s is None else s.data_ptr()]
    assert not (k.requires_grad or v.requires_grad)


# with the module and without it
@pytest.mark.parametrize("built", [True, False])
@pytest.mark.parametrize("v_dtype,scratch", [(torch.bfloat16, 64), (torch.float16, 0)])
def test_pools_of_host_built_lists_do_without_the_module(monkeypatch, built, v_dtype, scratch):
    tiers = pkg.TierSet(128)
    lists = pkg.build_page_lists(torch.ones(1, 2, 40, dtype=torch.uint8), tiers, 16)
    if not built:
        monkeypatch.setattr(torch, "__version__", "0.0.1")
        monkeypatch.setattr(pkg._lib, "_host", None)
    new_cache = pkg.encode_pages.__globals__["_new_cache"]
    cache, at = new_cache(lists, tiers, torch.zeros(1), 128, False, v_dtype, 0, torch.device("cpu"), scratch)
    assert cache.k_pages.numel() == lists.pool_bytes and not bool(cache.k_pages.any())
    assert (cache.v_pool.dtype, tuple(cache.v_pool.shape)) == (v_dtype, (lists.n_pages, 16, 128)) and not bool(cache.v_pool.any())
    s = cache.extra.get("encode_scratch")
    assert (s is None) if not scratch else s.numel() == scratch
    assert list(at) == [cache.k_pages.data_ptr(), cache.v_pool.data_ptr(), 0 if s is None else s.data_ptr()]


# A zeroed pool takes its time, at an allocation or a full launch queue more of it: other threads go on meanwhile.
def test_other_threads_run_while_pools_are_made():
    import threading
    import time
    pools = pkg._lib.host_tables().pools
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.wait(0.001):
            ticks.append(time.monotonic())

    thread = threading.Thread(target=tick)
    thread.start()
    try:
        begin = time.monotonic()
        made = pools(-1, 1 << 30, 1, 16, 64, 1, 1, 0)
        end = time.monotonic()
    finally:
        stop.set()
        thread.join()
    margin = (end - begin) / 8
    assert any(begin + margin < t < end - margin for t in ticks), (end - begin, len(ticks), made[0].shape)


def test_packed_parameters_are_the_struct_field_by_field():
    cls, C4 = pkg._lib.EncodeParams, pkg._lib.MAX_TIER_SLOTS
    assert cls._packer.size == C.sizeof(cls)
    tiers = pkg.TierSet(128, pkg.REFERENCE_TIERS).to_c()
    names = [n for n, _ in cls._fields_ if n not in ("code_r", "code_theta", "tiers")]
    v = dict(zip(names, range(1, 1 + len(names))))
    codes = tuple(range(100, 100 + 2 * C4))
    strides = tuple(v[n] for n in names[12:16])
    p = cls.packed(*[v[n] for n in names[:12]], strides, codes, *[v[n] for n in names[16:]], bytes(tiers))
    assert all(getattr(p, n) == v[n] for n in names)
    assert tuple(p.code_r) + tuple(p.code_theta) == codes and bytes(p.tiers) == bytes(tiers)
