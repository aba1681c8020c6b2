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
