"""Where a product of blocks runs (no GPU needed).  The solver's own FP64
kernels are for small products only; the integer tensor cores are used where
the caller allows them, which is the FP64 phase of a mixed solve, and for no
rotation; every other product is a library call."""
import ctypes as C

import pytest

import halfb200

BLOCK, INTEGER, LIBRARY = 1, 2, 3


@pytest.fixture(scope="module")
def lib():
    return C.CDLL(halfb200.library_path())


@pytest.mark.parametrize("n,m", [(725, 16), (3407, 64), (3407, 640), (11023, 200), (38089, 600)])
def test_only_small_products_take_the_block_kernels(n, m, lib):
    for np_ in range(4, m + 1, 4):
        for rows, cols in ((m, np_), (np_, np_), (m - np_ + 4, np_), (2 * np_, 2 * np_)):
            small = n * max(rows, cols) ** 2 < 2.0e8
            for route in (lib.hb_diag_gram_route, lib.hb_diag_update_route):
                assert (route(n, rows, cols, 0) == BLOCK) == small
                assert (route(n, rows, cols, 1) == BLOCK) == small


@pytest.mark.parametrize("n,m", [(3407, 640), (38089, 600), (38089, 1200)])
def test_integer_products_only_where_allowed(n, m, lib):
    assert lib.hb_diag_gram_route(n, m, m, 0) == LIBRARY and lib.hb_diag_update_route(n, m, m, 0) == LIBRARY
    assert lib.hb_diag_gram_route(38089, 600, 600, 1) == INTEGER
    assert lib.hb_diag_gram_route(70001, m, m, 1) == LIBRARY   # beyond the exact int32 sums
