"""The FP64 block products of the acc iteration, each route called directly:
the block kernels (1), the integer tensor cores (2) and ZGEMM (3), against
sums in 80-bit arithmetic.  Operands in one and two buffers, one and several
slices of K, remainders of every tile, upper triangles, beta, and values graded
over ten decades along K and over twenty across columns, as the iteration's
[X P] are.

Bounds, from the methods.  Routes 1 and 3 accumulate in FP64: each of the K
complex multiply-adds rounds a partial sum four times, so the error is below
4 K 2^-53 sum_k |a_k| |b_k|.  Route 2 holds a row of norm |a| in units of at
most 2^-61 |a|: half a unit per real part is 2^-61.5 |a| per element, and by
Cauchy-Schwarz both operands' roundings together change a sum by at most
2 sqrt(K) 2^-61.5 |a| |b|; putting the residues together adds 2^-60 |a| |b|.
All end with a few roundings of the result and of beta C."""
import ctypes as C

import numpy as np
import pytest

import halfb200
from conftest import rng

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _call(kind, route, n, a, b, c, alpha=1.0, beta=0.0, upper=False, c2=None):
    """a, b: one or two host blocks; c (and c2): host outputs, updated."""
    import torch
    lib = C.CDLL(halfb200.library_path())
    dev = [torch.from_numpy(np.ascontiguousarray(x.T)).cuda() for x in (*a, *b)]   # column-major
    da, db = dev[:len(a)], dev[len(a):]
    dc = torch.from_numpy(np.ascontiguousarray(c.T)).cuda()
    dc2 = torch.from_numpy(np.ascontiguousarray(c2.T)).cuda() if c2 is not None else None
    err = C.create_string_buffer(512)

    def ptr(x, i):
        return C.c_void_p(x[i].data_ptr()) if len(x) > i else None
    torch.cuda.synchronize()
    st = lib.hb_diag_block_product(C.c_char(kind.encode()), route, int(upper), n, a[0].shape[1],
                                   a[1].shape[1] if len(a) > 1 else 0, ptr(da, 0), ptr(da, 1), b[0].shape[1],
                                   b[1].shape[1] if len(b) > 1 else 0, ptr(db, 0), ptr(db, 1), C.c_double(alpha),
                                   C.c_double(beta), C.c_void_p(dc.data_ptr()),
                                   C.c_void_p(dc2.data_ptr()) if dc2 is not None else None, c.shape[0], err, 512)
    assert st == 0, err.value
    out = dc.cpu().numpy().T
    return (out, dc2.cpu().numpy().T) if c2 is not None else out


def _block(r, n, cols, decades, spread):
    x = r.normal(size=(n, cols)) + 1j * r.normal(size=(n, cols))
    x *= (10.0 ** (-decades * r.permutation(n) / max(1, n - 1)))[:, None]
    return x * 10.0 ** r.uniform(-spread, 0, size=cols)


def _exact(a, b):   # a^H b
    return a.conj().T.astype(np.clongdouble) @ b.astype(np.clongdouble)


def _bound(route, a, b, k):
    """Per element of a^H b, without the final roundings."""
    if route == 2:
        return (2 * np.sqrt(k) * 2 ** -61.5 + 2.0 ** -60) * np.outer(np.linalg.norm(a, axis=0), np.linalg.norm(b, axis=0))
    return 4 * k * U * (np.abs(a).T @ np.abs(b))


def _check(got, ref, bound, extra=0.0):
    err = np.abs(got.astype(np.clongdouble) - ref).astype(np.float64)
    assert np.all(err <= bound + 8 * U * (np.abs(ref).astype(np.float64) + extra))


@pytest.mark.parametrize("decades,spread", [(0, 0), (10, 20)])
@pytest.mark.parametrize("n,a,b,upper", [
    (1, (1,), (1,), False), (129, (5,), (3,), False), (700, (33, 4), (33, 4), True), (700, (161,), (9,), False),
    (1283, (130, 31), (100, 61), False), (3407, (97, 64), (97, 64), True), (9001, (17,), (29,), False)])
@pytest.mark.parametrize("route", [1, 2, 3])
def test_gram(route, n, a, b, upper, decades, spread):
    r = rng(n + sum(a))
    A = [_block(r, n, c, decades, spread) for c in a]
    B = [_block(r, n, c, decades, spread) for c in b]
    x, y = np.hstack(A), np.hstack(B)
    got = _call("G", route, n, A, B, np.zeros((sum(a), sum(b)), dtype=complex), upper=upper)
    ref, bound = _exact(x, y), _bound(route, x, y, n)
    if upper:
        keep = np.triu(np.ones(ref.shape, dtype=bool))
        got, ref = np.where(keep, got, 0), np.where(keep, ref, 0)
    _check(got, ref, bound)


@pytest.mark.parametrize("decades,spread", [(0, 0), (10, 3)])
@pytest.mark.parametrize("n,a,cols", [(1, (1,), 1), (129, (5,), 3), (3407, (17, 18), 161), (700, (401, 200), 33)])
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-1.0, 1.0)])
@pytest.mark.parametrize("route", [1, 2, 3])
def test_update(route, alpha, beta, n, a, cols, decades, spread):
    r = rng(n + cols)
    Z = [_block(r, n, c, decades, spread) for c in a]
    k = sum(a)
    y = _block(r, k, cols, decades, spread)
    c = r.normal(size=(n, cols)) + 1j * r.normal(size=(n, cols))
    z = np.hstack(Z)
    got = _call("U", route, n, Z, [y], c, alpha, beta)
    ref = alpha * _exact(z.conj().T, y) + beta * c.astype(np.clongdouble)
    _check(got, ref, _bound(route, z.T, y, k), beta * np.abs(c))


def test_projector_product():
    """Two right-hand buffers and two outputs, added to."""
    r = rng(3)
    n, k, nb = 1403, 150, 87
    a = _block(r, n, k, 3, 0)
    y = [_block(r, k, nb, 3, 5) for _ in range(2)]
    c = [r.normal(size=(n, nb)) + 1j * r.normal(size=(n, nb)) for _ in range(2)]
    got = _call("P", 2, n, [a], y, c[0], c2=c[1])
    for g, yy, cc in zip(got, y, c):
        _check(g, _exact(a.conj().T, yy) + cc.astype(np.clongdouble), _bound(2, a.T, yy, k), np.abs(cc))


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_columns_keep_to_themselves(bad):
    r = rng(4)
    a, b = _block(r, 900, 40, 0, 0), _block(r, 900, 30, 0, 0)
    clean = _call("G", 2, 900, [a], [b], np.zeros((40, 30), dtype=complex))
    b[5, 7] = bad
    got = _call("G", 2, 900, [a], [b], np.zeros((40, 30), dtype=complex))
    assert not np.isfinite(got[:, 7]).any()
    assert np.array_equal(np.delete(got, 7, axis=1), np.delete(clean, 7, axis=1))
