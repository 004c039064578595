"""Pencils of the plain FP64 iteration above order 164: an overlap that is not
positive definite is reported, as zhegvd, which served them, does; a positive
definite one is not, and its eigenvalues agree with a Cholesky reduction in
numpy.  The floored variant (the smaller orders and the guard-band modes)
accepts both.  Orders on either side of the cluster kernels' sizes and in the
grid-wide range."""
import ctypes as C
import time

import numpy as np
import pytest

import halfb200
from conftest import rng

pytestmark = pytest.mark.gpu


def _pencil(n, lowest, seed):
    r = rng(seed)
    q, _ = np.linalg.qr(r.normal(size=(n, n)) + 1j * r.normal(size=(n, n)))
    lam = r.uniform(0.5, 2.0, size=n)
    lam[n // 2] = lowest
    b = (q * lam) @ q.conj().T
    a = r.normal(size=(n, n)) + 1j * r.normal(size=(n, n))
    return (a + a.conj().T) / 2, (b + b.conj().T) / 2


def _solve(a, b, strict):
    import torch
    lib = C.CDLL(halfb200.library_path())
    n = len(a)
    da, db = (torch.from_numpy(np.ascontiguousarray(x.T)).cuda() for x in (a, b))
    w = torch.zeros(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    st, chol, err = C.c_int(-1), C.c_int(-1), C.create_string_buffer(256)
    rc = lib.hb_diag_pencil(n, n, int(strict), C.c_void_p(da.data_ptr()), C.c_void_p(db.data_ptr()),
                            C.c_void_p(w.data_ptr()), C.byref(st), C.byref(chol), err, 256)
    assert rc == 0, err.value
    return w.cpu().numpy(), st.value, chol.value


@pytest.fixture(scope="module", autouse=True)
def started():
    """torch, the CUDA context and the kernels are loaded before anything is timed."""
    _solve(*_pencil(40, 0.5, 0), False)
    _solve(*_pencil(440, 0.5, 0), False)


@pytest.mark.parametrize("n", [165, 177, 300, 432, 500])
def test_indefinite_overlap_is_reported(n):
    a, b = _pencil(n, -0.05, n)
    t = time.monotonic()
    assert _solve(a, b, True)[2] != 0
    assert time.monotonic() - t < 5.0   # no eigenvectors of a pencil that has failed


@pytest.mark.parametrize("n", [40, 170, 432, 500])
@pytest.mark.parametrize("where", ["a", "b"])
def test_pencil_with_nan_is_reported_soon(where, n):
    """Eigenvalues that are not numbers form one cluster, which a single thread
    would orthogonalise (25 s at order 500): it stops at the first."""
    a, b = _pencil(n, 0.5, n)
    (a if where == "a" else b)[n // 3, n // 2] = np.nan
    t = time.monotonic()
    _, st, chol = _solve(a, b, False)
    assert st != 0 or chol != 0
    assert time.monotonic() - t < 5.0


def test_floored_variant_accepts_it():
    a, b = _pencil(165, -0.05, 165)
    assert _solve(a, b, False)[2] == 0


@pytest.mark.parametrize("n", [165, 177, 300, 432, 500])
@pytest.mark.parametrize("strict", [True, False])
def test_definite_overlap(n, strict):
    a, b = _pencil(n, 1e-3, n)
    w, st, chol = _solve(a, b, strict)
    assert st == 0 and chol == 0
    li = np.linalg.inv(np.linalg.cholesky(b))
    ref = np.linalg.eigvalsh(li @ a @ li.conj().T)
    # both reductions are backward stable: n eps ||A|| ||B^-1|| with margin 4
    assert np.abs(w - ref).max() <= 4 * n * 2.0 ** -52 * np.linalg.norm(a, 2) / 1e-3
