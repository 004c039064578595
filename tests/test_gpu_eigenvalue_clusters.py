"""Pencils with clusters of (nearly) equal eigenvalues, as crystals of high
symmetry have: pairs, multiplicities up to a hundred and more members than a
thread block's slots, the identity, and a spread of 1e-9 inside a cluster.
Residuals and S-orthogonality of the vectors, bounded by the solver's backward
error (n eps ||A||, margin 8), and a second per solve: a cluster is shared by
a warp (one thread took 16 s for the identity of order 432)."""
import ctypes as C
import time

import numpy as np
import pytest

import halfb200
from conftest import rng

pytestmark = pytest.mark.gpu


def _solve(a, b):
    import torch
    lib = C.CDLL(halfb200.library_path())
    n = len(a)
    da, db = (torch.from_numpy(np.ascontiguousarray(x.T)).cuda() for x in (a, b))
    w = torch.zeros(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    st, chol, err = C.c_int(-1), C.c_int(-1), C.create_string_buffer(256)
    t = time.monotonic()
    rc = lib.hb_diag_pencil(n, n, 0, C.c_void_p(da.data_ptr()), C.c_void_p(db.data_ptr()), C.c_void_p(w.data_ptr()),
                            C.byref(st), C.byref(chol), err, 256)
    t = time.monotonic() - t
    assert rc == 0 and st.value == 0 and chol.value == 0, err.value
    return w.cpu().numpy(), da.cpu().numpy().T, t


@pytest.fixture(scope="module", autouse=True)
def started():
    for n in (40, 440):   # torch, the CUDA context and the kernels are loaded before anything is timed
        _solve(np.diag(np.arange(n) + 0j), np.eye(n, dtype=complex))


def _values(kind, n, r):
    if kind == "identity":
        return np.ones(n)
    if kind == "pairs":
        return np.repeat(r.uniform(-5, 5, size=(n + 1) // 2), 2)[:n]
    if kind == "levels":   # multiplicities 1, 2, 3, 6, 8, 24, 48, 100 in turn
        out = []
        for i, m in enumerate([1, 2, 3, 6, 8, 24, 48, 100] * n):
            out += [float(i)] * m
            if len(out) >= n:
                break
        return np.array(out[:n])
    if kind == "close":   # tens of values 1e-6 apart, three times what makes a cluster
        return np.sort(np.repeat(np.linspace(-4.0, 4.0, (n + 9) // 10), 10)[:n]) + 1e-6 * (np.arange(n) % 10)
    return np.sort(np.repeat(r.uniform(-5, 5, size=(n + 29) // 30), 30)[:n]) + 1e-9 * r.normal(size=n)   # "spread"


@pytest.mark.parametrize("kind", ["identity", "pairs", "levels", "spread", "close"])
@pytest.mark.parametrize("n", [7, 33, 100, 165, 300, 432, 434, 700])
def test_clusters(n, kind):
    r = rng(n)
    q, _ = np.linalg.qr(r.normal(size=(n, n)) + 1j * r.normal(size=(n, n)))
    lam = _values(kind, n, r)
    a = (q * lam) @ q.conj().T
    s = 10.0 ** r.uniform(-3, 0, size=n)            # the overlap of badly scaled vectors
    a, b = (a + a.conj().T) / 2 * np.outer(s, s), np.diag(s * s).astype(complex)
    w, y, t = _solve(a, b)
    y = y * s[:, None]                              # back to the pencil (Q lam Q^H, 1)
    a = a / np.outer(s, s)
    bound = 8 * n * 2.0 ** -52 * np.abs(lam).max()
    assert np.abs(w - np.sort(lam)).max() <= bound
    orth = np.abs(y.conj().T @ y - np.eye(n)).max()
    # up to order 164 what inverse iteration leaves between clusters, above it rounding
    assert orth <= (4e-9 if n <= 164 else 8 * n * 2.0 ** -52)
    assert np.linalg.norm(a @ y - y * w[None, :], axis=0).max() <= 4 * bound
    assert t < 1.0
