"""Rayleigh-Ritz pencils where the device cannot hold the library's cluster or
grid-wide launches (as in a process that may use part of the SMs only): the
orders concerned go to cuSOLVER and the solves converge to the same
eigenvalues.  The limit is set on the host; without one, this device holds
clusters of 16 and grid-wide launches."""
import ctypes as C

import numpy as np
import pytest

import halfb200

pytestmark = pytest.mark.gpu

K = (0.125, 0.25, 0.375)


@pytest.fixture(scope="module")
def dense(hfo2):
    w, ch, po = hfo2
    with halfb200.Context(ch, po, w.encut, xc=w.xc, solver="vasp") as ctx:
        return ctx.solve(K, 240)[0]


@pytest.fixture
def limit():
    lib = C.CDLL(halfb200.library_path())
    yield lib.hb_diag_limit_pencils
    lib.hb_diag_limit_pencils(16, 1)


def test_this_device_holds_them(limit):
    assert limit(16, 1) == 16 + 256


@pytest.mark.parametrize("cluster,grid", [(16, 0), (8, 1), (4, 0), (0, 0)])
@pytest.mark.parametrize("bands,precision", [(4, "fp64"), (12, "fp64_guarded"), (33, "mixed"), (70, "fp64_guarded"),
                                             (96, "fp64"), (120, "mixed"), (240, "fp64_guarded")])
def test_limited_launches_match_dense(bands, precision, cluster, grid, limit, hfo2, dense):
    w, ch, po = hfo2
    assert limit(cluster, grid) == cluster + 256 * grid
    with halfb200.Context(ch, po, w.encut, xc=w.xc, solver="acc") as ctx:
        ctx.set_acc(tol=2e-5, max_iterations=3000, precision=precision)
        eig = ctx.solve(K, bands)[0]
        assert ctx.info()["converged"] == 1
    assert np.abs(eig - dense[:bands]).max() <= 1e-8
