"""The force adjoint over band counts at the edges of its band tiles (32 and
64) and of the contraction's 32-band tiles, for atoms of up to 8 and of 18
channels, with several plane-wave slices (both cells are small enough to need
them), and staged host copies with padded leading dimensions.  Against the
oracle's restatement on random states: sums of products of order one over
N_pw terms in another order, 1e-11 of the largest component."""
import ctypes as C

import numpy as np
import pytest

import halfb200
from conftest import rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["si2", "hfo2"])
@pytest.mark.parametrize("nb", [1, 31, 33, 64, 65, 129])
def test_nonlocal_forces_over_band_counts(name, nb, si2, hfo2, oracle_system):
    from oracle import hamiltonian as H
    from oracle.forces import nonlocal_forces
    files = {"si2": si2, "hfo2": hfo2}[name]
    sysm = oracle_system(name, files, with_gradient=True)
    k = (0.125, 0.25, -0.375)
    op = H.prepare(sysm, k)
    r = rng(nb)
    v = (r.normal(size=(op.basis.npw, nb)) + 1j * r.normal(size=(op.basis.npw, nb))) / np.sqrt(2.0 * op.basis.npw)
    eps = np.sort(r.uniform(-5.0, 5.0, size=nb))
    occ = r.uniform(0.0, 2.0, size=nb)
    occ[nb // 2] = 0.0 if nb > 1 else occ[0]
    ref = nonlocal_forces(op.basis, op.species, sysm.dij_atoms, sysm.ddij_atoms, eps, occ, 0.7, v)
    w, ch, po = files
    with halfb200.Context(ch, po, w.encut, xc=w.xc, solver="acc") as ctx:
        f = ctx.nonlocal_forces(k, v, eps, occ, 0.7)
    assert np.abs(f - ref).max() <= 1e-11 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("nb,pad", [(1, 0), (40, 0), (40, 3), (333, 0), (333, 1)])
def test_staged_copies_keep_columns_and_padding(nb, pad, hfo2):
    """Blocks below and above the staging threshold, contiguous and with a
    padded leading dimension: the same H psi and S psi (to rounding: the projector
    products of another band count may sum in another order), and the
    rows beyond the basis untouched."""
    w, ch, po = hfo2
    k = (0.25, 0.0, 0.5)
    with halfb200.Context(ch, po, w.encut, xc=w.xc, solver="acc") as ctx:
        n = ctx.npw(k)
        r = rng(3)
        x = np.full((nb, n + pad), 7.0 + 1j)
        x[:, :n] = r.normal(size=(nb, n)) + 1j * r.normal(size=(nb, n))
        h = np.full((nb, n + pad), -3.0 + 2j)
        s = h.copy()
        kk = np.array(k)
        err = C.create_string_buffer(512)
        st = ctx.lib.half_apply_hs(ctx.handle, kk.ctypes.data_as(C.c_void_p), nb, n + pad,
                                   x.ctypes.data_as(C.c_void_p), h.ctypes.data_as(C.c_void_p),
                                   s.ctypes.data_as(C.c_void_p), err, 512)
        assert st == 0, err.value
        hr = np.empty((nb, n), dtype=complex)
        sr = np.empty((nb, n), dtype=complex)
        for b0 in range(0, nb, 16):   # 16 bands are below the threshold
            a, b = ctx.apply_hs(k, x[b0:b0 + 16, :n].T)
            hr[b0:b0 + 16], sr[b0:b0 + 16] = a.T, b.T
    assert np.all(h[:, n:] == -3.0 + 2j) and np.all(s[:, n:] == -3.0 + 2j)
    assert np.abs(h[:, :n] - hr).max() <= 1e-12 * np.abs(hr).max()
    assert np.abs(s[:, :n] - sr).max() <= 1e-12 * np.abs(sr).max()
