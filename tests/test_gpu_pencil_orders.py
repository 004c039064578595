"""The Rayleigh-Ritz pencils over the orders where their solver changes: the
CTA counts of the cluster kernels (1, 4, 8 and 16 CTAs up to orders 40, 80,
176 and 432), orders that leave the last CTAs with a column less, the
grid-wide factor and reduction from 434 to 1,280 and the first order beyond, which goes
to cuSOLVER.  The converged eigenvalues of the 12-atom cell against the FP64
dense solve (1e-8 eV, the parity tests' bound for converged solves)."""
import numpy as np
import pytest

import halfb200

pytestmark = pytest.mark.gpu

K = (0.125, 0.25, 0.375)


@pytest.fixture(scope="module")
def dense(hfo2):
    w, ch, po = hfo2
    with halfb200.Context(ch, po, w.encut, xc=w.xc, solver="vasp") as ctx:
        return ctx.solve(K, 515)[0]


# bands -> first pencil 2 (bands + max(4, bands / 4) guard bands); locking then shrinks it by even steps
@pytest.mark.parametrize("bands", [1, 3, 16, 17, 32, 33, 57, 70, 71, 120, 173, 174])
@pytest.mark.parametrize("precision", ["fp64_guarded", "mixed"])
def test_pencil_orders_match_dense(bands, precision, hfo2, dense):
    w, ch, po = hfo2
    with halfb200.Context(ch, po, w.encut, xc=w.xc, solver="acc") as ctx:
        ctx.set_acc(tol=2e-5, max_iterations=400, precision=precision)
        eig = ctx.solve(K, bands)[0]
        assert ctx.info()["converged"] == 1
    assert np.abs(eig - dense[:bands]).max() <= 1e-8


@pytest.mark.parametrize("bands", [240, 400, 483, 512, 515])   # first pencils of order 600 to 1,280, and 1,286
def test_grid_wide_pencils_match_dense(bands, hfo2, dense):
    w, ch, po = hfo2
    with halfb200.Context(ch, po, w.encut, xc=w.xc, solver="acc") as ctx:
        ctx.set_acc(tol=2e-5, max_iterations=400, precision="fp64_guarded")
        eig = ctx.solve(K, bands)[0]
        assert ctx.info()["converged"] == 1
        batch = ctx.solve_kpoints([K, K], bands)   # two streams, each with grid-wide launches
    assert np.abs(eig - dense[:bands]).max() <= 1e-8
    assert np.abs(batch - dense[:bands]).max() <= 1e-8


def test_fp64_mode_pencils_of_cluster_size(hfo2, dense):
    """The plain FP64 iteration: metric step and pencil both on the cluster kernels."""
    w, ch, po = hfo2
    with halfb200.Context(ch, po, w.encut, xc=w.xc, solver="acc") as ctx:
        ctx.set_acc(tol=2e-5, max_iterations=3000, precision="fp64")
        eig = ctx.solve(K, 96)[0]
        assert ctx.info()["converged"] == 1
    assert np.abs(eig - dense[:96]).max() <= 1e-8
