"""The local operator over FFT boxes of every pass count and of ragged sizes:
axes of one (up to 10 points), two and three (75, 125, 128) register passes,
widths that are no multiple of the x-line kernel's 16-column tile, and planes
small and large enough for every CTA size of the plane kernels.  FP64 results
against the oracle (numpy's FFTs), 1e-11 of the largest element as in the
parity tests; the FP32 operator to 1e-4."""
import os

import numpy as np
import pytest

import halfb200
from conftest import rng
from halfb200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,encut", [
    ((8, 9, 10), 40.0),       # one pass on every axis
    ((10, 12, 9), 40.0),      # one and two passes
    ((20, 27, 25), 200.0),
    ((45, 16, 30), 150.0),
    ((75, 18, 40), 150.0),    # three passes on x
    ((25, 125, 24), 150.0),   # three passes on y
    ((27, 20, 128), 150.0),   # three passes on z
    ((128, 54, 36), 150.0),
    ((48, 100, 81), 150.0),   # FP64 plane of 134 KB: one CTA per SM
])
def test_apply_hs_over_box_sizes(grid, encut, tmp_path):
    from oracle import hamiltonian as H
    w = synth.workload("si2")
    w.grid, w.encut = grid, encut
    ch, po = synth.write_inputs(w, os.path.join(tmp_path, "in"))
    k = (0.125, -0.25, 0.375)
    op = H.prepare(H.load_system(ch, po, w.encut, use_pbe=False, use_uspp=True), k)
    r = rng(7)
    psi = r.normal(size=(op.basis.npw, 19)) + 1j * r.normal(size=(op.basis.npw, 19))
    hr, sr = H.apply_hs(op, psi)
    with halfb200.Context(ch, po, w.encut, xc="lda", solver="acc") as ctx:
        hg, sg = ctx.apply_hs(k, psi)
        assert np.abs(hg - hr).max() <= 1e-11 * np.abs(hr).max()
        assert np.abs(sg - sr).max() <= 1e-11 * np.abs(sr).max()
        ctx.set_acc(precision="mixed")
        hg, sg = ctx.apply_hs(k, psi)
        assert np.abs(hg - hr).max() <= 1e-4 * np.abs(hr).max()
        assert np.abs(sg - sr).max() <= 1e-4 * np.abs(sr).max()
