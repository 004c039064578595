"""A mixed solve whose residue planes (zcrt.cu) do not fit on the device takes
ZGEMM for those products and gives the same eigenvalues (64-atom cell, 600
bands: blocks of 134 MB, planes of 184 MB and more)."""
import ctypes as C
import os

import numpy as np
import pytest

import halfb200
from halfb200 import synth

pytestmark = pytest.mark.gpu

K = (0.25, 0.0, 0.0)


@pytest.mark.parametrize("limit_mb", [150, 230])   # all planes refused; those of B fit, the blocks' do not
def test_solve_without_room_for_residue_planes(limit_mb, tmp_path):
    lib = C.CDLL(halfb200.library_path())
    lib.hb_diag_refuse_allocations.restype = C.c_longlong
    lib.hb_diag_refuse_allocations.argtypes = [C.c_size_t]
    w = synth.workload("si64")
    ch, po = synth.write_inputs(w, os.path.join(tmp_path, "in"))
    with halfb200.Context(ch, po, w.encut, xc=w.xc, solver="acc") as ctx:
        ctx.set_acc(tol=1e-6, max_iterations=200, precision="mixed")
        want = ctx.solve(K, 600)[0]
        lib.hb_diag_refuse_allocations(limit_mb << 20)
        try:
            got = ctx.solve(K, 600)[0]
        finally:
            refused = lib.hb_diag_refuse_allocations(0)
        assert ctx.info()["converged"] == 1
    assert refused > 0
    assert np.abs(got - want).max() <= 1e-9
