"""A guard-band solve whose overlaps are indefinite in many steps (displaced
64-atom cell, 217 bands at (1/2, 1/2, 1/2), locking off): each such step is
redone with the metric normalisation, and the solve converges.  Its
eigenvalues against the locked mixed solve's, which takes another path."""
import os

import numpy as np
import pytest

import halfb200
from halfb200 import synth

pytestmark = pytest.mark.gpu

K = (0.5, 0.5, 0.5)


@pytest.fixture(scope="module")
def ctx(tmp_path_factory):
    w = synth.workload("si64")
    r = np.random.default_rng(3)
    w.positions = np.mod(w.positions + r.normal(0, 0.02, w.positions.shape) @ np.linalg.inv(w.lattice), 1.0)
    ch, po = synth.write_inputs(w, os.path.join(tmp_path_factory.mktemp("redone"), "in"))
    with halfb200.Context(ch, po, w.encut, xc=w.xc, solver="acc") as c:
        yield c


@pytest.mark.parametrize("precision", ["fp64_guarded", "mixed"])
def test_steps_are_redone_until_convergence(precision, ctx, monkeypatch):
    ctx.set_acc(tol=2e-5, max_iterations=300, precision="mixed")
    ref = ctx.solve(K, 200)[0]
    assert ctx.info()["converged"] == 1
    monkeypatch.setenv("HALF_SOFT_LOCK", "0")
    ctx.set_acc(tol=2e-5, max_iterations=150, precision=precision)
    eig = ctx.solve(K, 217)[0]
    assert ctx.info()["converged"] == 1
    # residuals of 2e-5 eV: eigenvalues to the square of that over the gaps, 1e-6 eV is far outside
    assert np.abs(eig[:200] - ref).max() <= 1e-6
