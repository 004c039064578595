"""Guard-band solves with wide blocks at tight tolerances: their pencils keep
orders of about 1,000 to 1,280 down to the last iterations, where the
correction directions are as small as the residuals (12-atom cell).  The
solve converges in a few iterations and its vectors have the residuals that
it reports: recomputed from the returned vectors with the FP64 operator, whose
own rounding is about 1e-12 eV."""
import numpy as np
import pytest

import halfb200

pytestmark = pytest.mark.gpu

K = (0.125, 0.25, 0.375)


@pytest.mark.parametrize("tol", [1e-6, 1e-7])
@pytest.mark.parametrize("bands", [480, 512])
@pytest.mark.parametrize("precision", ["fp64_guarded", "mixed"])
def test_wide_blocks_converge_to_tight_tolerances(precision, bands, tol, hfo2):
    w, ch, po = hfo2
    with halfb200.Context(ch, po, w.encut, xc=w.xc, solver="acc") as ctx:
        ctx.set_acc(tol=tol, max_iterations=40, precision=precision)
        eig, vec, _, _ = ctx.solve(K, bands, vectors=True)
        info = ctx.info()
        ctx.set_acc(tol=tol, max_iterations=40, precision="fp64_guarded")
        h, s = ctx.apply_hs(K, vec)
    res = np.linalg.norm(h - s * eig[None, :], axis=0)
    assert info["converged"] == 1
    assert info["fp64_iterations"] <= 20
    assert res.max() <= tol + 1e-10
