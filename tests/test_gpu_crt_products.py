"""FP64 products on the integer tensor cores: blocks wide enough to take that
path against the same bands in blocks that stay on ZGEMM (64-atom cell, 512
projectors, about 11,000 plane waves; odd widths, so every tile has a
remainder).  Both round each product to about 2^-53 of |a| |b|; the operator
adds two of them, so 1e-13 of a column's largest element bounds the
difference.  Columns of very different scale, zero columns and columns with
NaN or infinity keep to themselves."""
import os

import numpy as np
import pytest

import halfb200
from conftest import rng
from halfb200 import synth

pytestmark = pytest.mark.gpu

K = (0.25, -0.125, 0.5)


@pytest.fixture(scope="module")
def ctx(tmp_path_factory):
    w = synth.workload("si64")
    ch, po = synth.write_inputs(w, os.path.join(tmp_path_factory.mktemp("crt"), "in"))
    with halfb200.Context(ch, po, w.encut, xc=w.xc, solver="acc") as c:
        yield c


def _narrow(ctx, x):
    h, s = zip(*(ctx.apply_hs(K, x[:, b:b + 64]) for b in range(0, x.shape[1], 64)))
    return np.concatenate(h, axis=1), np.concatenate(s, axis=1)


def _close(a, b):
    scale = np.abs(b).max(axis=0)
    return np.all(np.abs(a - b).max(axis=0) <= 1e-13 * scale)


@pytest.mark.parametrize("nb", [1203, 1601])
def test_wide_blocks_match_narrow_ones(nb, ctx):
    n = ctx.npw(K)
    r = rng(nb)
    x = r.normal(size=(n, nb)) + 1j * r.normal(size=(n, nb))
    x *= 10.0 ** r.uniform(-150, 150, size=nb)                # columns of any scale
    x[:, 1::5] *= np.exp(-8.0 * np.arange(n) / n)[:, None]    # decaying, as band vectors
    x[:, 7] = 0.0
    x[:, 11] = 0.0
    x[5, 11] = 1.0                                            # a unit vector
    h, s = ctx.apply_hs(K, x)
    hr, sr = _narrow(ctx, x)
    assert _close(h, hr) and _close(s, sr)


def test_non_finite_columns_keep_to_themselves(ctx):
    n = ctx.npw(K)
    r = rng(5)
    x = r.normal(size=(n, 1203)) + 1j * r.normal(size=(n, 1203))
    clean = x.copy()
    x[3, 100] = np.nan
    x[4, 700] = np.inf
    h, s = ctx.apply_hs(K, x)
    hr, sr = ctx.apply_hs(K, clean)
    bad = [100, 700]
    good = np.setdiff1d(np.arange(1203), bad)
    assert np.array_equal(h[:, good], hr[:, good]) and np.array_equal(s[:, good], sr[:, good])
    assert not np.isfinite(h[:, bad]).any() and not np.isfinite(s[:, bad]).any()
