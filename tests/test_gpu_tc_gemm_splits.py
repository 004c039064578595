"""The tensor-core GEMM where its split rule and operand passes change: few
splits run inside one CTA (2 to 4 accumulator pairs), many as partial sums;
short chains that leave room for a second CTA; K and row counts at the edges
of the 64-k and 32-row split tiles; two-output products.  Tolerance as for the
GEMM's other shapes: 4e-5 of sum_k |a_ik| |b_kj| per element (three-term bf16
split, 2^-16)."""
import pytest

from test_gpu_tc_gemm import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [
    (11023, 187, 193),   # 87 row tiles: 2 splits of 7 k blocks in one CTA
    (6000, 100, 256),    # 47 row tiles: 4 splits in one CTA
    (9000, 130, 1000),   # 2 splits of 32 k blocks in one CTA, two column tiles
    (7000, 250, 600),    # 3 splits
    (9000, 130, 1040),   # one k block more: partial sums in memory
    (128, 16, 64), (129, 17, 65), (97, 33, 63), (600, 600, 5000),
])
@pytest.mark.parametrize("op_a,op_b", [("N", "N"), ("C", "N"), ("N", "C")])
def test_split_products(m, n, k, op_a, op_b):
    ratio, _ = _run(op_a, op_b, m, n, k, lda_pad=1, ldb_pad=2, ldc_pad=1, alpha=0.5 - 2j, beta=0.25 + 1j, seed=m + k)
    assert ratio < 1.0
    ratio, _ = _run(op_a, op_b, m, n, k, c_fp64=True, seed=n)
    assert ratio < 1.0
