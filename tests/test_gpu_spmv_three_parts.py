"""Column parts of A^T beyond the first two, with several entries a row of A: equal to the whole-operand kernel, bit for
bit, and to numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_three_parts_equal_the_whole(ctx):
    import krans_b200 as kb
    from krans_b200 import _capi as K
    r = np.random.default_rng(18)
    m, n = 12_600_000, 300_007  # three parts of 4.2M columns of A^T
    cols = np.sort(r.integers(0, n, (m, 2), dtype=np.int32), axis=1)
    vals = r.standard_normal(2 * m)
    M = kb.CudaCsrMatrixAdapter(ctx, m, n, np.arange(0, 2 * m + 1, 2, dtype=np.int32), cols.ravel(), vals, fp32=True)
    xs = r.standard_normal(m)
    x = kb.CudaVectorAdapter.from_numpy(ctx, xs)
    y, z = kb.CudaVectorAdapter(ctx, n), kb.CudaVectorAdapter(ctx, n)
    for prec in (K.KRANS_PREC_FP64, K.KRANS_PREC_MIXED):
        M.set_spmv_tuning(True, K.KRANS_SPMV_AUTO)
        M.multiply_transpose(x, y, prec)
        M.set_spmv_tuning(True, K.KRANS_SPMV_ROWTILE)
        M.multiply_transpose(x, z, prec)
        assert np.array_equal(y.data(), z.data())
        if prec == K.KRANS_PREC_FP64:
            want = np.bincount(cols.ravel(), weights=vals * np.repeat(xs, 2), minlength=n)
            # about 84 products of order one a row: rounding below 84 * 84 ulp
            np.testing.assert_allclose(y.data(), want, rtol=0, atol=84 * 84 * 2.3e-16)
