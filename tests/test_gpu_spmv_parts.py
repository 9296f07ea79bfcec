"""Standalone A^T x of an operand whose x is larger than L2: the column-part path
(automatic from 12,582,912 rows of A) equals the whole-operand row-tile kernel bit
for bit in FP64 and FP32, with rows from empty to longer than a tile."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [12_582_912, 12_582_911])  # cut, and just below
def test_column_parts_equal_the_whole(ctx, m):
    import krans_b200 as kb
    from krans_b200 import _capi as K
    r = np.random.default_rng(8)
    n = 200_003
    # one entry per row of A; columns uneven: a few with thousands of entries, some with none
    cols = (n * r.random(m) ** 3).astype(np.int32)
    M = kb.CudaCsrMatrixAdapter(ctx, m, n, np.arange(m + 1, dtype=np.int32), cols, r.standard_normal(m), fp32=True)
    x = kb.CudaVectorAdapter.from_numpy(ctx, r.standard_normal(m))
    y, z = kb.CudaVectorAdapter(ctx, n), kb.CudaVectorAdapter(ctx, n)
    for prec in (K.KRANS_PREC_FP64, K.KRANS_PREC_MIXED):
        M.set_spmv_tuning(True, K.KRANS_SPMV_AUTO)
        M.multiply_transpose(x, y, prec)
        M.set_spmv_tuning(True, K.KRANS_SPMV_ROWTILE)
        M.multiply_transpose(x, z, prec)
        assert np.array_equal(y.data(), z.data())
