"""What a context with an HBM budget holds is what its callers ask for: nothing that the engine keeps for speed
(scratch between calls, second copies of matrices) counts against a call that fits beside it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plain_bytes(m, n, nnz):
    """The stored arrays of an FP64 matrix and its transpose, each from a 256-byte boundary."""
    return sum((b + 255) // 256 * 256 for b in (4 * (m + 1), 4 * (n + 1), 4 * nnz, 4 * nnz, 8 * nnz, 8 * nnz))


def _ring(n):
    """x_{i+1} - x_i around a ring: two entries a row and a column; the constants are its null space."""
    i = np.arange(n, dtype=np.int32)
    return np.arange(0, 2 * n + 1, 2, dtype=np.int32), np.stack([i, (i + 1) % n], 1).ravel(), np.tile([-1.0, 1.0], n)


def test_creation_scratch_is_outside_the_budget():
    import krans_b200 as kb
    n = 100_000
    ctx = kb.Context(0, hbm_budget=_plain_bytes(n, n, 2 * n))
    M = kb.CudaCsrMatrixAdapter(ctx, n, n, *_ring(n))  # the device transpose takes another 2.8 MB meanwhile
    assert ctx.memory_in_use() <= _plain_bytes(n, n, 2 * n)
    del M
