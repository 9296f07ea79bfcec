"""Long MT19937 draws are made in pieces of 2^22 values: wherever the last piece ends, with and without a
value carried into it, the draws that follow stay in the sequence of the CPU oracle (log and sqrt may differ
by an ulp or two, a skipped word changes everything after it)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
PIECE = 1 << 22


@pytest.mark.parametrize("lengths", [[1, PIECE + 1, 9001], [PIECE + 1, PIECE + 1, 7], [3, 2 * PIECE + 1, 9001],
                                     [1, PIECE + 2, 9001], [1, PIECE + 8191, 3], [1, PIECE + 8192, 3]])
def test_normals_after_the_last_piece(ctx, oracle, lengths):
    import krans_b200 as kb
    vf = kb.CudaVectorFactory(ctx, 1, seed=79)
    ref = oracle.Rng(79)
    for n in lengths:
        np.testing.assert_allclose(vf.create_random_of_size(n).data(), ref.normal(n), rtol=1e-14, atol=0)
