"""Sorted-slice SpMV of the solvers (operands whose rows differ in length and
hold at most 64 entries) at the edges of its slices and windows. The solver's
||A||_F estimate with one sample is ||A x|| for the factory's next vector x,
so it checks the product of every row structure against numpy."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _ragged(rows, cols, longest, seed):
    r = np.random.default_rng(seed)
    lens = np.minimum(r.poisson(4.0, rows), longest)
    lens[0] = 0
    lens[-1] = longest  # the last row, in the last (partial) slice, is the longest
    cap = min(longest, cols)
    lens = np.minimum(lens, cap)
    indptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    indices = np.concatenate([r.choice(cols, k, replace=False) for k in lens]).astype(np.int32)
    return sp.csr_matrix((r.standard_normal(indptr[-1]), indices, indptr), shape=(rows, cols))


@pytest.mark.parametrize("longest", [1, 8, 64, 65])  # 65: beyond the longest row a lane sums alone
@pytest.mark.parametrize("rows", [1, 31, 32, 33, 255, 256, 257, 1031])
def test_frobenius_sample_over_row_structures(rows, longest):
    import krans_b200 as kb
    ctx = kb.default_context()
    cols = 97
    A = _ragged(rows, cols, longest, 11 * rows + longest)
    x = kb.CudaVectorFactory(ctx, cols, seed=5).create_random().data()
    want = np.linalg.norm(A @ x)
    opt = kb.CyclicLanczosOptions(k=1, frob_samples=1, max_restarts=1, cg_maxit=5, grad_max_iters=1)
    R = kb.find_nullspace_cyclic_lanczos_ex(kb.CudaCsrMatrixAdapter.from_scipy(ctx, A),
                                            kb.CudaVectorFactory(ctx, cols, seed=5), opt)
    # at most 65 products per row and 1031 squares: rounding below 1e-12 relative
    assert R.frob_norm_est == pytest.approx(want, rel=1e-12)


@pytest.mark.parametrize("rows", [33, 257])
@pytest.mark.parametrize("mixed", [False, True])
def test_projector_cg_on_sliced_operands(rows, mixed):
    """A wide random matrix (both operands sliced): every vector of the null
    space found through the CG projector satisfies A u = 0."""
    import krans_b200 as kb
    ctx = kb.default_context()
    A = _ragged(rows, rows + 40, 8, 3 * rows)
    L = max(1.0, abs(A).max())
    opt = kb.CyclicLanczosOptions(k=3, tol_abs=1e-12 * L, tol_rel=0.0, cg_maxit=1000,
                                  precision=kb.Precision.MIXED if mixed else kb.Precision.FP64)
    R = kb.find_nullspace_cyclic_lanczos_ex(kb.CudaCsrMatrixAdapter.from_scipy(ctx, A, fp32=True),
                                            kb.CudaVectorFactory(ctx, A.shape[1], seed=9), opt)
    U = kb.basis_to_numpy(R.right_null)
    assert U.shape[0] == 3
    assert np.abs(U @ U.T - np.eye(3)).max() < 1e-10
    assert max(np.linalg.norm(A @ u) for u in U) <= 1e-12 * L
