"""Where operands are read by sorted slices and where not (row lengths 1 and 2, few slices of long rows on wide
teams, padding), on one block, on the cluster and on the whole GPU: ||A x|| against numpy, and null spaces of
incidence matrices, whose CG keeps vectors by slice position, against the exact ones, preconditioned too."""
import numpy as np
import pytest
import scipy.sparse as sp

from krans_b200 import generators as G

pytestmark = pytest.mark.gpu


def _rows(lens, cols, seed):
    r = np.random.default_rng(seed)
    ip = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    idx = np.concatenate([r.choice(cols, k, replace=False) for k in lens]).astype(np.int32)
    return sp.csr_matrix((r.standard_normal(ip[-1]), idx, ip), shape=(len(lens), cols))


def _operands():
    r = np.random.default_rng(2)
    spike = np.ones(2049, int)
    spike[::256] = 64  # 7.1 entries of a slice for each real one
    yield "one entry", _rows(np.ones(3001, int), 2500, 1)
    yield "few long rows", _rows(r.integers(20, 65, 333), 5000, 2)
    yield "many long rows", _rows(r.integers(20, 65, 2999), 2500, 3)
    yield "spikes", _rows(spike, 3500, 4)
    yield "more padding than kept", _rows(np.where(np.arange(2049) % 256 == 0, 64, r.integers(0, 2, 2049)), 3500, 5)


@pytest.mark.parametrize("team", [0, 1, 2])
@pytest.mark.parametrize("name,A", list(_operands()), ids=[n for n, _ in _operands()])
def test_products_of_every_team(name, A, team):
    import krans_b200 as kb
    ctx = kb.default_context()
    n = A.shape[1]
    x = kb.CudaVectorFactory(ctx, n, seed=5).create_random().data()
    want = np.linalg.norm(A @ x)
    opt = kb.CyclicLanczosOptions(k=1, frob_samples=1, max_restarts=1, cg_maxit=5, grad_max_iters=1, team=team)
    R = kb.find_nullspace_cyclic_lanczos_ex(kb.CudaCsrMatrixAdapter.from_scipy(ctx, A),
                                            kb.CudaVectorFactory(ctx, n, seed=5), opt)
    # at most 64 products per row and 3001 squares: rounding below 1e-12 relative
    assert R.frob_norm_est == pytest.approx(want, rel=1e-12)


@pytest.mark.parametrize("precond", [0, 1, 2])
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n,degree,team", [(3000, 6.0, 0), (3000, 6.0, 2), (300, 40.0, 0), (300, 40.0, 2)])
def test_incidence_null_spaces(n, degree, team, mixed, precond):
    import krans_b200 as kb
    ctx = kb.default_context()
    inst = G.graph_incidence(n, 3, degree, seed=6)
    M = kb.CudaCsrMatrixAdapter.from_scipy(ctx, inst.A, fp32=True)
    opt = kb.CyclicLanczosOptions(k=3, tol_abs=1e-12, tol_rel=0.0, cg_maxit=1000, team=team,
                                  precision=kb.Precision(int(mixed)), precond_aat=kb.Precond(precond))
    U = kb.basis_to_numpy(kb.find_nullspace_cyclic_lanczos(M, kb.CudaVectorFactory(ctx, n, seed=4), opt))
    assert U.shape[0] == 3
    assert max(np.linalg.norm(inst.A @ u) for u in U) <= 1e-12
    assert np.linalg.norm(U - (U @ inst.kernel.T) @ inst.kernel, 2) <= 1e-10
