"""What a context with an HBM budget holds is what its callers ask for: nothing that the engine keeps for speed
(scratch between calls, second copies of matrices) counts against a call that fits beside it."""
import numpy as np
import pytest

from krans_b200 import generators as G

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


def test_batch_after_a_solve_under_a_budget():
    """The smallest budget that holds a batch also holds it after a single solve and a block product."""
    import krans_b200 as kb
    from krans_b200.serving import SolveRequest, solve_batch
    n = 3000
    opt = kb.CyclicLanczosOptions(k=1, tol_abs=1e-12, tol_rel=0.0, cg_maxit=200, max_restarts=2, grad_max_iters=10)

    def runs(budget, before):
        ctx = kb.Context(0, hbm_budget=budget)
        try:
            M = kb.CudaCsrMatrixAdapter(ctx, n, n, *_ring(n))
            if before:
                held = ctx.memory_in_use()
                kb.find_nullspace_cyclic_lanczos(M, kb.CudaVectorFactory(ctx, n, seed=1), opt)
                assert ctx.memory_in_use() == held  # the basis and the factory are gone, nothing is kept
            solve_batch(ctx, [SolveRequest(M, opt, seed=1 + i, keep_basis=False) for i in range(3)])
            return True
        except kb.KransError:
            return False

    lo, hi = 0, 64 << 20
    assert runs(hi, False)
    while hi - lo > 1024:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if runs(mid, False) else (mid, hi)
    assert runs(hi, True)


def test_creation_without_room_for_slices():
    """Rows and columns of uneven lengths: the sorted slices do not count against the budget of the arrays."""
    import krans_b200 as kb
    A = G.planted_kernel(6000, 4000, 8, kernel=False).A
    m, n = A.shape
    ctx = kb.Context(0, hbm_budget=_plain_bytes(m, n, A.nnz) + 8 * (m + n) + 1024)
    M = kb.CudaCsrMatrixAdapter.from_scipy(ctx, A)
    x = kb.CudaVectorAdapter.from_numpy(ctx, np.ones(n))
    y = kb.CudaVectorAdapter(ctx, m)
    M.multiply(x, y)
    np.testing.assert_allclose(y.data(), A @ np.ones(n), rtol=1e-12, atol=1e-12)


@pytest.mark.parametrize("solver,n", [("lobpcg", 2500), ("lobpcg", 20001), ("cyclic", 50001)])  # cluster, whole GPU
def test_auto_team_under_the_smallest_budget_of_one_block(solver, n):
    """KRANS_TEAM_AUTO takes a larger team where there is room for its partial sums, and one block where not."""
    import krans_b200 as kb
    inst = G.shift_operator(n, 2, 0.5, kernel=False)

    def runs(budget, team):
        ctx = kb.Context(0, hbm_budget=budget)
        try:
            M = kb.CudaCsrMatrixAdapter.from_scipy(ctx, inst.A)
            vf = kb.CudaVectorFactory(ctx, n, seed=4)
            if solver == "lobpcg":
                kb.find_nullspace_lobpcg(M, vf, kb.LOBPCGOptions(nev=2, block_size=4, max_iters=2, team=team))
            else:
                kb.find_nullspace_cyclic_lanczos(M, vf, kb.CyclicLanczosOptions(
                    k=2, ncv=8, max_restarts=1, cg_maxit=2, grad_max_iters=1, team=team))
            return True
        except kb.KransError as e:
            assert "budget" in str(e)
            return False

    lo, hi = 0, 256 << 20
    assert runs(hi, 1)
    while hi - lo > 4096:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if runs(mid, 1) else (mid, hi)
    assert runs(hi, 0)


def test_workspace_of_a_solve_without_an_output_array():
    """LOBPCG finds vectors and has nowhere to put them: the error leaves no workspace behind."""
    import ctypes as C
    import krans_b200 as kb
    from krans_b200 import _capi as K
    n = 1000
    ctx = kb.Context(0, hbm_budget=64 << 20)
    M = kb.CudaCsrMatrixAdapter.from_scipy(ctx, G.shift_operator(n, 2, 0.5, kernel=False).A)
    vf = kb.CudaVectorFactory(ctx, n, seed=4)
    o = kb.LOBPCGOptions(nev=2, block_size=4, tol_abs=1e-10, tol_rel=0.0).to_c()
    held = ctx.memory_in_use()
    rc = ctx.lib.krans_solve_lobpcg(ctx.h, M.h, vf.h, C.byref(o), None, 0, None, None, None,
                                    C.byref(K.LobpcgResultC()))
    assert rc == K.KRANS_ERR_INVALID_ARGUMENT
    assert ctx.memory_in_use() == held
