"""KRANS_TEAM_AUTO on both sides of the lines between one block, a cluster and
the whole GPU, and beside a live server (where a solve stays on one block): the
null space of shift operators against the exact one."""
import numpy as np
import pytest

from krans_b200 import generators as G

pytestmark = pytest.mark.gpu


def _check(U, inst):
    assert U.shape[0] == inst.k
    R = U - (U @ inst.kernel.T) @ inst.kernel  # what lies outside the exact null space
    assert np.linalg.norm(R, 2) <= 1e-10


def _cyclic(ctx, inst, mixed):
    import krans_b200 as kb
    M = kb.CudaCsrMatrixAdapter.from_scipy(ctx, inst.A, fp32=True)
    o = kb.CyclicLanczosOptions(k=inst.k, tol_abs=1e-12, tol_rel=0.0, cg_maxit=1000,
                                precision=kb.Precision.MIXED if mixed else kb.Precision.FP64)
    return kb.basis_to_numpy(kb.find_nullspace_cyclic_lanczos(M, kb.CudaVectorFactory(ctx, inst.A.shape[1], seed=4), o))


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n", [2500, 2501, 50000, 50001])  # m + n = 2 n - 2: around 5000 and 100000
def test_cyclic_team_lines(ctx, n, mixed):
    inst = G.shift_operator(n, 2, 0.5)
    _check(_cyclic(ctx, inst, mixed), inst)


@pytest.mark.parametrize("n", [2000, 2001, 20000, 20001])  # around 4000 and 40000
def test_lobpcg_team_lines(ctx, n):
    import krans_b200 as kb
    inst = G.shift_operator(n, 2, 0.5)
    M = kb.CudaCsrMatrixAdapter.from_scipy(ctx, inst.A)
    o = kb.LOBPCGOptions(nev=2, block_size=4, tol_abs=1e-12, tol_rel=0.0)
    _check(kb.basis_to_numpy(kb.find_nullspace_lobpcg(M, kb.CudaVectorFactory(ctx, n, seed=4), o)), inst)


def test_solve_beside_a_server(ctx):
    from krans_b200.serving import Server
    inst = G.shift_operator(6000, 2, 0.5)
    srv = Server(ctx)
    try:
        _check(_cyclic(ctx, inst, True), inst)
    finally:
        srv.close()
    _check(_cyclic(ctx, inst, True), inst)
