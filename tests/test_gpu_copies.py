"""Second copies that matrices keep for speed (sorted slices, column parts) go back when the device is full, and
the matrix works on without them."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _ragged(m, n, seed):
    r = np.random.default_rng(seed)
    lens = r.integers(4, 13, m)
    ip = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    return sp.csr_matrix((r.standard_normal(ip[-1]), r.integers(0, n, ip[-1]).astype(np.int32), ip), shape=(m, n))


def test_slices_go_back_when_the_device_is_full():
    import torch
    import krans_b200 as kb
    ctx = kb.Context(0)
    m, n = 600_000, 400_000
    A = _ragged(m, n, 3)
    M = kb.CudaCsrMatrixAdapter.from_scipy(ctx, A)
    plain = sum((b + 255) // 256 * 256 for b in (4 * (m + 1), 4 * (n + 1)) + 2 * (4 * A.nnz, 8 * A.nnz))
    held = ctx.memory_in_use()
    assert held > plain + 2 * 12 * A.nnz  # the slices of A and of A^T
    x = kb.CudaVectorFactory(ctx, n, seed=5).create_random().data()
    want = np.linalg.norm(A @ x)
    opt = kb.CyclicLanczosOptions(k=1, ncv=4, frob_samples=1, max_restarts=1, cg_maxit=5, grad_max_iters=1)

    def frob():  # ||A x|| for the factory's next vector, through the solver's product
        return kb.find_nullspace_cyclic_lanczos_ex(M, kb.CudaVectorFactory(ctx, n, seed=5), opt).frob_norm_est

    assert frob() == pytest.approx(want, rel=1e-12)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (96 << 20), dtype=torch.uint8, device="cuda:0")
    vs = []
    with pytest.raises(kb.KransError, match="(?i)memory"):
        for _ in range(4096):
            vs.append(kb.CudaVectorAdapter(ctx, (16 << 20) // 8))
    # all that is left of the context's own are the matrix's arrays
    assert ctx.memory_in_use() - len(vs) * (16 << 20) == plain
    vs.clear()
    del hold
    torch.cuda.empty_cache()
    assert frob() == pytest.approx(want, rel=1e-12)


def test_slices_without_more_than_seven_padded_entries_for_each_real_one():
    """One row of 64 entries among 255 empty ones: its slice would be 31 / 32 padding."""
    import krans_b200 as kb
    r = np.random.default_rng(4)
    m, n = 2560, 3500
    lens = np.where(np.arange(m) % 256 == 7, 64, 0)
    ip = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    A = sp.csr_matrix((r.standard_normal(ip[-1]), r.integers(0, n, ip[-1]).astype(np.int32), ip), shape=(m, n))
    ctx = kb.Context(0)
    before = ctx.memory_in_use()
    M = kb.CudaCsrMatrixAdapter.from_scipy(ctx, A)
    plain = sum((b + 255) // 256 * 256 for b in (4 * (m + 1), 4 * (n + 1)) + 2 * (4 * A.nnz, 8 * A.nnz))
    scratch = 1 << 20  # the context keeps at least as much after a creation
    # at most 8 entries of 12 bytes in a slice for each one, a row number a slot and a bound a slice, of both operands
    assert ctx.memory_in_use() - before - plain - scratch <= 2 * 8 * 12 * A.nnz + 5 * (m + n) + 4096
    del M


def test_destroyed_matrices_leave_a_bounded_pool():
    """What the context's pool keeps unused after a matrix is gone: its scratch and 64 MB, not the copies."""
    import torch
    import krans_b200 as kb
    ctx = kb.Context(0)
    m, n = 1_500_000, 1_000_000
    A = _ragged(m, n, 9)  # 12M entries: 290 MB of slices, 300 MB of arrays, 145 MB of scratch grown by half
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    M = kb.CudaCsrMatrixAdapter.from_scipy(ctx, A)
    during = torch.cuda.mem_get_info()[0]
    assert before - during > (500 << 20)
    del M
    assert before - torch.cuda.mem_get_info()[0] <= ctx.memory_in_use() + (64 << 20) + (96 << 20)
