"""KRANS_SMEM_CG_KB (CG vectors of one-block solves in shared memory, read once per process) changes where the vectors
of each form of CG are, and no bit of the results: operators of 2 and of other row lengths, with and without a
preconditioner, one by one and in a batch."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = r"""
import hashlib, numpy as np, krans_b200 as kb
from krans_b200 import generators as G
from krans_b200.serving import SolveRequest, solve_batch
ctx = kb.Context(0)
h = hashlib.sha256()
for A in (G.graph_incidence(600, 3, 6.0, seed=2).A, G.planted_kernel(700, 500, 3, kernel=False).A):
    M = kb.CudaCsrMatrixAdapter.from_scipy(ctx, A, fp32=True)
    for precond in (0, 1, 2):
        o = kb.CyclicLanczosOptions(k=3, team=1, max_restarts=3, cg_maxit=40, grad_max_iters=5, precond_aat=kb.Precond(precond))
        R = kb.find_nullspace_cyclic_lanczos_ex(M, kb.CudaVectorFactory(ctx, A.shape[1], seed=42), o)
        h.update(kb.basis_to_numpy(R.right_null).tobytes() if R.right_null else b"none")
        h.update(np.array([R.spmv, R.spmvT, R.cg_solves, R.cg_maxit_hits, R.frob_norm_est]).tobytes())
        q = SolveRequest(M, o, seed=7)
        solve_batch(ctx, [q])
        h.update(q.basis().tobytes())
print(h.hexdigest())
"""


def _digest(kb_):
    out = subprocess.run([sys.executable, "-c", CODE], env=dict(os.environ, KRANS_SMEM_CG_KB=str(kb_)), cwd=ROOT,
                         capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    return out.stdout.split()[-1]


def test_shared_memory_vectors_change_no_bit():
    assert _digest(160) == _digest(0)
