"""A request cancelled between the queueing of its launch and the launch's set-up on the device ends as cancelled. The
set-up is held back by work on the context's stream, which every launch waits for (matrices finish there)."""
import time

import pytest

from krans_b200 import generators as G

pytestmark = pytest.mark.gpu


def test_cancel_before_the_launch_is_set_up(ctx):
    import krans_b200 as kb
    from krans_b200.serving import Server, SolveRequest
    inst = G.graph_incidence(6000, 6, 6.0, seed=3, kernel=False)  # a tenth of a second, if nothing stops it
    M = kb.CudaCsrMatrixAdapter.from_scipy(ctx, inst.A, fp32=True)
    opt = kb.CyclicLanczosOptions(k=6, tol_abs=1e-12, tol_rel=0.0, cg_maxit=1000, precision=kb.Precision.MIXED)
    n = 50_000_000
    x, y = kb.CudaVectorAdapter(ctx, n), kb.CudaVectorAdapter(ctx, n)
    srv = Server(ctx)
    try:
        warm = SolveRequest(M, opt, seed=1, keep_basis=False)
        srv.submit(warm)
        srv.drain(60.0)
        assert srv.poll(warm.ticket)[0] == "done"
        time.sleep(0.1)  # the open launch leaves after 20 ms without work
        ctx.synchronize()
        for _ in range(4000):  # about 0.7 s on the context's stream
            y.add_scaled(x, 0.5)
        rq = SolveRequest(M, opt, seed=2, keep_basis=False)
        srv.submit(rq)
        deadline = time.perf_counter() + 20.0
        while srv.poll(rq.ticket)[0] == "queued" and time.perf_counter() < deadline:
            time.sleep(0.0005)
        srv.cancel(rq.ticket)
        srv.drain(60.0)
        assert srv.poll(rq.ticket)[0] == "cancelled"
    finally:
        srv.close()
