"""Edges of the panel products' tiles: row counts around the 32-row panels,
column counts around the 64-column tiles, and the 8-byte copies of blocks
whose leading dimension is odd. Tolerance: 64 ulp of the sum of absolute
products of each entry, as for the other block products."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.220446049250313e-16


@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("n,p", [(131_072, 33), (131_073, 64), (131_103, 65), (131_104, 129)])
def test_panel_product_edges(ctx, n, p, pad):
    import torch
    import krans_b200 as kb
    rng = np.random.default_rng(n + p + pad)
    ld = n + (n % 2) + pad  # even, then odd
    Zc, Wc = rng.standard_normal((p, ld)), rng.standard_normal((p, ld))
    new = lambda *s: torch.zeros(*s, dtype=torch.float64, device="cuda:0")  # noqa: E731
    Z, W = torch.from_numpy(Zc).to("cuda:0"), torch.from_numpy(Wc).to("cuda:0")
    S, G, C, out = new(p, p), new(p, p), new(p, p), new(p, ld)
    torch.cuda.synchronize()
    kb.block_gram(ctx, n, p, Z.data_ptr(), ld, S.data_ptr(), W.data_ptr(), G.data_ptr())
    kb.block_gemm_tn(ctx, n, p, Z.data_ptr(), p, W.data_ptr(), ld, C.data_ptr())
    kb.block_combine(ctx, n, p, p, Z.data_ptr(), ld, C.data_ptr(), p, out.data_ptr())
    Zn, Wn = Zc[:, :n].T, Wc[:, :n].T
    tol = 64 * EPS * (np.abs(Zn).T @ np.abs(Wn))
    ZW = Zn.T @ Wn
    assert np.all(np.abs(C.cpu().numpy().T - ZW) <= tol)
    assert np.all(np.abs(S.cpu().numpy() - Zn.T @ Zn) <= 64 * EPS * (np.abs(Zn).T @ np.abs(Zn)))
    up = np.triu(np.ones((p, p), bool))
    Gd = G.cpu().numpy().T
    assert np.all(np.abs(Gd - ZW)[up] <= tol[up]) and np.array_equal(Gd, Gd.T)
    Cn = C.cpu().numpy().T
    assert np.all(np.abs(out.cpu().numpy()[:, :n].T - Zn @ Cn) <= 64 * EPS * (np.abs(Zn) @ np.abs(Cn)))
