"""The narrow form of the block combination (at most 16 output columns) around its steps of eight columns and at
both ends of its range, on odd and even numbers of rows. Tolerance: 64 ulp of the sum of absolute products."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.220446049250313e-16


@pytest.mark.parametrize("q", [1, 12, 16, 17])
@pytest.mark.parametrize("zc", [1, 7, 8, 9, 36])
def test_narrow_combine(ctx, zc, q):
    import torch
    import krans_b200 as kb
    for n in (1, 511, 20012):
        rng = np.random.default_rng(n + zc + q)
        Zc, Yc = rng.standard_normal((zc, n)), rng.standard_normal((q, zc))
        Z, Y = (torch.from_numpy(a).to("cuda:0") for a in (Zc, Yc))
        out = torch.full((q, n), np.nan, dtype=torch.float64, device="cuda:0")
        torch.cuda.synchronize()
        kb.block_combine(ctx, n, zc, q, Z.data_ptr(), n, Y.data_ptr(), zc, out.data_ptr())
        assert np.all(np.abs(out.cpu().numpy() - Yc @ Zc) <= 64 * EPS * (np.abs(Yc) @ np.abs(Zc)))
