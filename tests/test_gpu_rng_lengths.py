"""The factory's MT19937 normals on both sides of the line between the one-block
draw and the whole-GPU draw, odd and even, with the value and the state carried
from vector to vector, against the CPU oracle (a shifted or lost value would
change everything after it; log and sqrt may differ by an ulp or two)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [[1, 8191, 8192, 8193, 8192], [3, 20001, 20001, 2, 624, 50000],
                                     [8193, 1, 1, 8193, 300007], [4194305, 9001]])
def test_normals_over_lengths(ctx, oracle, lengths):
    import krans_b200 as kb
    vf = kb.CudaVectorFactory(ctx, 1, seed=77)
    ref = oracle.Rng(77)
    for n in lengths:
        np.testing.assert_allclose(vf.create_random_of_size(n).data(), ref.normal(n), rtol=1e-14, atol=0)


def test_normals_without_room_for_scratch(ctx, oracle):
    """A budget that holds the vector (160 kB) but not the words of a whole-GPU draw (240 kB): one block draws."""
    import krans_b200 as kb
    vf = kb.CudaVectorFactory(kb.Context(0, hbm_budget=300_000), 1, seed=78)
    ref = oracle.Rng(78)
    x = vf.create_random_of_size(20001)
    np.testing.assert_allclose(x.data(), ref.normal(20001), rtol=1e-14, atol=0)
