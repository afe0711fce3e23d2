"""The branches of a captured EM iteration (the likelihood update beside the M-step, the pairs of a
batch beside each other, the components of the per-axis tensor-core passes), on grids with and
without axes of equal length, which share their DCT matrices: a batch runs the same kernels on the same data as its members
alone and every sum that feeds the fields is an integer one, so the results are the same bits."""
import numpy as np
import pytest

from test_gpu_parity import make_case, new_reg

pytestmark = pytest.mark.gpu

SHAPES = [(13, 12, 11), (12, 12, 9), (9, 14, 14), (10, 7, 10), (16, 16, 16)]


@pytest.mark.parametrize("precision", [0, 1, 2, 3, 4])
def test_batch_equals_its_members(core, precision):
    cases = [make_case(shape=s, K=6, L=5, seed=i + 1) for i, s in enumerate(SHAPES)]
    alone, batched = ([new_reg(core, c, c["d0"]) for c in cases] for _ in range(2))
    for r in alone + batched:
        r.set_precision(precision)
    assert [r.EM(9, -1e300, 1, 0) for r in alone] == [9] * len(SHAPES)
    assert list(core.RegistrationBatch(batched).EM(9, -1e300, 1)) == [9] * len(SHAPES)
    for a, b in zip(alone, batched):
        np.testing.assert_array_equal(a.get_final_locations_as_numpy_array(),
                                      b.get_final_locations_as_numpy_array())
        np.testing.assert_array_equal(a.get_likelihood_parameters(),
                                      b.get_likelihood_parameters())
