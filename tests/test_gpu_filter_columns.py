"""The MI filter E-step with bin columns against the FP64 oracle where its rule draws the line: one to
four channels, bin counts that are not multiples of four, the 512-, 384- and 256-thread forms, and
likelihoods past it (five channels, more than 64 bins, columns that do not fit), which keep the
two-pass kernel.  Tolerances of the other filter tests."""
import numpy as np
import pytest

from test_gpu_mi_filter import filter_case, new_filter_reg, oracle_iteration

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,L", [(1, 5, 7), (2, 16, 9), (2, 48, 48), (2, 64, 61), (3, 31, 30),
                                   (4, 18, 17), (4, 64, 8), (5, 8, 6), (2, 100, 40), (4, 48, 60)])
def test_one_iteration(core, oracle, M, K, L):
    c = filter_case(K=K, L=L, M=M, seed=M + K)
    reg = new_filter_reg(core, c)
    assert reg.EM(1, -1e30, 1, 0) == 1
    mll, dream, th, _, final, _ = oracle_iteration(oracle, c, c["d0"].astype(np.float64),
                                                   c["thf"].astype(np.float64))
    np.testing.assert_allclose(reg.get_dream_locations(), dream, rtol=0, atol=5e-5)
    np.testing.assert_allclose(reg.get_likelihood_parameters(), th, rtol=1e-4, atol=1e-6)
    np.testing.assert_allclose(reg.get_final_locations_as_numpy_array().ravel(), final, rtol=0,
                               atol=2e-4)
    assert reg.iteration_stats()[0][0] == pytest.approx(mll, rel=1e-6)


def test_repeatable(core):
    """The merge is exact in integers: two runs are the same bit for bit."""
    c = filter_case(shape=(20, 19, 18), K=16, L=12, M=2, seed=3)
    runs = []
    for _ in range(2):
        reg = new_filter_reg(core, c)
        reg.EM(5, -1e30, 1, 0)
        runs.append((reg.get_final_locations_as_numpy_array(), reg.get_likelihood_parameters()))
    np.testing.assert_array_equal(runs[0][0], runs[1][0])
    np.testing.assert_array_equal(runs[0][1], runs[1][1])
