"""The single-pass EM E-step's flush (four bins at a time) and the merge of its histogram in the
likelihood update, against the FP64 oracle: bin counts that are and are not multiples of four, one
bin, the 768-thread form, FP16 columns with an odd count, and an EM call that leaves theta alone.
Tolerances as in the other one-iteration tests: FP32 weights, one FP32 rounding per theta cell and
the CTA histogram's fixed point (half a unit of 1 / 127,097 per voxel at worst, unbiased)."""
import numpy as np
import pytest

from test_gpu_edge_cases import one_iteration
from test_gpu_parity import make_case, new_reg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,L", [(1, 4), (3, 5), (4, 4), (5, 3), (63, 61), (64, 64)])
def test_bin_counts(core, oracle, K, L):
    one_iteration(core, oracle, make_case(shape=(13, 12, 11), K=K, L=L, seed=K + L))


def test_wide_form_with_odd_bins(core, oracle):
    """97^3 voxels: 768-thread CTAs."""
    one_iteration(core, oracle, make_case(shape=(97, 97, 97), K=63, L=61, seed=11))


@pytest.mark.parametrize("K", [5, 63])
def test_fp16_columns_with_odd_bins(core, oracle, K):
    c = make_case(shape=(13, 12, 11), K=K, L=6, seed=K)
    reg = new_reg(core, c, c["d0"])
    reg.set_histogram_precision(1)
    assert reg.EM(1, -1e30, 1, 0) == 1
    _, dream, hist, _ = oracle.estep(c["d0"].astype(np.float64), c["u"], c["v"],
                                     c["theta"].astype(np.float64), c["shape"], c["shape"], K, 6)
    np.testing.assert_allclose(reg.get_dream_locations(), dream, rtol=0, atol=5e-5)
    theta = oracle.theta_map(hist, K, 6, 2.0)
    # each mass rounded to FP16 (2^-11) and summed over the voxels of a cell
    np.testing.assert_allclose(reg.get_likelihood_parameters(), theta, rtol=2e-3, atol=1e-5)


def test_theta_left_alone(core, oracle):
    """update_likelihood_parameters 0: theta stays, the log-likelihood is still merged, and the
    sums do not leak into a later call."""
    c = make_case(shape=(13, 12, 11), K=9, L=7, seed=3)
    reg = new_reg(core, c, c["d0"])
    assert reg.EM(2, -1e30, 0, 0) == 2
    np.testing.assert_array_equal(reg.get_likelihood_parameters(), c["theta"].ravel())
    mll, _, _, _ = oracle.estep(c["d0"].astype(np.float64), c["u"], c["v"],
                                c["theta"].astype(np.float64), c["shape"], c["shape"], 9, 7)
    assert reg.iteration_stats()[0][0] == pytest.approx(mll, rel=1e-6)
    reg.reset()
    assert reg.EM(1, -1e30, 1, 0) == 1
    _, _, hist, _ = oracle.estep(c["d0"].astype(np.float64), c["u"], c["v"],
                                 c["theta"].astype(np.float64), c["shape"], c["shape"], 9, 7)
    np.testing.assert_allclose(reg.get_likelihood_parameters(), oracle.theta_map(hist, 9, 7, 2.0),
                               rtol=1e-4, atol=1e-6)
