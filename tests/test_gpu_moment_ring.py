"""The sampler's moments, which take several sweeps' positions at a time: they must equal the moments
of the same sweeps' positions one by one, for run lengths and burn-ins at every place of the ring
(eight slots, or as many as there are sweeps), for one chain and for a batch of chains.  FP64 updates
of FP32 positions: numpy's two-pass mean and covariance agree to a few roundings."""
import numpy as np
import pytest

from test_gpu_parity import make_case, new_reg

pytestmark = pytest.mark.gpu


def positions_after(core, c, sweeps):
    """positions of each of the first `sweeps` sweeps: the mean of a run of one sample"""
    out = []
    for s in range(sweeps):
        reg = new_reg(core, c)
        mean, _ = reg.sampler(5, s, 1, 1, 1, 1, 1, 1)
        out.append(mean)
    return np.stack(out)


def check(mean, cov, pos):
    np.testing.assert_allclose(mean, pos.mean(0), rtol=1e-12, atol=1e-12)
    d = pos - pos.mean(0)
    want = np.einsum("s...i,s...j->...ij", d, d) / (len(pos) - 1)
    np.testing.assert_allclose(cov, want, rtol=1e-9, atol=1e-12)


def test_moments_of_any_run_length(core):
    c = make_case(shape=(9, 10, 11), K=8, L=6, seed=2)
    pos = positions_after(core, c, 18)
    for burn, samples in [(0, 2), (0, 8), (1, 7), (3, 5), (3, 6), (7, 2), (8, 8), (5, 13), (0, 17)]:
        reg = new_reg(core, c)
        mean, cov = reg.sampler(5, burn, samples, 1, 1, 1, 1, 1)
        check(mean, cov, pos[burn:burn + samples])
        # the object keeps the last sweep's positions
        np.testing.assert_array_equal(reg.get_final_locations_as_numpy_array(),
                                      pos[burn + samples - 1].astype(np.float32))


def test_batch_of_chains_past_one_ring(core):
    c = make_case(shape=(9, 10, 11), K=8, L=6, seed=4)
    reg = new_reg(core, c)
    means, covs = reg.sampler_chains(5, 3, 2, 9, 1, 1, 1, 1, 1, per_chain=True, pooled=False)
    for chain in range(3):
        one = new_reg(core, c)
        one.set_chain(chain)
        mean, cov = one.sampler(5, 2, 9, 1, 1, 1, 1, 1)
        np.testing.assert_allclose(means[chain], mean, rtol=0, atol=1e-5)
        np.testing.assert_allclose(covs[chain], cov, rtol=0, atol=1e-4)
