"""Volumes whose planes do not fit the paired DCT passes (the two operand planes, two steps of each
ring and the matrices in 226 KB of shared memory; (y, z) = (240, 200) in the forward pass, (256, 256)
in both): BF16 operands then run the per-axis passes, a component per graph branch, and the samplers
keep one slot of positions.

Tolerances as in the tests of the paired passes: the two make the same products in the same order."""
import numpy as np
import pytest

from test_gpu_pair_passes import REL, SIGMA, case, close
from test_gpu_parity import make_case, new_reg

pytestmark = pytest.mark.gpu

SHAPES = [(3, 240, 200), (2, 256, 256), (2, 200, 256)]


@pytest.mark.parametrize("shape", SHAPES)
def test_smoothing_and_prior_samples_match_fp64(core, oracle, shape):
    field, D, gamma = case(shape, sum(shape))
    t = core.NonLinearTransformation(*gamma, 1, 1, 1, 1, 1, 1, D, *shape, 1, SIGMA, 0.0)
    cost, out = t.smooth_deformation(field)
    want_cost, want = oracle.smooth(field, np.zeros(field.size), D, gamma, SIGMA, shape)
    close(out, want)
    assert cost == pytest.approx(want_cost, rel=10 * REL)
    close(t.sampleDeformationField(field, 2), oracle.sample_field(field, D, gamma, SIGMA, shape, 2))


def test_em_and_samplers(core, oracle):
    shape = (2, 256, 256)
    c = make_case(shape=shape, K=8, L=6, seed=3)
    reg = new_reg(core, c)
    assert reg.EM(3, -1e30, 1, 0) == 3
    it, final, theta, _ = oracle.em(c["d0"], c["grid"], c["u"], c["v"], c["theta"], 2.0, c["D"],
                                    c["gamma"], SIGMA, shape, shape, 8, 6, float(np.prod(shape)),
                                    3, -1e30)
    np.testing.assert_allclose(reg.get_final_locations_as_numpy_array().ravel(), final, rtol=0,
                               atol=1e-3)
    np.testing.assert_allclose(reg.get_likelihood_parameters(), theta, rtol=1e-3, atol=1e-6)
    # a batch of chains is its chains one by one
    means, covs = new_reg(core, c).sampler_chains(5, 2, 1, 3, 0, 1, 1, 1, 1, per_chain=True,
                                                  pooled=False)
    for chain in range(2):
        one = new_reg(core, c)
        one.set_chain(chain)
        mean, cov = one.sampler(5, 1, 3, 0, 1, 1, 1, 1)
        np.testing.assert_allclose(means[chain], mean, rtol=0, atol=1e-5)
        np.testing.assert_allclose(covs[chain], cov, rtol=0, atol=1e-4)
