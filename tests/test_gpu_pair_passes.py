"""The paired DCT passes (two passes per launch, csrc/pair_transform.cu) against FP64 at the sizes
where their tiles, K steps and rings can go wrong: axes one short of and one past a 16-row K chunk,
a 32-row step and a 128-row tile, rows that are not whole float4, one-step and many-step products,
more tiles than SMs.

Tolerance.  A BF16 split keeps x = hi + lo with |x - hi - lo| <= 2^-18 |x|, and a product drops
lo * lo <= 2^-18: at most 3 * 2^-18 per product, of random sign, so 3 * 2^-18 of the 2-norm per
orthonormal pass and 6 * 3 * 2^-18 = 6.9e-5 over the six passes.  A misplaced row, column or chunk
is an error of the order of the field itself."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIGMA = math.sqrt(9.0 / (8.0 * math.pi))
REL = 6 * 3 * 2.0 ** -18
SHAPES = [(5, 16, 16), (3, 15, 17), (2, 31, 33), (4, 128, 129), (3, 129, 127), (33, 40, 36),
          (2, 200, 24), (3, 24, 200), (161, 9, 130), (129, 130, 7), (240, 5, 3), (2, 208, 160)]


def case(shape, seed):
    from binder_b200.utils import initialize_fourier_domain_smoothing
    rng = np.random.default_rng(seed)
    field = rng.standard_normal(shape + (3,)).astype(np.float32)
    D = initialize_fourier_domain_smoothing(shape, True, 2, 3).astype(np.float32)
    return field, D, (0.7, 1.3, 0.9)


def close(got, want):
    got, want = np.asarray(got, np.float64).ravel(), np.asarray(want).ravel()
    assert np.linalg.norm(got - want) <= REL * np.linalg.norm(want)
    # no single value far off either: 40 times the mean-square bound
    assert np.abs(got - want).max() <= 40 * REL * max(np.abs(want).max(), 1e-30)


@pytest.mark.parametrize("shape", SHAPES)
def test_smoothing_matches_fp64(core, oracle, shape):
    field, D, gamma = case(shape, sum(shape))
    t = core.NonLinearTransformation(*gamma, 1, 1, 1, 1, 1, 1, D, *shape, 1, SIGMA, 0.0)
    cost, out = t.smooth_deformation(field)
    want_cost, want = oracle.smooth(field, np.zeros(field.size), D, gamma, SIGMA, shape)
    close(out, want)
    assert cost == pytest.approx(want_cost, rel=10 * REL)


@pytest.mark.parametrize("shape", [(3, 15, 17), (4, 128, 129), (33, 40, 36)])
def test_prior_samples_match_fp64(core, oracle, shape):
    field, D, gamma = case(shape, 7 + sum(shape))
    t = core.NonLinearTransformation(*gamma, 1, 1, 1, 1, 1, 1, D, *shape, 1, SIGMA, 0.0)
    got = t.sampleDeformationField(field, 2)
    close(got, oracle.sample_field(field, D, gamma, SIGMA, shape, 2))


@pytest.mark.parametrize("shape", [(200, 130), (130, 200), (17, 240)])
def test_images_past_the_fused_size(core, oracle, shape):
    """An image with an axis over 128: its x passes are one paired launch."""
    from binder_b200.utils import initialize_fourier_domain_smoothing
    rng = np.random.default_rng(shape[0])
    field = rng.standard_normal(shape + (2,)).astype(np.float32)
    D = initialize_fourier_domain_smoothing(shape, True, 2, 2).astype(np.float32)
    t = core.NonLinearTransformation(0.7, 1.3, 0.9, 1, 1, 1, 1, 1, 1, D, *shape, 1, 1, SIGMA, 0.0)
    cost, out = t.smooth_deformation(field)
    vs = (*shape, 1)
    want_cost, want = oracle.smooth(field, np.zeros(field.size), D, (0.7, 1.3), SIGMA, vs)
    close(out, want)
    assert cost == pytest.approx(want_cost, rel=10 * REL)
