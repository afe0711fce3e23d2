"""The fused 2D M-step's tiles: images whose rows and columns leave part of a CTA's slab, part of a
vector or whole CTAs of the cluster empty, in both cluster sizes, against the FP64 transform."""
import numpy as np
import pytest
from scipy.fft import dctn, idctn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cluster", ["", "8"])
@pytest.mark.parametrize("shape", [(1, 7), (4, 4), (5, 3), (33, 17), (64, 127), (100, 36),
                                   (127, 65), (128, 128)])
def test_smoothing(core, monkeypatch, shape, cluster):
    """FP32 products of at most 128 terms in four passes: each rounds to 128 * 2^-24 of the sum of
    magnitudes, at most 128^(1/2) times the field's largest value (an orthonormal row has an
    l1 norm of n^(1/2)), so 4 * 128 * 2^-24 * 11.3 * 5 < 2e-3; typical errors are the square root
    of the term count, well under 1e-4."""
    monkeypatch.setenv("BINDER_B200_FUSED2D", cluster)
    rng = np.random.default_rng(shape[0] * 131 + shape[1])
    field = rng.standard_normal(shape + (2,)).astype(np.float32)
    D = rng.uniform(0.0, 4.0, shape).astype(np.float32)
    gamma, sigma = 0.3, 0.6
    tr = core.NonLinearTransformation(gamma, gamma, gamma, 1, 1, 1, 1, 1, 1, D, *shape, 1, 1,
                                      sigma, 0.0)
    cost, out = tr.smooth_deformation(field)
    want_cost = 0.0
    for c in range(2):
        w = dctn(field[..., c].astype(np.float64), norm="ortho")
        w /= 1.0 + gamma * sigma ** 2 * D.astype(np.float64)
        want_cost += 0.5 * gamma * (D.astype(np.float64) * w * w).sum()
        got = np.asarray(out)[..., 0, c] if np.ndim(out) == 4 else np.asarray(out)[..., c]
        np.testing.assert_allclose(got, idctn(w, norm="ortho"), rtol=0, atol=1e-4)
    assert cost == pytest.approx(want_cost, rel=1e-5)
