"""EM E-steps of voxels whose total weight is far below FP32's smallest normal reciprocal range: the
whole neighbourhood meets theta entries that are tiny, so 1 / S times the histogram's fixed-point
scale is past FP32's largest number although every posterior is an ordinary one.  Against the FP64
oracle.  Tolerances of the other one-iteration tests (FP32 weights; the product of four channels'
entries adds three roundings of 6e-8)."""
import numpy as np
import pytest

from test_gpu_edge_cases import one_iteration
from test_gpu_mi_filter import filter_case, new_filter_reg, oracle_iteration
from test_gpu_parity import make_case

pytestmark = pytest.mark.gpu


def floored(M, K, L, floor, v, u):
    """theta with `floor` off the diagonal, and half the volume's bins off it in every channel"""
    th = np.full((M, K, L), floor)
    for k in range(K):
        th[:, k, k % L] = 1.0 - (L - 1) * floor
    v, u = v.copy(), u.copy()
    half = v.shape[0] // 2
    v[:half], u[:half] = 1 + v[:half] % 2, 0
    return th.astype(np.float32), v, u


@pytest.mark.parametrize("M,floor", [(4, 1e-8), (4, 4e-9), (3, 1e-11), (2, 1e-16)])
def test_filter_channels(core, oracle, M, floor):
    c = filter_case(K=8, L=6, M=M, seed=M)
    V = int(np.prod(c["shape"]))
    c["thf"], v, u = floored(M, 8, 6, floor, c["vf"].reshape(V, M), c["uf"].reshape(V, M))
    c["vf"], c["uf"] = v.ravel(), u.ravel()
    reg = new_filter_reg(core, c)
    assert reg.EM(1, -1e30, 1, 0) == 1
    mll, dream, th, _, final, deg = oracle_iteration(oracle, c, c["d0"].astype(np.float64),
                                                     c["thf"].astype(np.float64))
    assert deg == 0
    np.testing.assert_allclose(reg.get_dream_locations(), dream, rtol=0, atol=5e-5)
    np.testing.assert_allclose(reg.get_likelihood_parameters(), th, rtol=1e-4, atol=1e-6)
    np.testing.assert_allclose(reg.get_final_locations_as_numpy_array().ravel(), final, rtol=0,
                               atol=2e-4)
    assert reg.iteration_stats()[0][0] == pytest.approx(mll, rel=1e-6)


@pytest.mark.parametrize("shape", [(12, 10, 9), (97, 97, 97)])
def test_one_channel(core, oracle, shape):
    """The 256- and the 768-thread form."""
    c = make_case(shape=shape, K=8, L=6, seed=7)
    V = int(np.prod(shape))
    th, v, u = floored(1, 8, 6, 1e-33, c["v"].reshape(V, 1), c["u"].reshape(V, 1))
    c["theta"] = th[0]
    c["v"], c["u"] = v.reshape(c["v"].shape), u.reshape(c["u"].shape)
    one_iteration(core, oracle, c)
