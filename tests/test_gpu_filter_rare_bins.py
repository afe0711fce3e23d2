"""The MI filter histogram's rare cells, with as many voxels to a CTA as the 1 mm volumes have: pairs of
bins whose whole mass is made of posteriors of 1e-9 to 1e-4, cell by cell against the FP64 oracle
(alpha 1: theta is the histogram's row over its sum, nothing hides a cell).

Tolerance: a mass is a product of two spline factors and two theta entries over a sum of 64 such
(some fifteen roundings of 6e-8, and the spline's own): 1e-5 of the cell.  It is then rounded to a
multiple of 2^-27, at most 2^-28 off for a voxel that has the pair and of either sign; with all but
those left out, 2^-29 per voxel of the volume over the row's sum."""
import numpy as np
import pytest

from test_gpu_mi_filter import filter_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,grid", [((32, 32, 32), 1), ((40, 41, 42), 2), ((32, 32, 32), 0)])
def test_rare_cells(core, oracle, shape, grid):
    K = L = 16
    M = 2
    c = filter_case(shape=shape, K=K, L=L, M=M, seed=9)
    V = int(np.prod(shape))
    rng = np.random.default_rng(1)
    th = 10.0 ** rng.uniform(-7.0, -3.0, (M, K, L))
    for k in range(K):
        th[:, k, k] = 1.0
    c["thf"] = (th / th.sum(-1, keepdims=True)).astype(np.float32)
    reg = core.Registration(c["d0"], 1, c["grid"], c["grid"], *shape, *shape, 3, float(V))
    reg.setNonLinearTransformation(*c["gamma"], 1, 1, 1, 1, 1, 1, c["D"])
    reg.setMILikelihoodFilter(1.0, c["thf"], 1, c["vf"], c["uf"], K, L, M)
    if grid:
        reg.set_estep_grid(grid)
    assert reg.EM(1, -1e30, 1, 0) == 1
    _, _, hist, _ = oracle.estep_filter(c["d0"].astype(np.float64), c["uf"], c["vf"],
                                        c["thf"].astype(np.float64), shape, shape, K, L, M)
    hist = hist.reshape(M * K, L)
    rows = hist.sum(1, keepdims=True)
    assert (rows > 1.0).all() and np.median(hist[hist < 0.1]) > 1e-6
    want = hist / rows
    got = reg.get_likelihood_parameters().reshape(M * K, L)
    worst = np.abs(got - want) / (1e-5 * want + V * 2.0 ** -29 / rows)
    assert worst.max() < 1.0, worst.max()
