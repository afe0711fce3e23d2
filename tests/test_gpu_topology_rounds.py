"""Topology correction's limiter rounds and folded FP64 Hartley passes against the FP64 oracle (the
reference's sequential walk, DFT Poisson solve): volumes whose cells fit one CTA's shared memory and
volumes whose do not, few and many folded corners, odd and even axes up to 250.  A wrong order of two
neighbouring cells, a lost cell or a misplaced coefficient is an error of 1e-3 and more; the two
solvers differ by rounding (1e-9, as in the golden test)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VS = (1.0, 1.25, 0.8)


def field(shape, rms, spacing, seed):
    from binder_b200 import phantoms
    rng = np.random.default_rng(seed)
    return (phantoms.identity_positions(shape).astype(np.float64) +
            phantoms.smooth_random_field(shape, rms, spacing, rng).astype(np.float64))


@pytest.mark.parametrize("shape,rms,spacing", [
    ((2, 2, 2), 1.5, 0.5), ((5, 4, 3), 1.0, 0.5), ((9, 16, 31), 0.8, 1.0), ((24, 23, 22), 1.2, 1.0),
    ((250, 4, 5), 0.8, 1.0), ((4, 131, 6), 0.8, 1.0), ((3, 5, 200), 0.8, 1.0),
    # more than 65,536 cells: a handful of folds, some thousands, and most of the volume
    ((43, 42, 41), 0.62, 3.0), ((43, 42, 41), 0.8, 2.0), ((43, 42, 41), 1.5, 1.0)])
def test_against_sequential_walk(core, oracle, shape, rms, spacing):
    f = field(shape, rms, spacing, sum(shape))
    tc = core.topology_correction_3D()
    got = tc.correct_topology(f, 0.05, 20.0, 1, 2, 1, VS, *shape)
    want, outer = oracle.topology3d(f, 0.05, 20.0, 1, 2, VS, shape)
    assert tc.last_stats["outer_iterations"] == outer
    np.testing.assert_allclose(got.ravel(), want, rtol=0, atol=1e-9)


def test_images(core, oracle):
    for shape in [(2, 2), (31, 18), (250, 9), (8, 129)]:
        f = field(shape, 1.0, 1.0, sum(shape))
        got = core.topology_correction_2D().correct_topology(f, 0.05, 20.0, 1, 2, 1, VS[:2], *shape)
        want, _ = oracle.topology2d(f, 0.05, 20.0, 1, 2, VS[:2], shape)
        np.testing.assert_allclose(got.ravel(), want, rtol=0, atol=1e-9)
