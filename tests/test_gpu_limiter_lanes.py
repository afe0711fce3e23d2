"""The limiter's rounds on images and on grids whose tables leave scratch for only some of the
groups of four lanes, with corners that the first and that only the last trials bring into range, against
the FP64 oracle (the reference's sequential walk).  A wrong order of two neighbouring cells, a lost
cell or a wrong trial is an error of 1e-3 and more; the Poisson solvers differ by rounding (1e-9, as
in the golden test)."""
import numpy as np
import pytest

from test_gpu_topology_rounds import VS, field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,rms,spacing,lo,hi", [
    ((2, 3), 1.0, 0.5, 0.05, 20.0), ((128, 128), 1.5, 1.0, 0.05, 20.0),
    ((256, 256), 1.2, 1.0, 0.05, 20.0), ((200, 37), 0.6, 3.0, 0.01, 100.0),
    ((40, 33), 0.8, 1.0, 0.95, 1.0), ((40, 33), 0.8, 1.0, 0.8, 1.2)])
def test_images(core, oracle, shape, rms, spacing, lo, hi):
    """A range that ends at 1 is reached by the last trials only (the identity)."""
    f = field(shape, rms, spacing, sum(shape))
    tc = core.topology_correction_2D()
    got = tc.correct_topology(f, lo, hi, 1, 2, 1, VS[:2], *shape)
    want, outer = oracle.topology2d(f, lo, hi, 1, 2, VS[:2], shape)
    assert tc.last_stats["outer_iterations"] == outer
    np.testing.assert_allclose(got.ravel(), want, rtol=0, atol=1e-9)


@pytest.mark.parametrize("shape,rms,lo,hi", [
    ((2, 256, 256), 0.8, 0.05, 20.0), ((41, 41, 41), 1.2, 0.05, 20.0),
    ((12, 11, 13), 0.8, 0.95, 1.0), ((12, 11, 13), 0.8, 0.8, 1.2), ((43, 42, 41), 0.8, 0.8, 1.2)])
def test_volumes(core, oracle, shape, rms, lo, hi):
    f = field(shape, rms, 1.0, sum(shape))
    tc = core.topology_correction_3D()
    got = tc.correct_topology(f, lo, hi, 1, 2, 1, VS, *shape)
    want, outer = oracle.topology3d(f, lo, hi, 1, 2, VS, shape)
    assert tc.last_stats["outer_iterations"] == outer
    np.testing.assert_allclose(got.ravel(), want, rtol=0, atol=1e-9)


@pytest.mark.parametrize("shape", [(256, 41, 42), (43, 200, 40), (41, 42, 223), (44, 192, 43)])
def test_hartley_forms(core, oracle, shape):
    """Axes of 13 to 17 row tiles on grids with a CTA of 32 lines for every SM."""
    f = field(shape, 0.62, 3.0, sum(shape))
    tc = core.topology_correction_3D()
    got = tc.correct_topology(f, 0.05, 20.0, 1, 1, 1, VS, *shape)
    want, outer = oracle.topology3d(f, 0.05, 20.0, 1, 1, VS, shape)
    assert tc.last_stats["outer_iterations"] == outer
    np.testing.assert_allclose(got.ravel(), want, rtol=0, atol=1e-9)


@pytest.mark.parametrize("vs", [(2.0, 0.5, 1.0), (2.0, 3.0, 1.0)])
def test_voxel_sizes(core, oracle, vs):
    """Voxel sizes that are all powers of two (no division) and not."""
    shape = (9, 16, 31)
    f = field(shape, 0.8, 1.0, 5)
    got = core.topology_correction_3D().correct_topology(f, 0.05, 20.0, 1, 2, 1, vs, *shape)
    want, _ = oracle.topology3d(f, 0.05, 20.0, 1, 2, vs, shape)
    np.testing.assert_allclose(got.ravel(), want, rtol=0, atol=1e-9)
