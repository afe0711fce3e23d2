"""An axis of more than 256 points is refused on the host, at every transform precision, before a
kernel of the M-step is launched: it is past the columns of an MMA and the rows of an FP32 slab."""
import numpy as np
import pytest

from test_gpu_parity import make_case, new_reg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(257, 3, 4), (3, 300, 4), (2, 3, 264), (300, 20), (20, 257)])
@pytest.mark.parametrize("precision", [0, 1, 2, 3, 4])
def test_prior_refuses(core, shape, precision):
    dims = shape + (1,) * (3 - len(shape))
    N = len(shape)
    t = core.NonLinearTransformation(1.0, 1.0, 1.0, 1, 1, 1, 1, 1, 1,
                                     np.ones(shape, np.float32), *dims, 1, 0.6, 0.0)
    t.set_precision(precision)
    field = np.ones(shape + (N,), np.float32)
    with pytest.raises(Exception, match=r"axis length must be in \[1, 256\]"):
        t.smooth_deformation(field)
    with pytest.raises(Exception, match=r"axis length must be in \[1, 256\]"):
        t.sampleDeformationField(field, 1)


def test_registration_refuses_and_stays_usable(core):
    reg = new_reg(core, make_case(shape=(5, 257, 6), seed=1))
    for _ in range(2):
        with pytest.raises(Exception, match=r"axis length must be in \[1, 256\]"):
            reg.EM(1, -1e30, 1, 0)
    assert np.isfinite(reg.get_final_locations_as_numpy_array()).all()
    with pytest.raises(Exception, match=r"axis length must be in \[1, 256\]"):
        reg.sampler(1, 1, 1, 1, 1, 1, 1, 1)
    other = new_reg(core, make_case(shape=(5, 7, 6), seed=1))
    assert other.EM(1, -1e30, 1, 0) == 1
