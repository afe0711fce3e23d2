"""The M-step's scratch: one field's worth for the paired and the fused passes, a second one for the
per-axis passes, which an object gets when its precision (or its size) asks for them.  Device memory
by the default pool's bytes in use; results at a precision do not depend on the ones before it."""
import numpy as np
import pytest

from test_gpu_parity import make_case, new_reg
from test_gpu_sampler_memory import USED_CURRENT, Pool

pytestmark = pytest.mark.gpu


def prior(core, shape):
    dims = shape + (1,) * (3 - len(shape))
    return core.NonLinearTransformation(0.8, 0.6, 1.1, 1, 1, 1, 1, 1, 1,
                                        np.ones(shape, np.float32), *dims, 1, 0.6, 0.0)


@pytest.mark.parametrize("shape", [(40, 41, 42), (128, 100)])
def test_second_buffer_on_demand(core, shape):
    V, pool = int(np.prod(shape)), Pool()
    t = prior(core, shape)
    at_first = pool.get(USED_CURRENT)
    for p in (4, 3):
        t.set_precision(p)
    assert pool.get(USED_CURRENT) == at_first
    t.set_precision(1)
    more = pool.get(USED_CURRENT) - at_first
    # a fused image M-step needs none at any precision
    assert (12 * V <= more <= 12 * V + 512) if len(shape) == 3 else more == 0
    t.set_precision(0)
    assert pool.get(USED_CURRENT) == at_first + more


@pytest.mark.parametrize("order", [(3, 1, 0, 3, 2, 4), (0, 4, 2, 3, 1)])
def test_precisions_in_any_order(core, order):
    c = make_case(shape=(13, 14, 11), K=6, L=5, seed=2)
    reg = new_reg(core, c, c["d0"])
    for p in order:
        reg.set_precision(p)
        reg.reset()
        assert reg.EM(3, -1e300, 1, 0) == 3
        fresh = new_reg(core, c, c["d0"])
        fresh.set_precision(p)
        assert fresh.EM(3, -1e300, 1, 0) == 3
        np.testing.assert_array_equal(reg.get_final_locations_as_numpy_array(),
                                      fresh.get_final_locations_as_numpy_array())
        reg.reset()
        # (chains keep their own scratch, made for the precision of the call before)
        assert np.isfinite(reg.sampler_chains(5, 2, 1, 2, 0, 1, 1, 1, 1, per_chain=True,
                                              pooled=False)[0]).all()
