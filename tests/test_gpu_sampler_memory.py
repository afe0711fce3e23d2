"""Device memory of a sampler call.  The ring of positions takes up to eight slots of 12 B per voxel
and chain, as much as the FP64 mean and covariance that are staged for the copy back (96 B): it must
be back in the pool before these are taken, so that a call needs the larger of the two, not both.
Measured by the high-water mark of the device's default pool, which the library allocates from."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_parity import make_case, new_reg

pytestmark = pytest.mark.gpu

USED_CURRENT, USED_HIGH = 7, 8  # CUmemPool_attribute


class Pool:
    def __init__(self):
        self.cu = C.CDLL("libcuda.so.1")
        self.pool = C.c_void_p()
        assert self.cu.cuInit(0) == 0
        assert self.cu.cuDeviceGetDefaultMemPool(C.byref(self.pool), 0) == 0

    def get(self, attr):
        v = C.c_uint64()
        assert self.cu.cuMemPoolGetAttribute(self.pool, attr, C.byref(v)) == 0
        return v.value

    def peak(self, call):
        """bytes of the pool in use at the most during `call`, beyond those before it"""
        before = self.get(USED_CURRENT)
        assert self.cu.cuMemPoolSetAttribute(self.pool, USED_HIGH, C.byref(C.c_uint64(0))) == 0
        call()
        assert self.get(USED_CURRENT) == before
        return self.get(USED_HIGH) - before


def test_ring_is_back_before_the_staging(core):
    shape, chains = (40, 41, 42), 3
    V = int(np.prod(shape))
    reg = new_reg(core, make_case(shape=shape, seed=5))
    one = lambda: reg.sampler(3, 2, 9, 1, 1, 1, 1, 1)
    many = lambda: reg.sampler_chains(3, chains, 2, 9, 1, 1, 1, 1, 1)
    one(), many()  # what the object keeps for the next call
    pool = Pool()
    assert pool.peak(one) < 1.1 * 96 * V
    assert pool.peak(many) < 1.1 * 96 * V * chains
