"""Scratch of a factorisation (needs a B200: -m gpu): taken from the stream-ordered
pool only where one of its products goes to the INT8 path, and enough for the
largest of those."""
import ctypes as C

import numpy as np
import pytest

import buffem
from test_gpu_parity import RawMatrix
from test_gpu_tiles import random_matrix

pytestmark = pytest.mark.gpu
USED_MEM_HIGH = 8      # CU_MEMPOOL_ATTR_USED_MEM_HIGH


class Pool:
    def __init__(self):
        self.cu, self.pool, dev = C.CDLL("libcuda.so.1"), C.c_void_p(), C.c_int()
        assert self.cu.cuDeviceGet(C.byref(dev), 0) == 0
        assert self.cu.cuDeviceGetDefaultMemPool(C.byref(self.pool), dev) == 0

    def reset(self):
        assert self.cu.cuMemPoolSetAttribute(self.pool, USED_MEM_HIGH, C.byref(C.c_uint64(0))) == 0

    def high(self):
        v = C.c_uint64()
        assert self.cu.cuMemPoolGetAttribute(self.pool, USED_MEM_HIGH, C.byref(v)) == 0
        return v.value


@pytest.mark.parametrize("N,digits", [(900, False), (1350, False), (1700, False), (2100, True)])
def test_scratch_only_for_products_that_use_it(N, digits):
    A = random_matrix(N, N).cpu().numpy()
    M = RawMatrix(N)
    M.upload(A)
    M.LUFactorize()      # workspace and kernel attributes in place
    M.upload(A)
    buffem.synchronize()
    pool = Pool()
    pool.reset()
    M.LUFactorize()
    high = pool.high()
    assert (high > 0) == digits
    x = np.asfortranarray(A @ np.ones((N, 1), complex))
    M.LUSolve(x)
    np.testing.assert_allclose(x, np.ones((N, 1)), rtol=0, atol=1e-9)
