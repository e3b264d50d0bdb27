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
USED_MEM_CURRENT, USED_MEM_HIGH = 7, 8      # CU_MEMPOOL_ATTR_USED_MEM_CURRENT, _HIGH


class Pool:
    def __init__(self):
        self.cu, self.pool, dev = C.CDLL("libcuda.so.1"), C.c_void_p(), C.c_int()
        assert self.cu.cuDeviceGet(C.byref(dev), 0) == 0
        assert self.cu.cuDeviceGetDefaultMemPool(C.byref(self.pool), dev) == 0

    def reset(self):
        assert self.cu.cuMemPoolSetAttribute(self.pool, USED_MEM_HIGH, C.byref(C.c_uint64(0))) == 0

    def get(self, what):
        v = C.c_uint64()
        assert self.cu.cuMemPoolGetAttribute(self.pool, what, C.byref(v)) == 0
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
    held = pool.get(USED_MEM_CURRENT)      # by objects of other tests
    M.LUFactorize()
    assert (pool.get(USED_MEM_HIGH) > held) == digits
    x = np.asfortranarray(A @ np.ones((N, 1), complex))
    M.LUSolve(x)
    np.testing.assert_allclose(x, np.ones((N, 1)), rtol=0, atol=1e-9)


def test_sweep_tunes_only_what_the_size_reaches(sphere):
    """A first sweep of a size class on one slot records the job's launches once for the
    tuning job and once for the sweep (no panel height and no GEMM tile to choose at
    N = 2,376), a later one once."""
    wave = buffem.PlaneWave([1, 0, 0], [0, 0, 1])
    small = buffem.SWGGeometry(meshfiles=sphere(2), materials=buffem.Material(eps=4 + 0.2j))
    buffem.BatchSweep([small], [0.5, 0.6], wave, max_streams=1)      # kernel attributes and tables in place
    G = buffem.SWGGeometry(meshfiles=sphere(6), materials=buffem.Material(eps=4 + 0.2j))
    G.precompute()
    omegas = np.linspace(0.5, 1.0, 14)
    n = [buffem.launch_count()]
    for _ in range(2):
        buffem.BatchSweep([G], omegas, wave, max_streams=1)
        n.append(buffem.launch_count())
    assert n[1] - n[0] <= 2 * (n[2] - n[1])
