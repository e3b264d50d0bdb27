"""
A matrix copied from the host is all there before the first kernel reads it.

The copy comes from pageable memory, and such a copy may return while its last
bytes are still on their way to the device; the library's stream has to wait
for them.  Rounding to complex64 right after the upload is the shortest kernel
that reads the whole matrix: what it read shows in its result, to the bit.
"""
import numpy as np
import pytest

import buffem
from test_gpu_parity import RawMatrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [96, 257, 258, 289, 700])
def test_upload_is_complete_before_the_next_kernel(N):
    rng = np.random.default_rng(N)
    M = RawMatrix(N)
    F = M.G.AllocateVIEMatrix(buffem.BG_C64)
    for rep in range(24):
        # other numbers each time: a column left from before is seen
        A = rng.normal(size=(N, N)) + 1j * rng.normal(size=(N, N))
        M.upload(A)
        F.convert_from(M.M)
        stale = np.flatnonzero((F.download() != A.astype(np.complex64)).any(axis=0))
        assert stale.size == 0, f"pass {rep}: columns {stale[:4]}...{stale[-1]} are not the uploaded ones"
