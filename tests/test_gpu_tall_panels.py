"""The tallest factorisation panels (needs a B200: -m gpu): complex64, 38,016 rows, so that
the first 128 columns go through the shared-memory panel (more than 37,888 rows) and the
next ones through the grid panel with all 148 CTAs at 256 rows each, then fewer.

Tolerances: the first 256 columns hold no TF32 product of more than 128 inner columns.
Their factors satisfy |P A - L U| <= 4 sqrt(256) 2^-11 of |A| in the norm over 32
columns (as the complex64 factorisation test), the first 128, in FP32 throughout, 4
sqrt(128) 2^-24 of | |L||U| |; the solution's residual |b - A x| <= 4 sqrt(N) 2^-11 |A||x|."""
import os

import numpy as np
import pytest

import buffem
from test_gpu_parity import _chain_mesh

pytestmark = pytest.mark.gpu


class Device:
    def __init__(self, M):
        ptr, self.ld = M.device_ptr()
        self.__cuda_array_interface__ = {"shape": (M.NC, M.NR), "strides": (8 * self.ld, 8), "typestr": "<c8",
                                         "data": (ptr, False), "version": 2}


N = 37888 + 128


@pytest.fixture(scope="module")
def matrix(tmp_path_factory):
    path = os.path.join(str(tmp_path_factory.mktemp("tall")), "chain.vmsh")
    _chain_mesh(path, N)
    return buffem.SWGGeometry(meshfiles=path, materials=buffem.Material(eps=2.0)).AllocateVIEMatrix(buffem.BG_C64)


def view(F):
    import torch
    return torch.as_tensor(Device(F), device="cuda")   # [column, row]


def test_columns_without_a_number_keep_their_rows(matrix):
    """NaNs in column 40 make every later column one of NaNs: no candidate is left to
    name a row, and the interchanges stay inside the matrix."""
    import torch
    V = view(matrix)
    V.zero_()
    V.diagonal().fill_(2.0)
    V[40] = float("nan")
    torch.cuda.synchronize()
    matrix.LUFactorize()
    assert np.array_equal(matrix.pivots() - 1, np.arange(N))
    assert bool(torch.isnan(V[40:300, 41:N].abs()).all())
    V.zero_()
    torch.cuda.synchronize()


def test_panels_of_all_ctas(matrix):
    import torch
    F, V = matrix, view(matrix)
    g = torch.Generator(device="cuda").manual_seed(1)
    for c in range(0, N, 4096):
        V[c:c + 4096] = torch.randn(min(4096, N - c), N, dtype=torch.complex64, device="cuda", generator=g)
    A = V.clone()
    torch.cuda.synchronize()
    F.LUFactorize()
    piv = F.pivots() - 1
    perm = np.arange(N)
    for i, p in enumerate(piv):
        perm[[i, p]] = perm[[p, i]]
    perm = torch.tensor(perm, device="cuda")
    cols = V[:256].T.to(torch.complex128)              # N x 256
    L = torch.tril(cols, -1)
    L[range(256), range(256)] = 1
    U = torch.triu(cols[:256])
    assert L.abs().max() <= np.sqrt(2) * (1 + 1e-6)
    PA = A[:256].T[perm].to(torch.complex128)
    D = PA - L @ U
    assert D[:, :128].norm() <= 4 * np.sqrt(128) * 2.0 ** -24 * (L[:, :128].abs() @ U[:128, :128].abs()).norm()
    for c in range(0, 256, 32):
        assert D[:, c:c + 32].norm() <= 4 * np.sqrt(256) * 2.0 ** -11 * PA[:, c:c + 32].norm()
    assert int(piv[0]) == int((A[0].real.abs() + A[0].imag.abs()).argmax())
    B = np.asfortranarray((np.random.default_rng(2).normal(size=(N, 2)) + 0j).astype(np.complex64).astype(complex))
    X = B.copy(order="F")
    F.LUSolve(X)
    x = torch.tensor(X, device="cuda").to(torch.complex64)
    r = torch.tensor(B, device="cuda") - torch.vstack([A[:, c:c + 4096].T @ x for c in range(0, N, 4096)])
    assert r.norm() <= 4 * np.sqrt(N) * 2.0 ** -11 * float(A.abs().pow(2).sum(dtype=torch.float64)) ** 0.5 * x.norm()
