"""Products on the INT8 tensor cores against FP64 ones (needs a B200: -m gpu).

C - A B through the public GEMM entry at sizes that take the split path: edges
of its 128 x 64 tiles, of the 16-column K blocks, of the 2,048-column K chunks
and of the 4,096-row and 4,096-column chunks.  Tolerances, per entry:
  * the FP64 reference is off by at most (K + 2) sqrt(2) 2^-52 (|A| |B|);
  * the split result by one rounding of C, 2^-53 of |C| and of the result, and
    the digit products it leaves out: 2 K terms of at most 9 x 2^14 x 2^-76 of
    the row's and the column's power-of-two scales (< 2 |max|), below
    2^-55 K max_k |A| max_k |B|.
"""
import pytest
import torch

import buffem

pytestmark = pytest.mark.gpu


def product(A, B, C):
    """C - A B by the library; column-major operands as transposed row-major ones"""
    (K, M), N = A.shape, B.shape[0]
    out = C.clone()
    torch.cuda.synchronize()
    buffem.zgemm_sub_device(M, N, K, A.data_ptr(), M, B.data_ptr(), K, out.data_ptr(), M)
    buffem.synchronize()
    return out.T


def draw(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, dtype=torch.complex128, device="cuda", generator=g)


def check(A, B, C, out):
    K = A.shape[0]
    a, b, c = A.T, B.T, C.T
    ref = c - a @ b
    bound = (K + 4) * 2 ** 0.5 * 2.0 ** -52 * (a.abs() @ b.abs() + c.abs())
    bound += 2.0 ** -55 * K * a.abs().amax(1)[:, None] * b.abs().amax(0)[None, :]
    assert bool(((out - ref).abs() <= bound).all())


@pytest.mark.parametrize("M,N,K", [(1024, 1024, 512), (1025, 1057, 521), (1151, 1000, 2100), (8200, 600, 240),
                                   (1000, 4130, 330), (4000, 900, 129)])
def test_split_product_matches_fp64(M, N, K):
    A, B, C = draw((K, M), 1), draw((N, K), 2), draw((N, M), 3)
    check(A, B, C, product(A, B, C))


def test_split_product_scales_and_special_values():
    """Rows and columns of very different size, zero rows, and rows and columns
    that hold an infinity or a NaN: those, and only those, are not finite."""
    M, N, K = 1100, 1090, 600
    A, B, C = draw((K, M), 4), draw((N, K), 5), draw((N, M), 6)
    A *= 10.0 ** torch.linspace(-120, 120, M, device="cuda", dtype=torch.float64)[None, :]
    B *= 10.0 ** torch.linspace(-120, 120, N, device="cuda", dtype=torch.float64)[:, None]
    A *= 10.0 ** torch.linspace(0, -6, K, device="cuda", dtype=torch.float64)[:, None]   # wide range inside a row
    A[:, 7] = 0
    B[9] = 0
    check(A, B, C, product(A, B, C))
    A[3, 70] = float("inf")
    B[800, 5] = float("nan")
    out = product(A, B, C)
    bad = torch.zeros(M, N, dtype=torch.bool, device="cuda")
    bad[70] = True
    bad[:, 800] = True
    assert not bool(torch.isfinite(out.abs())[bad].any())
    assert bool(torch.isfinite(out[~bad].abs()).all())
