"""Digit products on operands of uneven scale (needs a B200: -m gpu): exact sums,
inner, row and column scales, patterns that no scaling evens out, factors of
systems with rows and columns of two sizes.

Tolerances, by real and imaginary part, set before the first run:
  * operands whose digits are chosen so that nothing is left out and only the last
    operation rounds: equality with the correctly rounded sum;
  * else (K + 4) 2^-52 (S + |C|), S the sum of the 2K real terms' sizes: what a
    chain of FP64 operations is allowed (gamma_2K S) and the roundings of C; tiles in
    which the digits could lose more go to FP64;
  * factors: (N + 4) sqrt(2) 2^-52 |L||U| entry by entry, the bound of Gaussian
    elimination in complex FP64 arithmetic.
"""
import numpy as np
import pytest
import scipy.linalg as sl

import buffem
from test_gpu_parity import RawMatrix
from test_gpu_tiles import factors, random_matrix

pytestmark = pytest.mark.gpu
LD = np.longdouble


def product(A, B, C):
    """C - A B (A: K x M, B: N x K, C: N x M, transposed row-major) and the launches it took"""
    import torch
    (K, M), N = A.shape, B.shape[0]
    out = C.clone()
    torch.cuda.synchronize()
    n0 = buffem.launch_count()
    buffem.zgemm_sub_device(M, N, K, A.data_ptr(), M, B.data_ptr(), K, out.data_ptr(), M)
    buffem.synchronize()
    return out, buffem.launch_count() - n0


def sample(n, count):
    return np.unique(np.r_[0:n:max(1, n // count), n - 1])


def draws(M, N, K, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, dtype=torch.complex128, device="cuda", generator=g)
    return r(K, M), r(N, K), r(N, M)


def inner(A, B, C):
    import torch
    d = 10.0 ** torch.linspace(0, -12, A.shape[0], device="cuda", dtype=torch.float64)
    return A / d[:, None], B * d[None], 0 * C


def rows_and_columns(A, B, C):
    import torch
    t = lambda n, s: 10.0 ** torch.linspace(-s, s, n, device="cuda", dtype=torch.float64)
    return A * t(A.shape[1], 120)[None], B * t(B.shape[0], -120)[:, None], 0 * C


def blocks(A, B, C):
    """(1, s) over (s, 1): no diagonal matrix between A and B evens it out"""
    k, m, n = A.shape[0] // 2, A.shape[1] // 2, B.shape[0] // 2
    A, B = A.clone(), B.clone()
    A[:k, m:] *= 1e-9
    A[k:, :m] *= 1e-9
    B[n:, :k] *= 1e-9
    B[:n, k:] *= 1e-9
    return A, B, 0 * C


def small_imaginary(A, B, C):
    import torch
    return torch.complex(A.real, 1e-9 * A.imag), torch.complex(B.real, 1e-7 * B.imag), 0 * C


def zeros(A, B, C):
    A, B = A.clone(), B.clone()
    A[:, 7] = 0
    A[5] = 0
    B[9] = 0
    B[:, 11] = 0
    return A, B, C


KINDS = {"plain": lambda A, B, C: (A, B, C), "inner": inner, "rows_and_columns": rows_and_columns, "blocks": blocks,
         "small_imaginary": small_imaginary, "zeros": zeros}


@pytest.mark.parametrize("M,N,K", [(1151, 1000, 2100), (1351, 673, 712)])
@pytest.mark.parametrize("kind", KINDS)
def test_parts_of_products(M, N, K, kind):
    A, B, C = KINDS[kind](*draws(M, N, K, 3))
    out, launches = product(A, B, C)
    assert launches >= 7            # the digit path: an FP64 product is one launch
    i, j = sample(M, 32), sample(N, 32)
    a, b = A[:, i].T.cpu().numpy(), B[j].T.cpu().numpy()
    c, o = (X[j][:, i].T.cpu().numpy() for X in (C, out))
    ar, ai, br, bi = (x.astype(LD) for x in (a.real, a.imag, b.real, b.imag))
    u = (K + 4) * 2.0 ** -52
    assert np.all(np.abs(o.real - (c.real - (ar @ br - ai @ bi))) <=
                  u * (abs(ar) @ abs(br) + abs(ai) @ abs(bi) + abs(c.real)))
    assert np.all(np.abs(o.imag - (c.imag - (ar @ bi + ai @ br))) <=
                  u * (abs(ar) @ abs(bi) + abs(ai) @ abs(br) + abs(c.imag)))


@pytest.mark.parametrize("M,N,K", [(1351, 673, 712)])
def test_every_sum_of_digits(M, N, K):
    """Entries n 256^-i, n = -3 .. 3, with i + j <= 7 for every term: one digit
    each, all eight sums of digit products in use, no product left out.  The sums
    of each half are exact in FP64, so the result is the exact sum rounded once."""
    import torch
    rng = np.random.default_rng(8)
    top = np.arange(K) % 8

    def operand(rows, limit):
        n = rng.integers(-3, 4, size=(2, rows, K))
        i = rng.integers(0, limit + 1, size=(2, rows, K))
        n[:, :2], i[:, :2] = 3, 0          # every row of the inner index has the same largest part
        i[:, :, 0] = 0
        n[:, :, 0] = 3                     # and every row and column the same scale
        return n, i

    (an, ae), (bn, be) = operand(M, top), operand(N, 7 - top)
    num = lambda n, e: torch.tensor((n[0] * 256.0 ** -e[0]) + 1j * (n[1] * 256.0 ** -e[1]), device="cuda")
    A, B = num(an, ae).T.contiguous(), num(bn, be)
    out, launches = product(A, B, torch.zeros(N, M, dtype=torch.complex128, device="cuda"))
    assert launches >= 7
    out = out.T.cpu().numpy()
    for m in sample(M, 12):
        for n in sample(N, 12):
            def dot(p, q):
                return sum(int(x) * int(y) << (56 - 8 * int(s)) for x, y, s in zip(an[p, m], bn[q, n], ae[p, m] + be[q, n]))
            # int / int rounds correctly
            assert out[m, n].real == (dot(1, 1) - dot(0, 0)) / 2 ** 56
            assert out[m, n].imag == -(dot(0, 1) + dot(1, 0)) / 2 ** 56


@pytest.mark.parametrize("both", [True, False])
@pytest.mark.parametrize("ratio", [1.0, 1e-6, 1e-8, 1e-12, 1e-16])
def test_factors_of_two_sizes(both, ratio):
    """A symmetric random, rows (and columns) past 700 scaled: diagonal entries of the
    given ratio, as of bodies whose cells differ in size."""
    N = 2100
    A = random_matrix(N, 4).cpu().numpy()
    A = A + A.T
    d = np.where(np.arange(N) < 700, 1.0, np.sqrt(ratio) if both else ratio)
    A = d[:, None] * A * (d[None] if both else 1.0)
    M = RawMatrix(N)
    M.upload(A)
    M.LUFactorize()
    piv = M.pivots() - 1
    assert np.array_equal(piv, sl.lu_factor(A)[1])
    L, U, perm = factors(M.download(), piv)
    rows = sample(N, 20)
    size = (L.abs() @ U.abs()).cpu().numpy()[rows]
    L, U, PA = L.cpu().numpy()[rows], U.cpu().numpy(), A[perm.numpy()[rows]]
    lr, li, ur, ui = (x.astype(LD) for x in (L.real, L.imag, U.real, U.imag))
    err = np.hypot(PA.real - (lr @ ur - li @ ui), PA.imag - (lr @ ui + li @ ur))
    assert np.all(err <= (N + 4) * 2 ** 0.5 * 2.0 ** -52 * size)
