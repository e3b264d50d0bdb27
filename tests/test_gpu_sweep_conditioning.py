"""Triangular sweeps with ill-conditioned diagonal blocks (needs a B200: -m gpu).

Triangular systems whose factors are themselves (no interchange), right-hand
sides of known solutions.  Tolerance, set before the first run: substitution leaves
|b - T x| <= (N + 4) 2 sqrt(2) u |T||x| entry by entry whatever the condition (u =
2^-53, complex64 2^-24; complex products cost sqrt(2) more than real ones).
In complex64 only the systems whose solutions by substitution stay in its range."""
import numpy as np
import pytest

import buffem
from test_gpu_parity import RawMatrix

pytestmark = pytest.mark.gpu


def upper(N, diag, rng):
    A = np.triu(rng.normal(size=(N, N)) + 1j * rng.normal(size=(N, N)), 1)
    return A + np.diag(diag * np.exp(2j * np.pi * rng.random(N)))


def lower(N, size, rng):
    # pivots 1, the largest of their columns by |re| + |im|
    return np.tril(-size * (1 - 0.05 * rng.random((N, N))), -1) * (1 + 0j) + np.eye(N)


SYSTEMS = [("upper", 8.0), ("upper", 1.0), ("upper", 0.3), ("upper", 0.1), ("upper", 0.01), ("lower", 0.3), ("lower", 0.95)]
RANGE64 = {("upper", 0.3): (64,), ("upper", 0.1): (), ("upper", 0.01): ()}


@pytest.mark.parametrize("c64,N,kind,size", [(c64, N, k, s) for c64 in (False, True) for N in (64, 130) for k, s in SYSTEMS
                                             if not c64 or N in RANGE64.get((k, s), (64, 130))])
@pytest.mark.parametrize("nrhs", [1, 4])
def test_residual_is_that_of_substitution(c64, N, kind, size, nrhs):
    rng = np.random.default_rng(N + nrhs)
    T = {"upper": upper, "lower": lower}[kind](N, size, rng)
    # few columns beyond a diagonal block, so that solutions stay in range
    T[np.arange(N)[:, None] // 16 != np.arange(N)[None] // 16] *= 1e-3
    if c64:
        T = T.astype(np.complex64).astype(complex)
    x = rng.normal(size=(N, nrhs)) + 1j * rng.normal(size=(N, nrhs))
    B = np.asfortranarray(T @ x)
    if c64:
        B = np.asfortranarray(B.astype(np.complex64).astype(complex))
    M = RawMatrix(N)
    M.upload(T)
    F = M.G.AllocateVIEMatrix(buffem.BG_C64).convert_from(M.M) if c64 else M
    F.LUFactorize()
    assert np.array_equal(F.pivots() - 1, np.arange(N))
    X = B.copy(order="F")
    F.LUSolve(X)
    u = 2.0 ** -24 if c64 else 2.0 ** -53
    assert np.all(np.isfinite(X))
    assert np.all(np.abs(B - T @ X) <= (N + 4) * 2 * 2 ** 0.5 * u * (np.abs(T) @ np.abs(X)))
