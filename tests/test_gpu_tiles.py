"""Kernels at the edges of their tiles (needs a B200: -m gpu): factorisation
panels at the row counts where their layout changes, sweeps at remainders,
phases of the assembly and of the fields over their range, growth of the pair
table.

Tolerances, set before the first run: factors by ||PA - LU|| <= 4 sqrt(N) u
|| |L||U| || (u = 2^-53; complex64 as the factorisation test of the mixed form,
with TF32's 2^-11 and |A|), pivots equal to LAPACK's; solutions 1e-10 relative
(random matrices, condition about N); entries, fields and moments as in the
parity tests of each.  Matrix entries are compared up to |omega| = 4: the series
of the near pairs leaves the oracle's by 1e-7 at |omega| h around 10.
"""
import numpy as np
import pytest
import scipy.linalg as sl

import buffem
from test_gpu_fields import fields_close, points
from test_gpu_parity import RawMatrix, entry_close, pair

pytestmark = pytest.mark.gpu


def random_matrix(N, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(N, N, dtype=torch.complex128, device="cuda", generator=g)


def factors(LU, piv):
    """L, U and the row order of P A, on the device"""
    import torch
    lu = torch.tensor(LU, device="cuda").to(torch.complex128)
    perm = np.arange(len(piv))
    for i, p in enumerate(piv):
        perm[[i, p]] = perm[[p, i]]
    return torch.tril(lu, -1) + torch.eye(len(piv), dtype=lu.dtype, device="cuda"), torch.triu(lu), torch.tensor(perm)


# one and two CTAs of a cluster, remainders of a panel and of a 128-column
# block, 224- and 256-row layouts (16 CTAs of one cluster), the whole grid
@pytest.mark.parametrize("N", [127, 129, 161, 257, 3585, 4097])
def test_lu_panel_edges(N):
    A = random_matrix(N, N)
    M = RawMatrix(N)
    M.upload(A.cpu().numpy())
    M.LUFactorize()
    piv = M.pivots() - 1
    if N < 4000:
        assert np.array_equal(piv, sl.lu_factor(A.cpu().numpy())[1])
    L, U, perm = factors(M.download(), piv)
    bound = 4 * np.sqrt(N) * 2.0 ** -53 * (L.abs() @ U.abs()).norm()
    assert (A[perm.to(A.device)] - L @ U).norm() <= bound
    assert L.abs().max() <= np.sqrt(2) * (1 + 1e-12)


@pytest.mark.parametrize("N", [481, 7681, 8193])
def test_lu_c64_panel_edges(N):
    A = random_matrix(N, N)
    M = RawMatrix(N)
    M.upload(A.cpu().numpy())
    F = M.G.AllocateVIEMatrix(buffem.BG_C64).convert_from(M.M)
    F.LUFactorize()
    L, U, perm = factors(F.download(), F.pivots() - 1)
    assert (A[perm.to(A.device)] - L @ U).norm() <= 4 * np.sqrt(N) * 2.0 ** -11 * A.norm()
    assert L.abs().max() <= np.sqrt(2) * (1 + 1e-6)


@pytest.mark.parametrize("N", [1, 15, 17, 63, 64, 65, 130])
@pytest.mark.parametrize("nrhs", [1, 4, 5])
def test_sweep_remainders(N, nrhs):
    rng = np.random.default_rng(100 * N + nrhs)
    A = rng.normal(size=(N, N)) + 1j * rng.normal(size=(N, N)) + 2 * np.sqrt(N) * np.eye(N)
    B = np.asfortranarray(rng.normal(size=(N, nrhs)) + 1j * rng.normal(size=(N, nrhs)))
    want = np.linalg.solve(A, B)
    M = RawMatrix(N)
    M.upload(A)
    M.LUFactorize()
    M.LUSolve(B)
    assert np.linalg.norm(B - want) <= 1e-10 * np.linalg.norm(want)


# |k| times the extent of a pair: short series, series, sincos, complex k
@pytest.mark.parametrize("omega", [0.05, 0.9, 4.0, 1.2 + 0.3j])
def test_far_entries_over_the_phase_range(sphere, oracle_lib, omega):
    disp = np.array([[0, 0, 0], [0.2, 0.1, 3.0]], float)
    paths = [sphere(2, radius=1.0), sphere(3, radius=0.6)]
    Gb, Go = pair(paths, [buffem.Material(eps=3 + 0.1j)] * 2, [oracle_lib.material(eps=3 + 0.1j)] * 2, disp=disp,
                  oracle_lib=oracle_lib)
    ok, worst = entry_close(Gb.AssembleVIEMatrix(omega).download(), Go.assemble(complex(omega)))
    assert ok, worst


@pytest.mark.parametrize("omega", [0.05, 0.8, 3.0, 12.0, 2.0 + 0.5j])
def test_fields_over_the_phase_range(sphere, oracle_lib, omega):
    path = sphere(2, jitter=0.05, seed=9)
    Gb, Go = pair(path, buffem.Material(eps=4 + 0.2j), oracle_lib.material(eps=4 + 0.2j), oracle_lib=oracle_lib)
    rng = np.random.default_rng(2)
    J = rng.normal(size=Gb.TotalBFs) + 1j * rng.normal(size=Gb.TotalBFs)
    X = np.vstack([points(rng, 9, 0.0, 0.9), points(rng, 9, 1.05, 2.0), points(rng, 7, 5.0, 40.0)])
    fields_close(Gb.GetFields(None, J, omega, X), Go.get_fields(complex(omega), J, X, None, None))


def test_pair_table_grows(tmp_path, oracle_lib):
    """150 tetrahedra around one edge: every pair of them is near, more than
    the table holds at first."""
    n = 150
    t = 2 * np.pi * np.arange(n) / n
    V = np.vstack([[[0, 0, -0.5], [0, 0, 0.5]], np.column_stack([np.cos(t), np.sin(t), 0.3 * np.cos(5 * t)])])
    path = str(tmp_path / "fan.vmsh")
    with open(path, "w") as f:
        f.write("$MeshFormat\n2.2 0 8\n$EndMeshFormat\n$Nodes\n%d\n" % len(V))
        for i, v in enumerate(V):
            f.write("%d %.17g %.17g %.17g\n" % (i + 1, *v))
        f.write("$EndNodes\n$Elements\n%d\n" % n)
        for i in range(n):
            f.write("%d 4 2 0 1 1 2 %d %d\n" % (i + 1, 3 + i, 3 + (i + 1) % n))
        f.write("$EndElements\n")
    Gb, Go = pair(path, buffem.Material(eps=4.0), oracle_lib.material(eps=4.0), order=4, oracle_lib=oracle_lib)
    assert Gb.TotalBFs == n
    ok, worst = entry_close(Gb.AssembleVIEMatrix(0.8).download(), Go.assemble(0.8 + 0j))
    assert ok, worst


@pytest.mark.parametrize("n,z", [(2, 0.11), (3, 0.0637), (4, -0.21)])
def test_overlap_power_of_a_jump(sphere, oracle_lib, n, z):
    """eps that jumps across a plane through the cells: the overlap power takes
    every face's points by itself (no point of these meshes lies on the plane)."""
    kw = dict(eps=4 + 0.2j, eps2=12 + 1j, center=(0.0, 0.0, z))
    Gb, Go = pair(sphere(n), buffem.Material(kind=buffem.BG_MAT_JANUS_Z, **kw),
                  oracle_lib.material(kind=oracle_lib.MAT_JANUS_Z, **kw), oracle_lib=oracle_lib)
    rng = np.random.default_rng(n)
    J = rng.normal(size=Gb.TotalBFs) + 1j * rng.normal(size=Gb.TotalBFs)
    for omega in (0.9, 0.7 + 0.1j):
        got = Gb.GetPFTMatrix(J, omega, method=buffem.BG_PFT_OVERLAP)[0, 0]
        np.testing.assert_allclose(got, Go.pft_opft(complex(omega), J)[0], rtol=1e-9)
