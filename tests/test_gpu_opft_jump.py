"""Overlap power where the permittivity jumps through points of the rule (needs a
B200: -m gpu).  In spheres of an odd number of cells the middle layer straddles
z = 0 and points of the 33-point rule lie on that plane up to rounding: the side
they take is that of the coordinate rounded from the face's own vertex, QA + (u . L),
each face by itself, as the oracle has it.  A coordinate rounded from another vertex
puts some of them on the other side (at 9 and 11 cells the power moves by 2e-6 to
1e-4; at 3 to 7 cells it happens not to).

Tolerance: both sides add the same terms in FP64 in another order: 1e-9."""
import numpy as np
import pytest

import buffem
from test_gpu_parity import pair

pytestmark = pytest.mark.gpu


def height(n):
    """|z| of the centroids, which are points of the rule"""
    from meshgen import sphere_arrays
    V, T = sphere_arrays(n)
    return np.abs(V[T].mean(1)[:, 2])


@pytest.mark.parametrize("cells,radius", [((9,), 1.0), ((9,), 0.8), ((11,), 1.0), ((9, 5), 0.8)])
def test_points_on_the_jump(sphere, oracle_lib, cells, radius):
    kw = dict(eps=4 + 0.2j, eps2=12 + 1j, center=(0.0, 0.0, 0.0))
    meshes = [sphere(n, radius=radius) for n in cells]
    disp = [[2.5 * i, 0.0, 0.0] for i in range(len(cells))]
    Gb, Go = pair(meshes, [buffem.Material(kind=buffem.BG_MAT_JANUS_Z, **kw)] * len(cells),
                  [oracle_lib.material(kind=oracle_lib.MAT_JANUS_Z, **kw)] * len(cells), disp=disp, oracle_lib=oracle_lib)
    assert all(height(n).min() < 1e-15 for n in cells)
    rng = np.random.default_rng(sum(cells))
    J = rng.normal(size=Gb.TotalBFs) + 1j * rng.normal(size=Gb.TotalBFs)
    for omega in (0.9, 0.7 + 0.1j):
        got = Gb.GetPFTMatrix(J, omega, method=buffem.BG_PFT_OVERLAP)[:, 0]
        np.testing.assert_allclose(got, Go.pft_opft(complex(omega), J), rtol=1e-9)


def test_tetrahedron_without_basis_functions(sphere, tmp_path):
    """An object of one tetrahedron has no basis function and absorbs nothing, also
    where its permittivity is that of vacuum."""
    path = str(tmp_path / "one.vmsh")
    with open(path, "w") as f:
        f.write("$MeshFormat\n2.2 0 8\n$EndMeshFormat\n$Nodes\n4\n1 0 0 0\n2 1 0 0\n3 0 1 0\n4 0 0 1\n$EndNodes\n"
                "$Elements\n1\n1 4 2 0 1 1 2 3 4\n$EndElements\n")
    G = buffem.SWGGeometry(meshfiles=[sphere(2), path], materials=[buffem.Material(eps=4 + 0.2j), buffem.Material(eps=1.0)],
                           displacements=[[0, 0, 0], [0, 0, 3.0]])
    alone = buffem.SWGGeometry(meshfiles=sphere(2), materials=buffem.Material(eps=4 + 0.2j))
    J = np.exp(1j * np.arange(G.TotalBFs))
    got = G.GetPFTMatrix(J, 0.9, method=buffem.BG_PFT_OVERLAP)[:, 0]
    assert got[1] == 0
    np.testing.assert_allclose(got[0], alone.GetPFTMatrix(J, 0.9, method=buffem.BG_PFT_OVERLAP)[0, 0], rtol=1e-13)
