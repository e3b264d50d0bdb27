"""EMT pair sums through tetrahedra against the oracle's pair-by-pair sums:
every polynomial length, the sincos form, the switch to the pair-by-pair
kernels at |omega| R = 5, one to three objects (tiles with remainders, several
object pairs), currents and general (non-Hermitian) dressed Rytov matrices.

Tolerance: both sides add the same terms in FP64 in another order: 1e-9 of
the largest entry of a column kind, as the other EMT tests."""
import ctypes as C

import numpy as np
import pytest

import buffem

pytestmark = pytest.mark.gpu

DISP = [[0, 0, 0], [0.3, 0.1, 2.5], [0, -0.2, 5.0]]


def close(pb, po):
    for cols in (slice(0, 2), slice(2, 5), slice(5, 8)):
        np.testing.assert_allclose(pb[:, cols], po[:, cols], rtol=0, atol=1e-9 * np.abs(po[:, cols]).max())


@pytest.mark.parametrize("omega", [0.05, 0.45, 0.9, 1.8, 3.5, 4.9, 9.0, 0.8 + 0.1j])
@pytest.mark.parametrize("cells", [(3,), (2, 3), (2, 2, 1)])
def test_emt_pairs_match_oracle(sphere, oracle_lib, cells, omega):
    meshes = [sphere(n, radius=0.9 if n == 2 else 1.0) for n in cells]
    disp = DISP[:len(cells)]
    Gb = buffem.SWGGeometry(meshfiles=meshes, materials=[buffem.Material(eps=4 + 0.2j)] * len(cells), displacements=disp,
                            singular_order=4, singular_refine=False)
    Go = oracle_lib.Geometry(meshes, [oracle_lib.material(eps=4 + 0.2j)] * len(cells), displacements=disp, nang=4)
    rng = np.random.default_rng(17)
    N = Gb.TotalBFs
    J = rng.normal(size=N) + 1j * rng.normal(size=N)
    E0, nh = np.array([1, 0.3j, 0], complex), np.array([0.6, 0, 0.8])
    close(Gb.GetPFTMatrix(J, omega, buffem.PlaneWave(E0, nh), full=True), Go.pft_emt8(complex(omega), J, E0, nh))
    import torch
    DR = rng.normal(size=(N, N)) + 1j * rng.normal(size=(N, N))
    d = torch.tensor(np.asfortranarray(DR).T.copy(), device="cuda")
    out = np.zeros((len(cells), 8))
    w = complex(omega)
    buffem._check(buffem.lib().bg_pft_dr_device(Gb.h, w.real, w.imag, C.c_void_p(d.data_ptr()), N, buffem._ptr(out)))
    close(out, Go.pft_emt8_dr(w, DR))
