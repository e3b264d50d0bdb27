"""Fields at points that are no numbers or so far away that the phase differences
inside a tetrahedron are below the rounding of the distance (needs a B200: -m gpu).

Tolerance: beyond k r = 2^53 the phases are arbitrary; the fields stay below the sum of
the currents' far fields, |E| <= |w| Z0 / (4 pi r) sum_a |J_a| (integral of |b_a|, at
most twice the face's area times the radius over 3)."""
import numpy as np
import pytest

import buffem

pytestmark = pytest.mark.gpu
Z0 = 376.73031346177


@pytest.mark.parametrize("omega", [0.01, 0.3, 1.5, 30.0])
def test_far_and_undefined_points(sphere, omega):
    G = buffem.SWGGeometry(meshfiles=sphere(3), materials=buffem.Material(eps=4 + 0.2j))
    rng = np.random.default_rng(1)
    J = rng.normal(size=G.TotalBFs) + 1j * rng.normal(size=G.TotalBFs)
    d = np.array([0.6, 0.48, 0.64])
    far = np.array([1e3, 1e9, 1e14, 1e16, 1e18, 1e30])
    X = np.vstack([far[:, None] * d, np.diag([np.nan] * 3)])
    F = G.GetFields(None, J, omega, X)
    assert np.all(np.isnan(F[len(far):].real))
    # unit sphere: faces below 1, radii below 1.2
    bound = omega * Z0 / (4 * np.pi * far) * 0.8 * np.abs(J).sum()
    E, H = np.abs(F[:len(far), :3]).max(1), np.abs(F[:len(far), 3:]).max(1)
    assert np.all(np.isfinite(E)) and np.all(E <= bound) and np.all(H <= bound / Z0)
    # the far field falls off as 1 / r while its phases are those of the distance
    np.testing.assert_allclose(E[1] * far[1], E[0] * far[0], rtol=0.1)
