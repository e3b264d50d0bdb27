"""A training step at the edges of its kernels' tiles, against the numpy oracle
(needs a B200: -m gpu).

Sizes: fewer unknowns than one node tile (64), than one block of rows, and
remainders of both; probes at 1, at one tile of eight, one over it and the most
a step takes.  The network runs in FP32 with sums of up to 64 terms per layer
and four layers, the rest in FP64, so tolerances are those of the forward and
gradient test: 1e-4 of the loss, 2e-3 of the largest gradient entry; the FP64
probe map alone (error map applied `power` times) is below both.
"""
import os
import sys

import numpy as np
import pytest
import scipy.linalg as sl

import buffem
import meshgen

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import gnn_oracle as go  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,probes,power", [(1, 1, 1), (2, 9, 3), (3, 16, 0), (4, 8, 2)])
def test_step_matches_oracle(sphere, n, probes, power):
    omega = 1.1
    G = buffem.SWGGeometry(meshfiles=sphere(n), materials=buffem.Material(eps=6 + 0.5j))
    A = G.AssembleVIEMatrix(omega)
    N, Ah = G.TotalBFs, A.download()
    rng = np.random.default_rng(100 + n)
    net = buffem.GNN(seed=3)
    flat = net.params()
    off, _ = go.layout()
    for k in ("Wo", "bo"):                   # a readout that is not zero: every layer carries gradient
        o, m = off[k]
        flat[o:o + m] = rng.normal(scale=0.05, size=m).astype(np.float32)
    net.set_params(flat)
    faces = G.faces(0)
    rowptr, col, _ = go.pattern(faces)
    F, Ef, ratio, dinv = go.features(meshgen.sphere_arrays(n)[0], faces, Ah, omega, rowptr, col)
    Z = rng.normal(size=(N, probes)) + 1j * rng.normal(size=(N, probes))
    b = G.AssembleRHSVector(omega, buffem.PlaneWave([1, 0, 0], [0, 0, 1]))
    x = sl.lu_solve(sl.lu_factor(Ah), b)
    loss = net.train_step(G, A, omega, Z, b, x, lam=0.5, lr=0.0, probe_power=power)
    grads = net.grads() * loss               # the device descends log L
    for _ in range(power):
        Z = Z - Ah @ (dinv[:, None] * Z)
        Z *= np.sqrt(2 * N / np.sum(np.abs(Z) ** 2, axis=0))
    want, gw, _ = go.loss_and_grad(flat.astype(np.float64), F, Ef, rowptr, col, ratio, dinv, Ah, Z, b, x, 0.5)
    assert abs(loss - want) <= 1e-4 * abs(want)
    assert np.abs(grads - gw).max() <= 2e-3 * np.abs(gw).max()
