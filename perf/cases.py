"""The work that a user of the dense VIE path has it do, as measurable cases.

Every case goes through the public binding (buff-em_b200/buffem.py) as a
program written on it does: a geometry handle and its matrices are kept, the
frequency, the incident waves and (where they vary in use) the meshes are the
inputs.  Sizes are those of the synthetic spheres that the tests and the
benchmark use: n^3 cells, N = 12 n^3 - 6 n^2 unknowns per sphere.
"""
import math
import os
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "buff-em_b200"))

import buffem  # noqa: E402
import meshgen  # noqa: E402

ZVAC = 376.73031346177


def listed():
    return [
        # a test-sized body: what a call costs when the arithmetic is nothing
        {"name": "scatter_n2", "kind": "scatter", "n": 2, "n2": 0, "eps": "iso", "omega": 1.0, "omega_im": 0.0,
         "rhs": 1},
        # the small-sphere configuration: one frequency of buff-scatter
        {"name": "scatter_n5", "kind": "scatter", "n": 5, "n2": 0, "eps": "iso", "omega": 1.0, "omega_im": 0.0,
         "rhs": 1},
        # two bodies with eps(x) at a complex frequency, of uneven size
        {"name": "scatter_two_n7_n4", "kind": "scatter", "n": 7, "n2": 4, "eps": "gauss", "omega": 0.7,
         "omega_im": 0.1, "rhs": 2},
        # the plain method at scale: anisotropic tensor, three polarisations
        {"name": "scatter_tensor_n12", "kind": "scatter", "n": 12, "n2": 0, "eps": "tensor", "omega": 1.0,
         "omega_im": 0.0, "rhs": 3},
        # factor and solve of a matrix that the program itself holds on the device
        {"name": "lu_device_n4092", "kind": "lu", "n": 7, "n2": 3, "rhs": 3},
        # the precision form: jittered two-material sphere
        {"name": "precision_janus_n12", "kind": "precision", "n": 12, "jitter": 0.05, "eps": "janus", "omega": 1.0,
         "rhs": 1},
        # the learned form at a size of which the card holds several matrices
        {"name": "learned_n15", "kind": "learned", "n": 15, "eps": "six", "omega": 1.0, "rhs": 3},
        # the batching form: heat-transfer sweep over pairs of spheres
        {"name": "batch_two_spheres", "kind": "batch", "geoms": 2, "n": 6, "n2": 3, "omegas": 32, "streams": 8},
        # fields on a plane cut through and around the body after a solve
        {"name": "fields_plane_n17", "kind": "fields", "n": 17, "points": 65, "extent": 3.0, "omega": 1.0,
         "incident": True},
        # one frequency of buff-neq for two spheres
        {"name": "neq_two_n5_n4", "kind": "neq", "n": 5, "n2": 4, "omega": 0.3},
        # a new mesh: reading it and its near-field integrals
        {"name": "new_mesh_n8", "kind": "mesh", "n": 8, "jitter": 0.05},
        # one optimiser step of the learned preconditioner (forward and backward)
        {"name": "train_n7", "kind": "train", "n": 7, "probes": 8, "power": 8, "omega": 1.0},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["scatter", "scatter", "scatter", "lu", "precision", "learned", "batch", "fields", "neq",
                       "mesh", "train"])
    if kind == "scatter":
        n2 = rng.choice([0, 0, 2, 3, 4, 5])
        return {"kind": kind, "n": _log_int(rng, 2, 10), "n2": n2,
                "eps": rng.choice(["iso", "tensor", "janus", "gauss"]), "omega": _log(rng, 0.1, 3.0),
                "omega_im": rng.choice([0.0, 0.0, 0.1]), "rhs": rng.randint(1, 5)}
    if kind == "lu":
        return {"kind": kind, "n": _log_int(rng, 3, 9), "n2": rng.choice([0, 2, 3, 4, 5]), "rhs": rng.randint(1, 6)}
    if kind == "precision":
        return {"kind": kind, "n": _log_int(rng, 4, 10), "jitter": rng.uniform(0.0, 0.05),
                "eps": rng.choice(["janus", "iso", "tensor"]), "omega": _log(rng, 0.3, 1.2), "rhs": rng.randint(1, 4)}
    if kind == "learned":
        return {"kind": kind, "n": _log_int(rng, 5, 13), "eps": rng.choice(["six", "tensor"]),
                "omega": rng.uniform(0.5, 1.2), "rhs": rng.randint(1, 4)}
    if kind == "batch":
        return {"kind": kind, "geoms": rng.randint(1, 2), "n": rng.randint(3, 6), "n2": rng.randint(2, 4),
                "omegas": _log_int(rng, 8, 40), "streams": rng.choice([4, 8])}
    if kind == "fields":
        return {"kind": kind, "n": _log_int(rng, 3, 17), "points": rng.randint(3, 65), "extent": _log(rng, 1.2, 30.0),
                "omega": _log(rng, 0.1, 3.0), "incident": rng.random() < 0.5}
    if kind == "neq":
        return {"kind": kind, "n": rng.randint(2, 5), "n2": rng.choice([0, 2, 3, 4]), "omega": _log(rng, 0.1, 1.0)}
    if kind == "mesh":
        return {"kind": kind, "n": _log_int(rng, 2, 8), "jitter": rng.uniform(0.01, 0.06)}
    return {"kind": "train", "n": rng.randint(4, 7), "probes": rng.randint(2, 8), "power": rng.choice([0, 8]),
            "omega": rng.uniform(0.5, 1.5)}


# ------------------------------------------------------------------ inputs
def _mesh(n, jitter=0.0, seed=0):
    return meshgen.cached_sphere(os.path.join(tempfile.gettempdir(), "buffem_perf_meshes_%d" % os.getuid()), n, 1.0,
                                 jitter, seed)


def _material(eps, center=(0.0, 0.0, 0.0)):
    if eps == "iso":
        return buffem.Material(eps=4 + 0.2j)
    if eps == "six":
        return buffem.Material(eps=6 + 0.5j)
    if eps == "tensor":
        return buffem.Material(kind=buffem.BG_MAT_CONST_TENSOR,
                               tensor=np.array([[4, 0.5, 0], [0.5, 6, 0], [0, 0, 9]]) + 0.1j * np.eye(3))
    if eps == "janus":
        return buffem.Material(kind=buffem.BG_MAT_JANUS_Z, eps=4 + 0.2j, eps2=12 + 1j)
    return buffem.Material(kind=buffem.BG_MAT_GAUSSIAN, eps=3 + 0.1j, center=center, amp=1.5, width=1.0)


_geometries = {}


def _geometry(n, n2=0, eps="iso", jitter=0.0, gap=0.4):
    """A program sweeps frequencies on one geometry handle; so do the states
    of one case."""
    key = (n, n2, eps, jitter, gap)
    if key not in _geometries:
        while len(_geometries) >= 3:
            _geometries.pop(next(iter(_geometries)))
        meshes, mats, disp = [_mesh(n, jitter, 2)], [_material(eps)], [[0.0, 0.0, 0.0]]
        if n2:
            z = 2.0 + gap
            meshes.append(_mesh(n2))
            mats.append(_material(eps, (0.0, 0.0, z)))
            disp.append([0.0, 0.0, z])
        G = buffem.SWGGeometry(meshfiles=meshes, materials=mats, displacements=disp)
        _geometries[key] = G
    return _geometries[key]


def _wave(rng):
    n = rng.normal(size=3)
    n /= np.linalg.norm(n)
    e = rng.normal(size=3)
    e -= n * (n @ e)
    return buffem.PlaneWave(e / np.linalg.norm(e), n)


def _omega(case, rng):
    return complex(case["omega"] * (1 + 0.02 * rng.uniform(-1, 1)), case.get("omega_im", 0.0))


class _DeviceArray:
    """A matrix handle's device memory for torch (column-major)."""

    def __init__(self, M):
        ptr, ld = M.device_ptr()
        self.owner = M
        self.__cuda_array_interface__ = {"shape": (M.NC, M.NR), "strides": (16 * ld, 16), "typestr": "<c16",
                                         "data": (ptr, False), "version": 2}


def _view(M):
    return torch.as_tensor(_DeviceArray(M), device="cuda").T


def _num(case):
    return meshgen.num_bfs(case["n"]) + (meshgen.num_bfs(case["n2"]) if case.get("n2") else 0)


def _system(case, seed):
    """A dense symmetric system like the VIE one: a Helmholtz kernel between
    points of a ball plus a banded block of the Gram terms' size."""
    N = _num(case)
    g = torch.Generator(device="cuda").manual_seed(seed)
    f8 = dict(dtype=torch.float64, device="cuda", generator=g)
    x = torch.randn(N, 3, **f8)
    x = x / x.norm(dim=1, keepdim=True) * torch.rand(N, 1, **f8) ** (1 / 3)
    r = torch.sqrt(torch.cdist(x, x, compute_mode="donot_use_mm_for_euclid_dist") ** 2 + 0.02)
    A = torch.polar(1.0 / (math.pi * N * r), r)
    for k in range(1, 8):
        v = 0.15 * torch.complex(torch.randn(N - k, **f8), torch.randn(N - k, **f8))
        A.diagonal(k).add_(v)
        A.diagonal(-k).add_(v)
    A.diagonal().add_(torch.complex(0.3 + 0.1 * torch.rand(N, **f8), 0.05 * torch.ones(N, dtype=torch.float64,
                                                                                      device="cuda")))
    B = torch.complex(torch.randn(N, case["rhs"], **f8), torch.randn(N, case["rhs"], **f8))
    return A, B


def _currents(case, seed):
    N = _num(case)
    rng = np.random.default_rng(seed)
    J = rng.normal(size=N) + 1j * rng.normal(size=N)
    p = np.linspace(-case["extent"], case["extent"], case["points"])
    a, b = np.meshgrid(p, p * 0.97, indexing="ij")
    X = np.stack([a.ravel(), np.full(a.size, 0.013 + 0.01 * rng.random()), b.ravel()], axis=1)
    return J, X, _omega(case, rng), _wave(rng) if case["incident"] else None


def prepare(case, seed):
    kind, rng = case["kind"], np.random.default_rng(seed)
    s = {"kind": kind, "case": case}
    if kind == "lu":
        s["A"], B = _system(case, seed)
        s["B"] = np.asfortranarray(B.cpu().numpy())
        s["G"] = _geometry(case["n"], case["n2"])
        s["M"] = s["G"].AllocateVIEMatrix()
        s["view"] = _view(s["M"])
        return s
    if kind == "fields":
        s["J"], s["X"], s["omega"], s["wave"] = _currents(case, seed)
        s["G"] = _geometry(case["n"])
        return s
    if kind == "mesh":
        s["mesh"] = _mesh(case["n"], case["jitter"], seed)
        return s
    if kind == "batch":
        rs = np.random.default_rng(1)
        s["G"] = [_geometry(case["n"] - g, case["n2"] + g, "gauss", gap=round(rs.uniform(0.2, 1.0), 3))
                  for g in range(case["geoms"])]
        lo = 0.01 * (1 + 0.02 * rng.random())
        s["omega"] = np.geomspace(lo, 1000 * lo, case["omegas"])
        s["wave"] = _wave(rng)
        for G in s["G"]:
            G.precompute()
        return s
    if kind == "neq":
        s["omega"] = _omega(case, rng)
        s["G"] = _geometry(case["n"], case["n2"])
        s["G"].precompute()
        s["neq"] = buffem.NEQ(s["G"])
        return s
    G = s["G"] = _geometry(case["n"], case.get("n2", 0), case.get("eps", "six"), case.get("jitter", 0.0))
    G.precompute()
    s["omega"] = _omega(case, rng)
    s["waves"] = [_wave(rng) for _ in range(case.get("rhs", 1))]
    s["M"] = G.AllocateVIEMatrix()
    if kind in ("precision", "learned"):
        s["F"] = G.AllocateVIEMatrix(buffem.BG_C64)
    if kind == "precision":
        s["view"] = _view(s["M"])
    if kind == "learned":
        s["net"] = buffem.GNN.load()
    if kind == "train":
        w, N = s["omega"].real, G.TotalBFs
        G.AssembleVIEMatrix(w, s["M"])
        s["b"] = G.AssembleRHSVector(w, s["waves"][0])
        L = G.AssembleVIEMatrix(w)
        s["x"] = L.LUFactorize().LUSolve(s["b"].copy())
        s["Z"] = rng.normal(size=(N, case["probes"])) + 1j * rng.normal(size=(N, case["probes"]))
        s["net"] = buffem.GNN.load()
    return s


# ------------------------------------------------------------------ a pass
def _rhs(s):
    B = np.zeros((s["G"].TotalBFs, len(s["waves"])), complex, order="F")
    for j, wave in enumerate(s["waves"]):
        s["G"].AssembleRHSVector(s["omega"], wave, B[:, j])
    return B


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "lu":
        s["view"].copy_(s["A"])
        torch.cuda.current_stream().synchronize()   # the library works on a stream of its own
        return s["M"].LUFactorize().LUSolve(s["B"].copy(order="F"))
    if kind == "fields":
        return s["G"].GetFields(s["wave"], s["J"], s["omega"], s["X"])
    if kind == "mesh":
        G = buffem.SWGGeometry(meshfiles=s["mesh"], materials=_material("iso"))
        G.precompute()
        return G.near_data()
    if kind == "batch":
        return buffem.BatchSweep(s["G"], s["omega"], s["wave"], max_streams=case["streams"])[0]
    if kind == "neq":
        return s["neq"].GetFlux(s["omega"])
    if kind == "train":
        loss = s["net"].train_step(s["G"], s["M"], s["omega"].real, s["Z"], s["b"], s["x"], lam=0.5, lr=1e-3,
                                   probe_power=case["power"])
        return {"loss": loss, "grads": s["net"].grads(), "params": s["net"].params()}
    G, w, M = s["G"], s["omega"], s["M"]
    if kind == "scatter":
        G.AssembleVIEMatrix(w, M)
        M.LUFactorize()
        J = _rhs(s)
        M.LUSolve(J)
        return {"J": J, "pft": G.GetPFTMatrix(J[:, 0], w, s["waves"][0], full=True),
                "pabs": G.GetPFTMatrix(J[:, 0], w, s["waves"][0], method=buffem.BG_PFT_OVERLAP)}
    G.AssembleVIEMatrixWithCopy(w, M, s["F"])
    B = _rhs(s)
    if kind == "precision":
        s["F"].LUFactorize()
        X, _ = M.LUSolveRefined(s["F"], B, tol=1e-12, maxit=40)
        return {"J": X, "matrix": s["view"]}
    P = buffem.Preconditioner.learned(G, M, w.real, s["net"])
    return buffem.SolveLearned(M, s["F"], B, P, tol=1e-10)[0]


# -------------------------------------------------------------- least work
def work(case):
    """Each matrix entry: one 4-point-rule sum over shared tetrahedron pairs
    (about 0.8 pairs of 16 kernel values, 50 flops each); 8/3 N^3 flops for a
    complex LU; 32 N^2 per right-hand side of a solve."""
    kind, N = case["kind"], _num(case) if "n" in case else 0
    far = 0.5 * N * N * 0.8 * 16 * 50
    rhs = case.get("rhs", 1)
    if kind == "scatter":
        return {"bytes": 16 * N * (rhs + 1) + 200 * N, "flops": far + 8 / 3 * N ** 3 + 8 * N * N * rhs}
    if kind == "lu":
        return {"bytes": 32 * N * N + 32 * N * rhs, "flops": 8 / 3 * N ** 3 + 8 * N * N * rhs}
    if kind == "precision":
        return {"bytes": 24 * N * N, "flops": far + 8 / 3 * N ** 3 + 6 * 16 * N * N * rhs}
    if kind == "learned":
        steps = 100 if N > 10000 else 60
        return {"bytes": 24 * N * N + 4 * N * N * steps, "flops": far + 8 * N * N * steps * rhs}
    if kind == "batch":
        sizes = [meshgen.num_bfs(case["n"] - g) + meshgen.num_bfs(case["n2"] + g) for g in range(case["geoms"])]
        return {"bytes": 200 * sum(sizes) * case["omegas"],
                "flops": case["omegas"] * sum(0.5 * n * n * 0.8 * 16 * 50 + 8 / 3 * n ** 3 + 8 * n * n for n in sizes)}
    if kind == "fields":
        tets, pts = 6 * case["n"] ** 3, case["points"] ** 2
        return {"bytes": 200 * tets + 120 * pts, "flops": 156.0 * tets * pts * 4}
    if kind == "neq":
        return {"bytes": 64 * N * N, "flops": far + (8 / 3 + 32) * N ** 3}
    if kind == "mesh":
        # about 80 near pairs a row, 1,500 angular points a singular tetrahedron pair
        return {"bytes": 56 * 80 * N, "flops": 6 * case["n"] ** 3 * 20 * 1500 * 60.0}
    edges = 175 * N
    return {"bytes": 16 * N * N * (1 + case["power"]), "flops": 6.0 * edges * (64 * 8 + 64 * 64) +
            8 * N * N * case["probes"] * (1 + case["power"])}


# ------------------------------------------------- the same in plain 64 bits
def _swg(V, T):
    """Rows of the basis in the order of their faces' second visit: first and
    second tetrahedron and the local index of the vertex opposite the face."""
    seen, rows = {}, []
    for t, tet in enumerate(T.tolist()):
        for f in range(4):
            key = tuple(sorted(tet[:f] + tet[f + 1:]))
            if key in seen:
                rows.append(seen.pop(key) + (t, f))
            else:
                seen[key] = (t, f)
    return np.array(rows)


def _rule(n):
    """Symmetric tetrahedron rules of 4 and 16 points: barycentric
    coordinates and weights that sum to 1."""
    if n == 4:
        a, b = 0.5854101966249685, 0.1381966011250105
        return np.array([[a if i == j else b for j in range(4)] for i in range(4)]), np.full(4, 0.25)
    a, b = 0.771642902067237, 0.076119032644254315
    p = [[a if i == j else b for j in range(4)] for i in range(4)]
    c, d, e = 0.07183164526766925, 0.11970052779780202, 0.40423391346726440
    for i in range(4):
        for j in range(4):
            if i != j:
                p.append([c if k == i else d if k == j else e for k in range(4)])
    return np.array(p), 6.0 * np.array([8.3956323500204695e-3] * 4 + [0.011090344772215399] * 12)


def _fields_exact(case, seed):
    """Fields of the currents by the rules themselves: 16 points per
    tetrahedron within ten radii of a face, 4 beyond."""
    J, X, w, wave = _currents(case, seed)
    V, T = meshgen.sphere_arrays(case["n"])
    rows = _swg(V, T)
    V, X = torch.from_numpy(V).cuda(), torch.from_numpy(X).cuda()
    T, J = torch.from_numpy(T).long().cuda(), torch.from_numpy(J).cuda()
    t = [torch.from_numpy(rows[:, i]).cuda() for i in (0, 2)]
    f = [torch.from_numpy(rows[:, i]).cuda() for i in (1, 3)]
    face = torch.stack([T[t[0], (f[0] + 1 + i) % 4] for i in range(3)], 1)
    c = V[face].mean(1)
    area = 0.5 * torch.linalg.cross(V[face[:, 1]] - V[face[:, 0]], V[face[:, 2]] - V[face[:, 0]]).norm(dim=1)
    Q = [V[T[t[i], f[i]]] for i in (0, 1)]
    radius = torch.stack([(V[face[:, i]] - c).norm(dim=1) for i in range(3)] + [(q - c).norm(dim=1) for q in Q]).amax(0)
    out = torch.zeros(len(X), 6, dtype=torch.complex128, device="cuda")
    for lo in range(0, len(X), 32):
        x = X[lo:lo + 32]
        near = (x[:, None] - c[None]).norm(dim=2) / radius[None] <= 10.0
        for npts in (4, 16):
            use = (near if npts == 16 else ~near)
            some = use.any(0).nonzero()[:, 0]
            if not len(some):
                continue
            bary, wt = _rule(npts)
            weight = torch.where(use[:, some], J[None, some], torch.zeros((), dtype=J.dtype, device="cuda"))
            for side, sign in ((0, 1.0), (1, -1.0)):
                tv = V[T[t[side][some]]]
                for p in range(npts):
                    y = (torch.from_numpy(bary[p]).cuda()[None, :, None] * tv).sum(1)
                    b = sign * (area[some] / 3.0 * wt[p])[:, None] * (y - Q[side][some])
                    R = x[:, None] - y[None]
                    r = R.norm(dim=2)
                    ok = r >= 1e-12
                    r = torch.where(ok, r, torch.ones_like(r))
                    R = R / r[..., None]
                    ikr = 1j * w * r
                    g = torch.where(ok, weight * torch.exp(ikr) / (4 * math.pi * r), torch.zeros_like(ikr))
                    rb = (R * b[None]).sum(2)
                    e1, e2 = 1j * w * ZVAC * g * (1 - 1 / ikr + 1 / ikr ** 2), 1j * w * ZVAC * g * (
                        -1 + 3 / ikr - 3 / ikr ** 2) * rb
                    h = g * (1j * w - 1 / r)
                    out[lo:lo + 32, :3] += e1 @ b.to(e1.dtype) + (e2[..., None] * R).sum(1)
                    out[lo:lo + 32, 3:] += (h[..., None] * torch.linalg.cross(R, b[None].expand_as(R))).sum(1)
    if wave is not None:
        n = torch.from_numpy(wave.nHat).cuda()
        E = torch.from_numpy(wave.E0).cuda()[None] * torch.exp(1j * w * (X @ n))[:, None]
        out[:, :3] += E
        out[:, 3:] += torch.linalg.cross(n.to(E.dtype)[None].expand_as(E), E) / ZVAC
    return out.cpu().numpy()


def exact(case, seed):
    """The solved systems and the radiated fields.  The assembled matrices
    hold singular integrals by adaptive refinement, which plain 64-bit code
    does not reach in seconds: the cases that start from them have none."""
    if case["kind"] == "lu":
        A, B = _system(case, seed)
        X = torch.linalg.solve(A, B)
        X += torch.linalg.solve(A, B - A @ X)
        return X.cpu().numpy()
    if case["kind"] == "fields" and 6 * case["n"] ** 3 * case["points"] ** 2 < 2.0e8:
        return _fields_exact(case, seed)
    return None
