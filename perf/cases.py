"""The work a user of the library has it do, as cases to time: matrix assembly,
LU factorisation and solution in FP64, mixed-precision and refined solves,
batches, the Casimir integrand and the shape gradient, over the sizes of the
repository's own workloads (PEC and dielectric icospheres, jittered rounded
cubes, open shells; N = 480 to 15360).

``listed`` gives the named cases, ``draw`` more of the same ranges; ``prepare``
makes what a program holds before the call, ``run`` is one pass through the
public entry points, ``work`` the bytes and operations a pass cannot do
without, ``exact`` the 64-bit result where numpy alone can form it.
"""
import os
import sys

import numpy as np
import torch

PKG = os.path.join(os.getcwd(), "scuff-em_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import gbem  # noqa: E402
from gbem import C64, C128, HMatrix, Material, RWGGeometry, mesh, solve_mixed_batch  # noqa: E402
from gbem.casimir import CasimirIntegrand  # noqa: E402

# polarisation and direction of the plane waves of a 4-wave solve
WAVES = [((1, 0, 0), (0, 0, 1)), ((0, 1, 0), (0, 0, 1)), ((1, 0, 0), (0, 0, -1)), ((0, 1, 0), (0, 0, -1))]

# Residual every mixed or refined solve is taken to, in place of the entry
# points' 1e-10: what a program asks for when it takes differences of currents
# (finite differences of a power, convergence studies).
TOL = 3e-12


def listed():
    return [
        # one incident field on the small PEC sphere: the shortest call there is,
        # made for every wave of every frequency of a sweep
        {"name": "rhs_sphere_480", "kind": "rhs", "body": "sphere", "size": 2, "pec": True, "kR": 1.0},
        # the small plain workload: one FP64 assembly, factorisation and solve
        {"name": "fp64_sphere_480", "kind": "fp64", "body": "sphere", "size": 2, "pec": True, "kR": 1.0, "nrhs": 1},
        # the same for a dielectric sphere of ordinary size, four waves
        {"name": "fp64_sphere_3840", "kind": "fp64", "body": "sphere", "size": 3, "pec": False, "kR": 2.0, "nrhs": 4},
        # FP64 matrix of a jittered rounded cube, left on the device (a caller
        # that wants the matrix for its own solver)
        {"name": "assemble64_cube_6084", "kind": "assemble64", "body": "cube", "size": 13, "pec": False, "kR": 1.5},
        # LUFactorize and LUSolve of a host matrix of odd size (the HMatrix drop-in)
        {"name": "lu64_shell_1909", "kind": "lu64", "body": "shell", "size": 3, "holes": 5, "pec": True, "kR": 2.0,
         "nrhs": 8},
        # mixed-precision solves: the smallest dielectric sphere, the middle one,
        # and the headline workload
        {"name": "mixed_sphere_960", "kind": "mixed", "body": "sphere", "size": 2, "pec": False, "kR": 2.0, "nrhs": 2},
        {"name": "mixed_sphere_3840", "kind": "mixed", "body": "sphere", "size": 3, "pec": False, "kR": 2.0, "nrhs": 4},
        {"name": "mixed_sphere_15360", "kind": "mixed", "body": "sphere", "size": 4, "pec": False, "kR": 2.0,
         "nrhs": 4},
        # the FP64 solution by refinement of a complex64 factor, on a rounded cube
        {"name": "refined_cube_4356", "kind": "refined", "body": "cube", "size": 11, "pec": False, "kR": 1.0,
         "nrhs": 2},
        # a sweep of uneven bodies as one batch (the batching workload in small)
        {"name": "batch_8", "kind": "batch", "sphere_to": 3, "cube_to": 12, "jobs": 8, "kR": 1.0, "nrhs": 2},
        # energy and force integrand of two PEC spheres at one imaginary
        # frequency (real storage, determinants and a trace)
        {"name": "casimir_3840", "kind": "casimir", "body": "sphere", "size": 3, "pec": True, "xi": 0.4, "gap": 1.0},
        # the adjoint contraction of a shape gradient
        {"name": "vjp_sphere_960", "kind": "vjp", "body": "sphere", "size": 2, "pec": False, "kR": 2.0, "nrhs": 1},
    ]


def draw(rng):
    kind = rng.choice(["rhs", "fp64", "fp64", "assemble64", "assemble32", "lu64", "mixed", "mixed", "mixed", "refined",
                       "batch", "casimir", "vjp"])
    c = {"kind": kind, "kR": round(0.5 * 8.0 ** rng.random(), 4)}
    if kind == "batch":
        c.update(sphere_to=rng.choice([2, 3]), cube_to=rng.randint(6, 12), jobs=rng.randint(4, 8), kR=round(rng.uniform(0.6, 2.0), 4),
                 nrhs=rng.randint(1, 3))
        return c
    if kind == "casimir":
        del c["kR"]
        c.update(body=rng.choice(["sphere", "cube"]), pec=True, xi=round(rng.uniform(0.1, 0.9), 4),
                 gap=round(rng.uniform(0.6, 1.5), 4))
        c["size"] = rng.choice([2, 3]) if c["body"] == "sphere" else rng.randint(5, 10)
        return c
    c["pec"] = rng.random() < 0.4
    c["body"] = rng.choice(["sphere", "cube", "shell"] if c["pec"] else ["sphere", "cube", "cube"])
    # panels per workload: N goes with the panels, times 2 on a dielectric
    most = {"rhs": 16, "fp64": 11, "assemble64": 13, "assemble32": 16, "lu64": 13, "mixed": 16, "refined": 12, "vjp": 6}[kind]
    if c["body"] == "cube":
        c["size"] = int(round(5 * (most / 5.0) ** rng.random()))
    else:
        c["size"] = rng.choice([2, 3, 4] if kind in ("rhs", "mixed", "assemble32") else [2] if kind == "vjp" else [2, 3])
    if c["body"] == "shell":
        c["holes"] = rng.randint(1, 9)
    if kind not in ("rhs", "assemble64", "assemble32"):
        c["nrhs"] = rng.randint(1, 8) if kind != "vjp" else rng.randint(1, 2)
    return c


def _mesh(case, rng, body=None, size=None):
    body, size = body or case["body"], size or case["size"]
    if body == "cube":
        return mesh.rounded_cube(12 * size * size, side=float(rng.uniform(0.9, 1.1)), seed=int(rng.integers(1 << 30)))
    V, P = mesh.icosphere(size)
    V = V * rng.uniform(0.95, 1.05) * rng.uniform(0.98, 1.02, 3)  # slightly ellipsoidal
    if body == "shell":  # open: the panels nearest the pole left out
        z = V[P].mean(axis=1)[:, 2]
        P = P[np.sort(np.argsort(-z, kind="stable")[case["holes"]:])]
        used = np.unique(P)
        new = np.full(len(V), -1, dtype=np.int64)
        new[used] = np.arange(len(used))
        V, P = V[used], new[P].astype(np.int32)
    return V, P


def _geometry(case, rng, body=None, size=None):
    V, P = _mesh(case, rng, body, size)
    mat = None if case.get("pec") else Material(complex(rng.uniform(2.0, 2.5), rng.uniform(0.005, 0.02)))
    R = 0.5 if (body or case["body"]) == "cube" else 1.0
    return RWGGeometry([{"V": V, "P": P, "material": mat}]), case["kR"] / R * float(rng.uniform(0.97, 1.03))


def _waves(G, w, n):
    k = 2.0 ** 0.5 / 2
    more = WAVES + [((0, 0, 1), (1, 0, 0)), ((0, 1, 0), (1, 0, 0)), ((k, 0, -k), (k, 0, k)), ((0, 1, 0), (k, 0, k))]
    return np.asfortranarray(np.stack([G.AssembleRHSVector(w, e, d) for e, d in more[:n]], axis=1))


class _DeviceMatrix:
    """A matrix on the device as a torch tensor's source (it keeps the matrix)."""

    def __init__(self, M):
        p, ld = M.device_ptr()
        size = {C128: 16, C64: 8}[M.dtype]
        self.M = M
        self.__cuda_array_interface__ = {"shape": (M.N, M.N), "typestr": "<c%d" % size, "data": (p, False),
                                         "strides": (size, size * ld), "version": 3}


def _points_matrix(n, rng, k):
    """A host matrix of the kind HMatrix callers factor: the Helmholtz kernel
    between n points of a unit sphere, with the points' self terms."""
    x = rng.standard_normal((n, 3))
    x /= np.linalg.norm(x, axis=1, keepdims=True)
    r = np.sqrt(np.maximum(2.0 - 2.0 * (x @ x.T), 0.0))
    np.fill_diagonal(r, 1.0)
    A = np.exp(1j * k * r) / (4.0 * np.pi * r)
    A[np.diag_indices(n)] = 0.28 * n ** 0.5 + 1j * k / (4.0 * np.pi)
    return np.asfortranarray(A)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "batch":
        jobs, geos = [], []
        for j in range(case["jobs"]):
            if j % 2 == 0:  # two frequencies of each body, spheres and cubes in turn
                body = "sphere" if j % 4 == 0 else "cube"
                size = 2 + (j // 4) % (case["sphere_to"] - 1) if body == "sphere" else max(5, case["cube_to"] - 2 * (j // 4))
                geos.append(_geometry(case, rng, body, size))
            G, w = geos[-1]
            w *= 1.0 + 0.25 * (j % 2)
            jobs.append((G, w, _waves(G, w, case["nrhs"])))
        return {"kind": kind, "jobs": jobs}
    if kind == "casimir":
        V, P = _mesh(case, rng)
        d = case["gap"] + float(V[:, 2].max() - V[:, 2].min())
        bodies = [{"V": V, "P": P, "material": None}, {"V": V + [0.0, 0.0, d], "P": P, "material": None}]
        return {"kind": kind, "cas": CasimirIntegrand(bodies), "xi": case["xi"] * float(rng.uniform(0.97, 1.03))}
    G, w = _geometry(case, rng)
    s = {"kind": kind, "G": G, "w": w}
    if kind == "rhs":
        d = rng.standard_normal(3)
        d /= np.linalg.norm(d)
        e = np.cross(d, [0.3, 0.5, 0.8])
        s["wave"] = (tuple(e / np.linalg.norm(e)), tuple(d))
    elif kind in ("assemble64", "assemble32"):
        s["M"] = HMatrix(G, C128 if kind == "assemble64" else C64)
        s["view"] = torch.as_tensor(_DeviceMatrix(s["M"]), device="cuda")
    elif kind == "fp64":
        s["M"] = HMatrix(G, C128)
        s["B"] = _waves(G, w, case["nrhs"])
    elif kind == "lu64":
        s["M"] = HMatrix(G, C128)
        s["A"], s["B"] = _lu_inputs(case, G.TotalBFs, seed)
    elif kind in ("mixed", "refined"):
        s["B"] = _waves(G, w, case["nrhs"])
    elif kind == "vjp":
        shape = (G.TotalBFs, case["nrhs"])
        s["lam"], s["x"] = (np.asfortranarray(rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) for _ in range(2))
    else:
        raise ValueError(kind)
    return s


def _lu_inputs(case, n, seed):
    rng = np.random.default_rng([seed, n])
    A = _points_matrix(n, rng, 2.0 * case["kR"])
    shape = (n, case["nrhs"])
    return A, np.asfortranarray(rng.standard_normal(shape) + 1j * rng.standard_normal(shape))


def run(s):
    kind = s["kind"]
    if kind == "rhs":
        return s["G"].AssembleRHSVector(s["w"], *s["wave"])
    if kind == "assemble64":
        s["G"].AssembleBEMMatrix(s["w"], s["M"])
        return s["view"]
    if kind == "assemble32":
        s["G"].AssembleBEMMatrix(s["w"], s["M"], precision="mixed")
        return s["view"]
    if kind == "fp64":
        s["G"].AssembleBEMMatrix(s["w"], s["M"])
        s["M"].LUFactorize()
        return s["M"].LUSolve(s["B"])
    if kind == "lu64":
        s["M"].set(s["A"])
        s["M"].LUFactorize()
        return {"X": s["M"].LUSolve(s["B"]), "ipiv": s["M"].ipiv}
    if kind == "mixed":
        return s["G"].solve_mixed(s["w"], s["B"], tol=TOL, max_iter=12)[0]
    if kind == "refined":
        return s["G"].solve_refined(s["w"], s["B"], tol=TOL, max_iter=12)[0]
    if kind == "batch":
        return [x for x, _, _ in solve_mixed_batch(s["jobs"], tol=TOL, max_iter=12)]
    if kind == "casimir":
        return s["cas"](s["xi"])
    return s["G"].VertexVJP(s["w"], s["lam"], s["x"])


def _panels_edges(body, size, holes=0):
    if body == "cube":
        return 12 * size * size, 18 * size * size
    npan = 20 * 4 ** size
    return npan - holes, 3 * npan // 2 - (2 * holes + 1 if holes else 0)


def work(case):
    """Assembly: 36 samples of 100 operations for each unordered panel pair
    and region, the matrix written once.  LU: 8 N^3 / 3 real operations
    (2 N^3 / 3 in real storage), the matrix read and written once."""
    kind = case["kind"]
    if kind == "batch":
        tot = {"bytes": 0.0, "flops": 0.0}
        for j in range(case["jobs"]):
            b = "sphere" if j % 4 < 2 else "cube"
            k = j // 2 * 2 // 4
            size = 2 + k % (case["sphere_to"] - 1) if b == "sphere" else max(5, case["cube_to"] - 2 * k)
            w = work({"kind": "mixed", "body": b, "size": size, "pec": False, "nrhs": case["nrhs"]})
            tot = {q: tot[q] + w[q] for q in tot}
        return tot
    npan, n = _panels_edges(case["body"], case["size"], case.get("holes", 0))
    regions = 1 if case["pec"] else 2
    N = n * regions
    nrhs = case.get("nrhs", 1)
    fill = 1800.0 * npan * npan * regions
    lu = 8.0 * N ** 3 / 3.0
    if kind == "rhs":
        return {"bytes": 72.0 * npan + 16.0 * N, "flops": 2.0 * 121 * n * 40}
    if kind == "assemble64":
        return {"bytes": 16.0 * N * N, "flops": fill}
    if kind == "assemble32":
        return {"bytes": 8.0 * N * N, "flops": fill}
    if kind == "fp64":
        return {"bytes": 32.0 * N * N + 32.0 * N * nrhs, "flops": fill + lu + 8.0 * N * N * nrhs}
    if kind == "lu64":
        return {"bytes": 32.0 * N * N + 32.0 * N * nrhs, "flops": lu + 8.0 * N * N * nrhs}
    if kind == "mixed":
        return {"bytes": 16.0 * N * N + 32.0 * N * nrhs, "flops": fill + lu + 16.0 * N * N * nrhs}
    if kind == "refined":
        return {"bytes": 32.0 * N * N + 32.0 * N * nrhs, "flops": fill + lu + 16.0 * N * N * nrhs}
    if kind == "casimir":  # both bodies' matrix, one T block, the trace solve
        return {"bytes": 8.0 * (2 * N) ** 2 * 2 + 8.0 * N * N * 4,
                "flops": 4 * fill + 2.0 * (2 * N) ** 3 / 3 + 2.0 * N ** 3 / 3 + 2.0 * (2 * N) ** 2 * N}
    return {"bytes": 72.0 * npan + 32.0 * N * nrhs, "flops": 2.5 * fill}


def exact(case, seed):
    """The factorisation and solution of a host matrix; the other outputs need
    the singular panel integrals, which numpy alone does not give."""
    if case["kind"] != "lu64":
        return None
    rng = np.random.default_rng(seed)
    V, P = _mesh(case, rng)
    e = np.sort(np.concatenate([P[:, [0, 1]], P[:, [1, 2]], P[:, [2, 0]]]), axis=1)
    _, count = np.unique(e, axis=0, return_counts=True)
    if not case["pec"]:
        count = np.concatenate([count, count])
    A, B = _lu_inputs(case, int((count == 2).sum()), seed)
    return {"X": np.linalg.solve(A, B), "ipiv": None}
