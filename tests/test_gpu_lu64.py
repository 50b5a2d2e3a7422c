"""FP64 LU whose updates run on the tensor cores (integer slices of the
operands), at the sizes where a tile, a slice or a panel ends, against
LAPACK and against the factorisation's own backward error."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _factor(A):
    from gbem._lib import lib
    N = A.shape[0]
    LU = np.asfortranarray(A.astype(np.complex128))
    ipiv = np.zeros(N, dtype=np.int32)
    info = ctypes.c_int()
    st = lib().gbem_lu_factor_host(LU.ctypes.data, N, N, ipiv.ctypes.data, ctypes.byref(info))
    assert st == 0 and info.value == 0
    return LU, ipiv - 1


def _check_backward(A, LU, piv):
    """|P A - L U| <= c N u (row maximum of |L|) (column maximum of |U|): the
    standard bound of Gaussian elimination, sum_k |l_ik| |u_kj| <= N max max,
    with c = 8 for complex products and the slices' rounding."""
    N = A.shape[0]
    perm = np.arange(N)
    for i, p in enumerate(piv):
        assert i <= p < N
        perm[[i, p]] = perm[[p, i]]
    L, R = np.tril(LU, -1) + np.eye(N), np.triu(LU)
    assert np.abs(L).max() <= np.sqrt(2.0) * (1 + 1e-12)
    bound = 8 * N * U * np.outer(np.abs(L).max(axis=1), np.abs(R).max(axis=0))
    assert (np.abs(A[perm] - L @ R) <= bound + 8 * N * U * np.abs(A[perm])).all()


@pytest.mark.parametrize("N", [255, 256, 272, 319, 320, 321, 383, 384, 385, 513, 640, 777])
def test_factor_edges(N):
    import scipy.linalg as sl
    rng = np.random.default_rng(N)
    A = rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))
    LU, piv = _factor(A)
    lu_ref, piv_ref = sl.lu_factor(A)
    assert np.array_equal(piv, piv_ref)
    assert np.abs(LU - lu_ref).max() <= 1e-11 * np.abs(lu_ref).max()
    _check_backward(A, LU, piv)


@pytest.mark.parametrize("span", [40, 400])
def test_factor_badly_scaled_columns(span):
    """Columns spread over 2^(2 span) and entries over 2^20: each column of U
    keeps its own scale."""
    N = 400
    rng = np.random.default_rng(span)
    A = rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))
    A *= 2.0 ** rng.uniform(-10, 10, (N, N))
    A *= 2.0 ** np.round(rng.uniform(-span, span, N))
    LU, piv = _factor(A)
    _check_backward(A, LU, piv)


def test_factor_keeps_non_finite_visible():
    """A NaN in the last column stays in that column's U and leaves the other
    columns' factors alone (the row updates never mix columns)."""
    N = 400
    rng = np.random.default_rng(5)
    A = rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))
    ref, piv = _factor(A)
    A[:, N - 1] = np.nan
    from gbem._lib import lib
    LU = np.asfortranarray(A)
    ipiv = np.zeros(N, dtype=np.int32)
    info = ctypes.c_int()
    lib().gbem_lu_factor_host(LU.ctypes.data, N, N, ipiv.ctypes.data, ctypes.byref(info))
    assert np.array_equal(ipiv[:N - 1] - 1, piv[:N - 1])
    assert np.array_equal(LU[:, :256], ref[:, :256])
    assert np.abs(LU[:, :N - 1] - ref[:, :N - 1]).max() <= 1e-12 * np.abs(ref).max()
    assert not np.isfinite(LU[:, N - 1]).any()


def _strip(n):
    """An open PEC strip of n + 1 triangles: n interior edges, N = n."""
    from gbem import RWGGeometry
    V = np.array([[0.5 * i, i % 2, 0.01 * i * i / (n + 1)] for i in range(n + 3)], dtype=np.float64)
    P = np.array([[i, i + 1, i + 2] if i % 2 == 0 else [i + 1, i, i + 2] for i in range(n + 1)], dtype=np.int32)
    return RWGGeometry([{"V": V, "P": P, "material": None}])


@pytest.mark.parametrize("N", [1, 2, 15, 16, 17, 31, 33, 65, 255, 257, 320, 513, 777])
def test_real_factor_solve_and_trace_edges(N):
    """F64 matrices in real arithmetic: dgetrf's pivots and factors, and
    Tr[M^-1 B] over the first columns, at leaf, panel and tile edges."""
    import scipy.linalg as sl
    from gbem._lib import F64
    from gbem.api import HMatrix
    G = _strip(N)
    M = HMatrix(G, F64)
    rng = np.random.default_rng(N)
    A = rng.standard_normal((N, N))
    M.set(A)
    assert M.LUFactorize() == 0
    lu_ref, piv_ref = sl.lu_factor(A)
    assert np.array_equal(M.ipiv - 1, piv_ref)
    LU = M.numpy()
    assert np.abs(LU - lu_ref).max() <= 1e-11 * np.abs(lu_ref).max()
    _check_backward(A, LU, M.ipiv - 1)
    nc = max(1, (2 * N) // 3)
    B = rng.standard_normal((N, nc))
    t = M.TraceMInvdM(B)
    X = sl.lu_solve((lu_ref, piv_ref), B)
    # forward error of one solution: cond(A) N u, times the root of nc terms
    tol = np.linalg.cond(A) * N * U * np.linalg.norm(X)
    assert t.imag == 0.0 and abs(t.real - np.trace(X[:nc])) <= tol


@pytest.mark.parametrize("pec", [True, False])
def test_complex_trace_matches_lapack(pec):
    """Tr[M^-1 B] of a complex128 matrix: halves of 32-row blocks with
    remainders (N = 400 and 800, a panel and three quarters)."""
    import scipy.linalg as sl
    from gbem import RWGGeometry, mesh
    from gbem._lib import C128
    from gbem.api import HMatrix, Material
    V, P = mesh.rounded_cube(270, seed=1)
    G = RWGGeometry([{"V": V, "P": P, "material": None if pec else Material(2.0)}])
    M = HMatrix(G, C128)
    N = M.N
    rng = np.random.default_rng(N)
    A = rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))
    M.set(A)
    assert M.LUFactorize() == 0
    B = rng.standard_normal((N, 100)) + 1j * rng.standard_normal((N, 100))
    X = sl.solve(A, B)
    tol = np.linalg.cond(A) * N * U * np.linalg.norm(X)
    assert abs(M.TraceMInvdM(B) - np.trace(X[:100])) <= tol


@pytest.mark.parametrize("N,nrhs", [(1, 1), (31, 2), (32, 3), (33, 8), (64, 9), (65, 1), (200, 5), (609, 8), (777, 17)])
def test_triangular_solve_edges(N, nrhs):
    """Blocks of 32 rows, columns in groups of eight, more blocks than CTAs of
    a group.  The solve applies the inverses of the diagonal blocks, so its
    backward error is N u |L| |U| |x| times the blocks' condition, componentwise
    || |D^-1| |D| ||."""
    from gbem._lib import lib
    rng = np.random.default_rng(N + nrhs)
    A = rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))
    B = rng.standard_normal((N, nrhs)) + 1j * rng.standard_normal((N, nrhs))
    LU, piv = _factor(A)
    X = np.asfortranarray(B.copy())
    ipiv = (piv + 1).astype(np.int32)
    assert lib().gbem_lu_solve_host(LU.ctypes.data, N, N, ipiv.ctypes.data, b"N", nrhs, X.ctypes.data, N) == 0
    L, R = np.tril(LU, -1) + np.eye(N), np.triu(LU)
    cond = 1.0
    for k in range(0, N, 32):
        for D in (L[k:k + 32, k:k + 32], R[k:k + 32, k:k + 32]):
            cond = max(cond, (np.abs(np.linalg.inv(D)) @ np.abs(D)).sum(axis=1).max())
    bound = 16 * N * U * cond * (np.abs(L) @ (np.abs(R) @ np.abs(X))).max(axis=0)
    assert (np.abs(A @ X - B).max(axis=0) <= bound).all()


@pytest.mark.parametrize("N", [272, 288, 304, 336, 400, 417, 560, 600, 1700])
def test_block_row_solve_edges(N):
    """The block rows right of a panel (substitution of 128 rows up to 1280
    columns, by halves with tensor-core updates beyond) and inside it, one, two
    and four columns per CTA, a last block of half its rows."""
    rng = np.random.default_rng(3 * N)
    A = rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))
    LU, piv = _factor(A)
    _check_backward(A, LU, piv)


@pytest.mark.parametrize("N", [1, 2, 3, 4, 5, 15, 16, 17, 20, 31, 33, 47, 63, 65, 130, 512, 1023, 1025, 1041])
def test_leaf_lanes_per_row(N):
    """Panels whose rows are spread over four lanes (up to 64 rows a CTA), where
    a leaf, a group of four columns or that range ends."""
    import scipy.linalg as sl
    rng = np.random.default_rng(7 * N)
    A = rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))
    LU, piv = _factor(A)
    assert np.array_equal(piv, sl.lu_factor(A)[1])
    _check_backward(A, LU, piv)


def _componentwise(A, LU, piv):
    """max |P A - L U| / (|L| |U|) over sampled rows, in extended precision."""
    N = A.shape[0]
    perm = np.arange(N)
    for i, p in enumerate(piv):
        perm[[i, p]] = perm[[p, i]]
    rows = np.unique(np.concatenate([np.linspace(0, N - 1, 24).astype(int), np.arange(max(0, N - 8), N)]))
    ext = np.longdouble if not np.iscomplexobj(A) else np.clongdouble
    L, R = (np.tril(LU, -1) + np.eye(N))[rows].astype(ext), np.triu(LU).astype(ext)
    scale = np.abs(L) @ np.abs(R)
    err = np.abs(A[perm][rows].astype(ext) - L @ R)
    return float((err[scale > 0] / scale[scale > 0]).max())


def _graded(kind, N, rng, real):
    A = rng.standard_normal((N, N))
    if not real:
        A = A + 1j * rng.standard_normal((N, N))
    if kind[0] == "rows":        # row scales spread evenly, the smallest first
        return A * 10.0 ** np.linspace(-kind[1], 0.0, N)[:, None]
    if kind[0] == "both":
        s = 10.0 ** rng.uniform(-kind[1], 0.0, N)
        return A * s[:, None] * rng.permutation(s)
    if kind[0] == "coupled":     # two sets of unknowns in turn, weakly coupled
        i = np.arange(N)
        return A * np.where((i[:, None] + i) % 2, 10.0 ** -kind[1], 1.0)
    if kind[0] == "entries":
        return A * 10.0 ** rng.uniform(-kind[1], 0.0, (N, N))
    i = np.arange(N)             # "arrow": zero except a band, a full row and a full column
    return A * ((np.abs(i[:, None] - i) < 40) | (i[:, None] > N - 4) | (i > N - 4)) * 10.0 ** np.linspace(-kind[1], 0.0, N)[:, None]


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("kind", [("rows", 0), ("rows", 12), ("rows", 18), ("rows", 30), ("both", 20), ("coupled", 2),
                                  ("coupled", 6), ("coupled", 12), ("entries", 8), ("arrow", 18)])
def test_factor_is_as_accurate_as_lapack_entry_by_entry(kind, real):
    """|P A - L U| against |L| |U|, entry by entry, where rows, columns or
    blocks differ in scale: within eight times LAPACK's own factorisation of the
    same matrix (another order of the same FP64 sums) and eight roundings."""
    import scipy.linalg as sl
    N = 400
    A = _graded(kind, N, np.random.default_rng(int(kind[1]) + 100 * real), real)
    lu_ref, piv_ref = sl.lu_factor(A)
    ref = _componentwise(A, lu_ref, piv_ref)
    if real:
        from gbem._lib import F64
        from gbem.api import HMatrix
        M = HMatrix(_strip(N), F64)
        M.set(A)
        assert M.LUFactorize() == 0
        LU, piv = M.numpy(), M.ipiv - 1
    else:
        LU, piv = _factor(A)
    got = _componentwise(A, LU, piv)
    print("componentwise error / u: %.2f (LAPACK %.2f)" % (got / U, ref / U))
    assert got <= 8 * ref + 8 * U


def test_wide_tiles_are_as_accurate_as_lapack_entry_by_entry():
    """The same where the trailing update takes 128-column tiles (N = 1300),
    some of them with graded rows, some with even ones, a ragged last one."""
    import scipy.linalg as sl
    N = 1300
    rng = np.random.default_rng(5)
    A = rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))
    A[:700] *= 10.0 ** np.linspace(-18.0, 0.0, 700)[:, None]
    lu_ref, piv_ref = sl.lu_factor(A)
    LU, piv = _factor(A)
    got, ref = _componentwise(A, LU, piv), _componentwise(A, lu_ref, piv_ref)
    print("componentwise error / u: %.2f (LAPACK %.2f)" % (got / U, ref / U))
    assert got <= 8 * ref + 8 * U


_NO_TENSOR = r"""
import sys
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/tests", sys.argv[1] + "/scuff-em_gb300"]
import numpy as np, scipy.linalg as sl
import test_gpu_lu64 as t
A = t._graded(("rows", 18), 400, np.random.default_rng(1), False)
LU, piv = t._factor(A)
assert t._componentwise(A, LU, piv) <= 8 * t._componentwise(A, *sl.lu_factor(A)) + 8 * t.U
np.save(sys.argv[2], LU)
"""


def test_tensor_updates_can_be_switched_off(tmp_path):
    """GBEM_LU_TC=0 takes every update in FP64 multiplications: as accurate, and
    not the same last bits as the slices'."""
    import os
    import subprocess
    import sys
    repo = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    for tc in ("0", "1"):
        subprocess.run([sys.executable, "-c", _NO_TENSOR, repo, str(tmp_path / ("lu%s.npy" % tc))],
                       env=dict(os.environ, GBEM_LU_TC=tc), check=True, timeout=600)
    assert not np.array_equal(np.load(tmp_path / "lu0.npy"), np.load(tmp_path / "lu1.npy"))


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("power", [-530, -520, -505, 505, 520, 900])
def test_pivots_of_extreme_size(power, real):
    """Pivots whose |z|^2 leaves the FP64 range: a matrix times a power of two
    has the same L, and U times that power, exactly."""
    N = 150
    rng = np.random.default_rng(9)
    A = rng.standard_normal((N, N))
    if not real:
        A = A + 1j * rng.standard_normal((N, N))
    out = []
    for s in (1.0, 2.0 ** power):
        if real:
            from gbem._lib import F64
            from gbem.api import HMatrix
            M = HMatrix(_strip(N), F64)
            M.set(A * s)
            assert M.LUFactorize() == 0
            out.append((M.numpy(), M.ipiv))
        else:
            out.append(_factor(A * s))
    (F0, p0), (F1, p1) = out
    assert np.array_equal(p0, p1)
    assert np.array_equal(np.tril(F0, -1), np.tril(F1, -1))
    assert np.array_equal(np.triu(F0) * 2.0 ** power, np.triu(F1))


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("power", [-1015, -960, 960, 1015])
def test_updates_at_the_ends_of_the_range(power, real):
    """Sums of the updates that are subnormal or close to overflow: the backward
    error of the scaled factors, entry by entry, with one subnormal spacing of
    2^-1074 for each of the N subtractions beside the relative error."""
    N = 300
    rng = np.random.default_rng(13)
    A = rng.standard_normal((N, N))
    if not real:
        A = A + 1j * rng.standard_normal((N, N))
    A = A * 2.0 ** power
    if real:
        from gbem._lib import F64
        from gbem.api import HMatrix
        M = HMatrix(_strip(N), F64)
        M.set(A)
        assert M.LUFactorize() == 0
        LU, piv = M.numpy(), M.ipiv - 1
    else:
        LU, piv = _factor(A)
    perm = np.arange(N)
    for i, p in enumerate(piv):
        perm[[i, p]] = perm[[p, i]]
    L, R = np.tril(LU, -1) + np.eye(N), np.triu(LU)
    assert np.isfinite(R).all() and np.abs(L).max() <= np.sqrt(2.0) * (1 + 1e-12)
    # in units of 2^power, where every product is a normal number
    R0 = R * 2.0 ** (-power // 2) * 2.0 ** (-power - (-power // 2))
    A0 = A * 2.0 ** (-power // 2) * 2.0 ** (-power - (-power // 2))
    tiny = 2.0 ** max(-1074 - power, -1074)
    bound = 8 * N * (U * (np.abs(L) @ np.abs(R0) + np.abs(A0[perm])) + tiny)
    assert (np.abs(A0[perm] - L @ R0) <= bound).all()
