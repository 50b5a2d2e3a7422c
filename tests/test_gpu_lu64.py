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
