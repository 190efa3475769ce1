"""The FP64 LU: panels, row interchanges and the sliced tensor-core trailing update at the edges
of their tiles, against extended-precision products of the factors."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from fluidlets_gb300 import _device as dv  # noqa: E402
from fluidlets_gb300 import _lib  # noqa: E402

pytestmark = pytest.mark.gpu


def factor(A, ld=None):
    """(L, U, permuted row order, packed factors) of the library's LU, leading dimension ld."""
    L = _lib.load()
    n = A.shape[0]
    ld = n if ld is None else ld
    Ad = torch.full((n, ld), 7.5, dtype=torch.float64, device="cuda")
    Ad[:, :n] = torch.tensor(A, device="cuda")
    piv = torch.empty(n, dtype=torch.int32, device="cuda")
    nb = L.flg_lu_factor_f64_workspace(n)
    ws = dv.workspace(nb)
    info = ctypes.c_int(0)
    _lib.check(L.flg_lu_factor_f64(n, dv.ptr(Ad), ld, dv.ptr(piv), ctypes.byref(info), dv.ptr(ws), nb, dv.stream()))
    assert torch.all(Ad[:, n:] == 7.5)
    F, p = Ad[:, :n].cpu().numpy(), piv.cpu().numpy()
    rows = np.arange(n)
    for k in range(n):
        rows[[k, p[k]]] = rows[[p[k], k]]
    return np.tril(F, -1) + np.eye(n), np.triu(F), rows


def residual(A, Lo, U, rows, sample):
    """max |P A - L U| over sampled rows, the products in extended precision, and max |L| |U|."""
    Ll, Ul = Lo[sample].astype(np.longdouble), U.astype(np.longdouble)
    R = A[rows][sample].astype(np.longdouble) - Ll @ Ul
    return float(np.abs(R).max()), float((np.abs(Lo[sample]) @ np.abs(U)).max())


@pytest.mark.parametrize("n", [64, 65, 96, 97, 127, 128, 129, 160, 191, 192, 193, 257, 320, 700])
def test_factors_reproduce_the_matrix(n):
    rng = np.random.default_rng(n)
    A = rng.normal(size=(n, n))
    Lo, U, rows = factor(A, ld=n + n % 3)
    assert np.abs(Lo).max() <= 1.0 + 2.0**-52  # partial pivoting
    sample = np.unique(np.r_[0, n - 1, rng.integers(0, n, 40)])
    r, scale = residual(A, Lo, U, rows, sample)
    # the classical componentwise bound n u |L| |U| of Gaussian elimination in FP64
    assert r <= n * 2.0**-53 * scale


def test_trailing_update_rounds_less_than_an_fma_chain():
    """A matrix whose Schur complement is a plain product: [[I, B], [C, S + C B]] with |C| < 1 is
    eliminated without interchanges, U12 = B and L21 = C exactly, so U22 of a diagonal S shows
    the update's own rounding: at most one rounding of the product and one of the difference."""
    rng = np.random.default_rng(5)
    k, m = 64, 130
    B = rng.normal(size=(k, m)) * 10.0 ** rng.integers(-3, 4, m)
    C = rng.uniform(-0.99, 0.99, (m, k)) * 2.0 ** -rng.integers(0, 12, (m, 1))
    P = (C.astype(np.longdouble) @ B.astype(np.longdouble))
    scale = np.abs(C).max(1)[:, None] * np.abs(B).max(0)[None, :]
    D = np.zeros((m, m))
    A = np.block([[np.eye(k), B], [C, D]])
    Lo, U, rows = factor(A)
    assert np.array_equal(rows[:k], np.arange(k)) and np.array_equal(U[:k, k:], B)
    first = rows[k] - k  # the first row of the Schur complement that is eliminated keeps its values
    u = U[k, k:]
    err = np.abs(u.astype(np.longdouble) + P[first])
    assert np.all(err <= 2.0**-53 * np.abs(P[first]) * 2 + 2.0**-55 * scale[first])


@pytest.mark.parametrize("er,ec", [(0, 300), (-300, 0), (-280, 280), (200, 200)])
def test_extreme_row_and_column_scales(er, ec):
    rng = np.random.default_rng(3000 + er + 7 * ec)
    n = 150
    A = rng.normal(size=(n, n)) + 4 * np.eye(n)
    sr, sc = 2.0 ** rng.integers(min(er, 0), max(er, 0) + 1, n), 2.0 ** rng.integers(min(ec, 0), max(ec, 0) + 1, n)
    S = A * sr[:, None] * sc[None, :]
    Lo, U, rows = factor(S)
    # column scaling by powers of two scales U exactly, so the bound holds column by column
    R = S[rows].astype(np.longdouble) - Lo.astype(np.longdouble) @ U.astype(np.longdouble)
    assert np.all(np.abs(R).max(0) <= n * 2.0**-53 * (np.abs(Lo) @ np.abs(U)).max(0))


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("at", [(3, 5), (100, 140), (150, 20)])
def test_non_finite_entries_are_reported(bad, at):
    rng = np.random.default_rng(1)
    A = rng.normal(size=(170, 170))
    A[at] = bad
    with pytest.raises(np.linalg.LinAlgError):
        factor(A)


def test_zero_rows_are_singular():
    rng = np.random.default_rng(2)
    A = rng.normal(size=(200, 200))
    A[130] = 0.0
    with pytest.raises(np.linalg.LinAlgError):
        factor(A)


@pytest.mark.parametrize("n,nrhs", [(1, 1), (31, 1), (32, 2), (33, 1), (64, 3), (65, 1), (511, 1), (513, 2), (1030, 1),
                                    (100, 33)])
def test_triangular_solves_backward_error(n, nrhs):
    """The library's solve with its own factors: componentwise backward error of two substitutions,
    (2 n + 2) u |L| |U| |x|, taken as 3 n u for small n's constants."""
    rng = np.random.default_rng(n + nrhs)
    A = rng.normal(size=(n, n))
    b = rng.normal(size=(n, nrhs))
    L = _lib.load()
    Ad = torch.tensor(A, device="cuda")
    B = torch.full((n, nrhs + 2), 3.25, dtype=torch.float64, device="cuda")
    B[:, :nrhs] = torch.tensor(b, device="cuda")
    piv = torch.empty(n, dtype=torch.int32, device="cuda")
    nb = L.flg_lu_factor_f64_workspace(n)
    ws = dv.workspace(nb)
    info = ctypes.c_int(0)
    _lib.check(L.flg_lu_factor_f64(n, dv.ptr(Ad), n, dv.ptr(piv), ctypes.byref(info), dv.ptr(ws), nb, dv.stream()))
    _lib.check(L.flg_lu_solve_f64(n, nrhs, dv.ptr(Ad), n, dv.ptr(piv), dv.ptr(B), nrhs + 2, dv.stream()))
    assert torch.all(B[:, nrhs:] == 3.25)
    F, p, x = Ad.cpu().numpy(), piv.cpu().numpy(), B[:, :nrhs].cpu().numpy()
    for k in range(n):
        b[[k, p[k]]] = b[[p[k], k]]
    Lo, U = np.tril(F, -1) + np.eye(n), np.triu(F)
    r = Lo.astype(np.longdouble) @ (U.astype(np.longdouble) @ x.astype(np.longdouble)) - b
    assert np.all(np.abs(r) <= 3 * max(n, 4) * 2.0**-53 * (np.abs(Lo) @ (np.abs(U) @ np.abs(x)) + np.abs(b)))
