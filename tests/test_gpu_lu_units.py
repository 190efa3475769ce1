"""The FP64 LU on matrices whose rows and columns differ in scale: the bound of Gaussian elimination in
FP64, |P A - L U| <= n u |L| |U|, holds entry by entry, and systems of mixed units keep their digits."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fluidlets_gb300 as fl  # noqa: E402
import oracle as O  # noqa: E402
from fluidlets_gb300 import _device as dv  # noqa: E402
from fluidlets_gb300 import _lib  # noqa: E402

pytestmark = pytest.mark.gpu


def factor(A):
    L = _lib.load()
    n = A.shape[0]
    Ad = torch.tensor(A, device="cuda")
    piv = torch.empty(n, dtype=torch.int32, device="cuda")
    nb = L.flg_lu_factor_f64_workspace(n)
    ws = dv.workspace(nb)
    info = ctypes.c_int(0)
    _lib.check(L.flg_lu_factor_f64(n, dv.ptr(Ad), n, dv.ptr(piv), ctypes.byref(info), dv.ptr(ws), nb, dv.stream()))
    F, p = Ad.cpu().numpy(), piv.cpu().numpy()
    rows = np.arange(n)
    for k in range(n):
        rows[[k, p[k]]] = rows[[p[k], k]]
    return np.tril(F, -1) + np.eye(n), np.triu(F), rows


def matrix(kind, n, rng):
    A = rng.normal(size=(n, n))
    if kind == "half the rows":
        A[n // 2:] *= 1e-20
    elif kind == "half the columns":
        A[:, n // 2:] *= 1e-20
    elif kind == "every third row":
        A[::3] *= 1e-12
    elif kind == "rows over 24 decades":
        A *= 10.0 ** rng.uniform(-12, 12, (n, 1))
    elif kind == "rows over 90 decades":
        A *= 2.0 ** rng.integers(-300, 1, (n, 1))
    elif kind == "rows and columns":
        A *= 10.0 ** rng.uniform(-12, 12, (n, 1)) * 10.0 ** rng.uniform(-12, 12, n)
    elif kind == "entries over 16 decades":
        A *= 10.0 ** rng.uniform(-8, 8, (n, n))
    elif kind == "sparse":
        A *= rng.random((n, n)) < 0.03
        A[np.arange(n), rng.permutation(n)] += 2.0
    elif kind == "weakly coupled":  # two systems whose unknowns alternate
        A *= np.where((np.arange(n)[:, None] + np.arange(n)) % 2, 1e-25, 1.0)
    elif kind == "filament":
        t = np.linspace(0.0, 1.0, (n + 2) // 3)
        A = O.assemble("stokeslet", np.c_[t, 0.1 * np.sin(9 * t), 0 * t], np.c_[t, 0.1 * np.sin(9 * t), 0 * t],
                       1.0 / len(t))[:n, :n]
    return np.ascontiguousarray(A)


KINDS = ["half the rows", "half the columns", "every third row", "rows over 24 decades", "rows over 90 decades",
         "rows and columns", "entries over 16 decades", "sparse", "weakly coupled", "filament"]


@pytest.mark.parametrize("n", [129, 200, 257])
@pytest.mark.parametrize("kind", KINDS)
def test_bound_of_every_entry(kind, n):
    A = matrix(kind, n, np.random.default_rng(n))
    Lo, U, rows = factor(A)
    R = np.abs(A[rows].astype(np.longdouble) - Lo.astype(np.longdouble) @ U.astype(np.longdouble))
    assert np.all(R <= n * 2.0**-53 * (np.abs(Lo) @ np.abs(U)))


@pytest.mark.parametrize("exponent", [0, 13, 20, 30, 40, -30])
def test_rigid_body_in_a_very_viscous_fluid(exponent):
    """The mobility rows scale as 1 / mu, the force and torque rows not at all.  The forces do not depend on
    mu, velocities are proportional to 1 / mu; for a power of two both exactly so."""
    X = O.fibonacci_sphere(100)
    e = 0.5 * np.sqrt(4 * np.pi / 100)
    F, T = np.array([1.0, -2.0, 0.5]), np.array([0.3, 0.1, -0.7])
    mu = 2.0**exponent
    U, W, f = fl.rigid_body_mobility(fl.Stokeslet3D(), X, e, F, T, mu=mu)
    # the system at mu = 1 in NumPy
    n = 300
    A = np.zeros((n + 6, n + 6))
    A[:n, :n] = O.assemble("stokeslet", X, X, e)
    C = np.zeros((n, 3))
    for k, (x, y, z) in enumerate(X - X.mean(0)):
        C[3 * k:3 * k + 3] = [[0, -z, y], [z, 0, -x], [-y, x, 0]]
    D = np.zeros((3, n))
    for k, (x, y, z) in enumerate(X):
        D[:, 3 * k:3 * k + 3] = [[0, -z, y], [z, 0, -x], [-y, x, 0]]
    A[:n, n:] = np.c_[-np.tile(np.eye(3), (100, 1)), C]
    A[n:, :n] = np.r_[np.tile(np.eye(3), (1, 100)), D]
    rhs = np.r_[np.zeros(n), F, T + np.cross(X.mean(0), F)]
    ref = np.linalg.solve(A, rhs)
    tol = (n + 6) * 2.0**-53 * np.linalg.cond(A)
    assert np.linalg.norm(f.ravel() - ref[:n]) <= tol * np.linalg.norm(ref)
    assert np.linalg.norm(np.r_[U, W] * mu - ref[n:]) <= tol * np.linalg.norm(ref)
    # 1e-12: a thousand roundings, where the condition number lets both solves differ by more
    if exponent:
        U1, W1, f1 = fl.rigid_body_mobility(fl.Stokeslet3D(), X, e, F, T)
        assert np.abs(f - f1).max() <= 1e-12 * np.abs(f1).max()
        assert np.abs(np.r_[U, W] * mu - np.r_[U1, W1]).max() <= 1e-12 * np.abs(np.r_[U1, W1]).max()
