"""The one-launch triangular solves: every value sent between the CTAs of a cluster is awaited before
its place is used again, so a solve gives the same bits every time, whatever runs beside it."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from fluidlets_gb300 import _device as dv  # noqa: E402
from fluidlets_gb300 import _lib  # noqa: E402

pytestmark = pytest.mark.gpu


def factored(n, seed):
    rng = np.random.default_rng(seed)
    A = rng.normal(size=(n, n))
    L = _lib.load()
    Ad = torch.tensor(A, device="cuda")
    piv = torch.empty(n, dtype=torch.int32, device="cuda")
    nb = L.flg_lu_factor_f64_workspace(n)
    ws = dv.workspace(nb)
    info = ctypes.c_int(0)
    _lib.check(L.flg_lu_factor_f64(n, dv.ptr(Ad), n, dv.ptr(piv), ctypes.byref(info), dv.ptr(ws), nb, dv.stream()))
    return A, Ad, piv


# block counts of one, one per CTA of the cluster, one more, two per CTA, and a ragged last block
@pytest.mark.parametrize("n", [32, 500, 512, 513, 544, 1024, 1025, 1537])
def test_repeated_solves_give_the_same_bits(n):
    A, LU, piv = factored(n, n)
    L = _lib.load()
    rng = np.random.default_rng(n + 1)
    nrhs = 3
    b = rng.normal(size=(n, nrhs))
    bd = torch.tensor(b, device="cuda")
    junk = torch.empty(1 << 24, dtype=torch.float32, device="cuda")
    other = torch.cuda.Stream()
    first = None
    for k in range(40):
        B = bd.clone()
        if k % 2:  # traffic beside the exchange
            with torch.cuda.stream(other):
                junk.fill_(float(k))
        _lib.check(L.flg_lu_solve_f64(n, nrhs, dv.ptr(LU), n, dv.ptr(piv), dv.ptr(B), nrhs, dv.stream()))
        first = B if first is None else first
        assert torch.equal(B, first)
    torch.cuda.synchronize()
    x = first.cpu().numpy().astype(np.longdouble)
    F = LU.cpu().numpy()
    scale = np.abs(np.tril(F, -1) + np.eye(n)) @ (np.abs(np.triu(F)) @ np.abs(x).astype(float))
    # backward error of the factors and the substitutions, 3 n u |L| |U| |x| in all, in the largest row
    assert np.abs(A @ x - b).max() <= 3 * n * 2.0**-53 * scale.max()


@pytest.mark.parametrize("n,nrhs", [(1, 1), (513, 2), (100, 40)])
def test_flagged_solves(n, nrhs):
    """The same bits, with the outcome of the waits in a word of the caller's."""
    _, LU, piv = factored(n, n + 7)
    L = _lib.load()
    B = torch.randn((n, nrhs), dtype=torch.float64, device="cuda")
    X, Y = B.clone(), B.clone()
    flag = torch.full((1,), 77, dtype=torch.int32, device="cuda")
    args = (n, nrhs, dv.ptr(LU), n, dv.ptr(piv))
    _lib.check(L.flg_lu_solve_f64(*args, dv.ptr(X), nrhs, dv.stream()))
    _lib.check(L.flg_lu_solve_f64_flag(*args, dv.ptr(Y), nrhs, dv.ptr(flag), dv.stream()))
    assert torch.equal(X, Y) and int(flag) == 0
    assert L.flg_lu_solve_f64_flag(*args, dv.ptr(Y), nrhs, None, dv.stream()) == _lib.FLG_ERR_INVALID
    assert L.flg_lu_solve_f64_flag(n, nrhs, dv.ptr(LU), n - 1, dv.ptr(piv), dv.ptr(Y), nrhs, dv.ptr(flag),
                                   dv.stream()) == _lib.FLG_ERR_INVALID


def test_a_raised_flag_reaches_python():
    from fluidlets_gb300.core import _SolveFlag

    flag = _SolveFlag("cuda")
    flag.word.zero_()
    flag.check()
    flag.word.fill_(1)
    with pytest.raises(RuntimeError, match="timed out"):
        flag.check()


@pytest.mark.parametrize("n,col", [(20, 19), (32, 31), (40, 39), (70, 50)])
@pytest.mark.parametrize("big,small", [(1e160, 1e-160), (1e-200, 1e150)])
def test_columns_far_from_their_pivots(n, col, big, small):
    """An upper-triangular matrix with one column that is 1e320 times its diagonal entry (or 1e-350 of it): the
    quotient of the two is not a number, the solution is."""
    rng = np.random.default_rng(n)
    A = np.eye(n)
    A[:col, col] = big * rng.uniform(1, 2, col)
    A[col, col] = small
    b = rng.normal(size=(n, 1))
    b[col] = 1e-200 * small if big > 1 else 1e130 * small
    x = b.copy()
    x[col] = b[col] / small
    x[:col] -= A[:col, col:col + 1] * x[col]
    L = _lib.load()
    Ad, B = torch.tensor(A, device="cuda"), torch.tensor(b, device="cuda")
    piv = torch.arange(n, dtype=torch.int32, device="cuda")
    _lib.check(L.flg_lu_solve_f64(n, 1, dv.ptr(Ad), n, dv.ptr(piv), dv.ptr(B), 1, dv.stream()))
    got = B.cpu().numpy()
    assert np.all(np.abs(got - x) <= 4 * 2.0**-53 * (np.abs(b) + np.abs(A[:, col:col + 1] * x[col])) + 4 * 2.0**-53 * np.abs(x))
