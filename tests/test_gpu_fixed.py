"""FP64 sums whose pairs run in fixed point: short and ragged splits, the ranges that leave the
fixed-point path, and scales far from one, against the oracle's FP64 loops."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fluidlets_gb300 as fl  # noqa: E402
import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu

KERNELS = [(fl.Stokeslet3D(), "stokeslet", 0.0), (fl.WallStokeslet3D(), "wall", 0.0),
           (fl.Brinkmanlet3D(0.0), "brinkman", 0.0), (fl.Brinkmanlet3D(2.5), "brinkman", 2.5),
           (fl.Brinkmanlet3D(40.0), "brinkman", 40.0)]
IDS = ["stokeslet", "wall", "alpha0", "alpha2.5", "alpha40"]


def points(rng, m, n, scale=1.0):
    X = np.c_[rng.uniform(-1, 1, (m, 2)), rng.uniform(0.0, 2.0, m)] * scale
    Y = np.c_[rng.uniform(-1, 1, (n, 2)), rng.uniform(0.02, 2.0, n)] * scale
    return X, Y


def oracle_sum(name, alpha, *args):
    return O.evaluate(name, *args, alpha=alpha) if name == "brinkman" else O.evaluate(name, *args)


def check(kernel, name, alpha, X, Y, F, e, tol):
    """Relative L2 against the oracle: n terms of a few roundings each on both sides."""
    u = fl.evaluate(kernel, X, Y, F, e)
    ref = oracle_sum(name, alpha, X, Y, F, e)
    assert np.linalg.norm(u - ref) <= tol * np.linalg.norm(ref)
    return u, ref


@pytest.mark.parametrize("m,n", [(1, 1), (1, 7), (3, 8), (127, 15), (128, 16), (129, 17), (5, 63), (130, 65), (40, 1025)])
@pytest.mark.parametrize("kernel,name,alpha", KERNELS, ids=IDS)
def test_ragged_sizes(kernel, name, alpha, m, n):
    rng = np.random.default_rng(m * 1000 + n)
    X, Y = points(rng, m, n)
    X[0] = Y[0]  # a pair at distance zero
    F = rng.normal(size=(n, 3))
    F[::5, 1] = 0.0
    check(kernel, name, alpha, X, Y, F, 0.05 * rng.uniform(0.5, 2.0, n), 1e-13)


@pytest.mark.parametrize("scale", [1e-90, 1e-12, 1e9, 1e85])
@pytest.mark.parametrize("kernel,name,alpha", KERNELS[:3], ids=IDS[:3])
def test_scales(kernel, name, alpha, scale):
    rng = np.random.default_rng(3)
    X, Y = points(rng, 40, 60, scale)
    F = rng.normal(size=(60, 3)) * 10.0 ** rng.integers(-8, 8, (60, 1))
    # the kernels are homogeneous of degree -1: the oracle runs at scale 1, where its s^5 cannot overflow
    ref = oracle_sum(name, alpha, X / scale, Y / scale, F, 0.03) / scale
    u = fl.evaluate(kernel, X, Y, F, 0.03 * scale)
    assert np.linalg.norm(u * scale - ref * scale) <= 1e-13 * np.linalg.norm(ref * scale)


@pytest.mark.parametrize("kernel,name,alpha", KERNELS[:2], ids=IDS[:2])
def test_complex_strengths_and_tiny_blobs(kernel, name, alpha):
    rng = np.random.default_rng(4)
    X, Y = points(rng, 70, 90)
    X[:30] = Y[:30] + 1e-7 * rng.normal(size=(30, 3))
    X[:, 2] = np.abs(X[:, 2])
    F = rng.normal(size=(90, 3)) + 1j * rng.normal(size=(90, 3))
    check(kernel, name, alpha, X, Y, F, 1e-6, 1e-12)


def test_targets_on_and_below_the_wall():
    rng = np.random.default_rng(5)
    X, Y = points(rng, 60, 50)
    X[:20, 2] = 0.0
    X[20:30, 2] *= -1.0
    F = rng.normal(size=(50, 3))
    u, ref = check(fl.WallStokeslet3D(), "wall", 0.0, X, Y, F, 0.05, 1e-12)
    assert np.all(u[:20] == 0.0)


def test_plane_problems_stay_in_the_plane():
    rng = np.random.default_rng(6)
    X, Y = points(rng, 50, 200)
    X[:, 1] = Y[:, 1] = 0.25
    F = rng.normal(size=(200, 3))
    F[:, 1] = 0.0
    for kernel, name, alpha in KERNELS:
        u, _ = check(kernel, name, alpha, X, Y, F, 0.05, 1e-13)
        assert np.all(u[:, 1] == 0.0)


def test_non_finite_and_extreme_strengths():
    rng = np.random.default_rng(7)
    X, Y = points(rng, 20, 40)
    F = rng.normal(size=(40, 3))
    F[3] = 1e-305
    F[4] = [1e300, -1e280, 0.0]
    F[5] = 0.0
    check(fl.Stokeslet3D(), "stokeslet", 0.0, X, Y, F, 0.05, 1e-13)
    F[7, 1] = np.nan
    assert np.all(np.isnan(fl.evaluate(fl.Stokeslet3D(), X, Y, F, 0.05)).any(axis=1))
    F[7, 1] = np.inf
    assert not np.isfinite(fl.evaluate(fl.Stokeslet3D(), X, Y, F, 0.05)).all(axis=1).any()
    X[4] = np.nan
    F[7] = 0.0
    u = fl.evaluate(fl.WallStokeslet3D(), X, Y, F, 0.05)
    assert np.all(np.isnan(u[4])) and np.isfinite(u[:4]).all()


def test_zero_blob_on_a_source_is_not_finite():
    X = np.array([[0.1, 0.2, 0.3], [0.4, 0.5, 0.6]])
    u = fl.evaluate(fl.Stokeslet3D(), X, X[:1], np.ones((1, 3)), 0.0)
    assert not np.isfinite(u[0]).any() and np.isfinite(u[1]).all()


COMPLEX = [complex(0.7, 0.7), 3.0 - 1.0j, 1.0 + 1.6j, 60.0 * (1 + 1j), 1e-4 * (1 + 1j), 0.05 + 0.9j, 2.0 + 0.01j]


@pytest.mark.parametrize("m,n", [(1, 1), (3, 8), (129, 17), (40, 1025)])
@pytest.mark.parametrize("alpha", COMPLEX)
@pytest.mark.parametrize("strengths", ["real", "complex"])
def test_complex_alpha(alpha, strengths, m, n):
    """All of |z| from the series to vanished exponentials; the last two alphas take the FP64 pairs."""
    rng = np.random.default_rng(m * 1000 + n)
    X, Y = points(rng, m, n)
    X[0] = Y[0]
    F = rng.normal(size=(n, 3))
    F = F + 1j * rng.normal(size=(n, 3)) if strengths == "complex" else F
    e = 0.05 * rng.uniform(0.5, 2.0, n)
    u, ref = check(fl.Brinkmanlet3D(alpha), "brinkman", alpha, X, Y, F, e, 1e-13)
    if strengths == "real":  # both parts to their own precision (a loss of |Re| / |Im| <= 100 in the last)
        for a, b in ((u.real, ref.real), (u.imag, ref.imag)):
            assert np.linalg.norm(a - b) <= 1e-11 * np.linalg.norm(b)


def test_complex_alpha_scales_and_tiny_imaginary_strengths():
    rng = np.random.default_rng(8)
    X, Y = points(rng, 50, 70)
    F = rng.normal(size=(70, 3)) + 1e-9j * rng.normal(size=(70, 3))
    for s in (1e-40, 1.0, 1e40):  # alpha L fixed: homogeneous of degree -1
        u = fl.evaluate(fl.Brinkmanlet3D((0.8 + 0.6j) / s), X * s, Y * s, F, 0.03 * s) * s
        ref = O.evaluate("brinkman", X, Y, F, 0.03, alpha=0.8 + 0.6j)
        assert np.linalg.norm(u - ref) <= 1e-13 * np.linalg.norm(ref)
    for kernel, name in ((fl.Stokeslet3D(), "stokeslet"), (fl.WallStokeslet3D(), "wall")):
        u, ref = fl.evaluate(kernel, X, Y, F, 0.03), O.evaluate(name, X, Y, F, 0.03)
        assert np.linalg.norm(u.imag - ref.imag) <= 1e-12 * np.linalg.norm(ref.imag)


def test_complex_alpha_non_finite_strengths():
    rng = np.random.default_rng(9)
    X, Y = points(rng, 20, 40)
    F = rng.normal(size=(40, 3)) + 1j * rng.normal(size=(40, 3))
    F[7, 1] = complex(0.0, np.nan)
    assert np.all(np.isnan(fl.evaluate(fl.Brinkmanlet3D(1 + 1j), X, Y, F, 0.05)).any(axis=1))


@pytest.mark.parametrize("strengths", ["real", "complex"])
def test_complex_alpha_near_field(strengths):
    rng = np.random.default_rng(10)
    X, Y = points(rng, 600, 900)
    F = rng.normal(size=(900, 3))
    F = F + 1j * rng.normal(size=(900, 3)) if strengths == "complex" else F
    for alpha in (2.0 + 2.0j, 0.3 + 2.0j):
        ref = O.evaluate("brinkman", X, Y, F, 0.05, alpha=alpha)
        u = fl.evaluate(fl.Brinkmanlet3D(alpha), X, Y, F, 0.05, precision="mixed")
        assert np.linalg.norm(u - ref) <= 5e-6 * np.linalg.norm(ref)


# ---- matrices ---------------------------------------------------------------------------------
def oracle_matrix(name, alpha, *args):
    return O.assemble(name, *args, alpha=alpha) if name == "brinkman" else O.assemble(name, *args)


@pytest.mark.parametrize("m,n", [(1, 1), (2, 31), (9, 32), (8, 33), (17, 127), (3, 128), (5, 129), (40, 161)])
@pytest.mark.parametrize("kernel,name,alpha", KERNELS, ids=IDS)
def test_matrix_ragged_sizes(kernel, name, alpha, m, n):
    rng = np.random.default_rng(m * 100 + n)
    X, Y = points(rng, m, n)
    X[0] = Y[0]
    e = 0.05 * rng.uniform(0.5, 2.0, n)
    K, ref = fl.assemble(kernel, X, Y, e), oracle_matrix(name, alpha, X, Y, e)
    B, R = (A.reshape(m, 3, n, 3).transpose(0, 2, 1, 3) for A in (K, ref))
    # blocks of a few dozen roundings on each side; the wall's cancel towards z = 0
    err = np.linalg.norm(B - R, axis=(2, 3)) / np.linalg.norm(R, axis=(2, 3))
    assert np.median(err) < 1e-15 and err.max() < 1e-12


@pytest.mark.parametrize("n", [1, 31, 33, 127, 130, 257])
def test_symmetric_matrix_with_leading_dimension(n):
    from fluidlets_gb300.core import _assemble_dev

    rng = np.random.default_rng(n)
    X = torch.tensor(np.c_[rng.uniform(-1, 1, (n, 2)), rng.uniform(0.05, 2.0, n)], device="cuda")
    e = torch.full((n,), 0.06, dtype=torch.float64, device="cuda")
    ld = 3 * n + 5
    for kernel, name, alpha in KERNELS:
        out = torch.full((3 * n, ld), 7.0, dtype=torch.float64, device="cuda")
        _assemble_dev(kernel, X, X, e, 2.0, out=out, ld=ld, sym_eps=0.06, reciprocal=True)
        full = _assemble_dev(kernel, X, X, e, 2.0)
        assert torch.all(out[:, 3 * n:] == 7.0)
        d = (out[:, :3 * n] - full).abs().max().item()
        assert d == 0.0 if name != "wall" else d <= 1e-14 * full.abs().max().item()


def test_matrix_on_and_below_the_wall():
    rng = np.random.default_rng(8)
    X, Y = points(rng, 12, 20)
    X[:4, 2] = 0.0
    X[4:8, 2] *= -1.0
    K, ref = fl.assemble(fl.WallStokeslet3D(), X, Y, 0.05), O.assemble("wall", X, Y, 0.05)
    assert np.all(K[:12] == 0.0)
    assert np.abs(K - ref).max() <= 1e-13 * np.abs(ref).max()


# ---- the mixed sum's plan and near field ------------------------------------------------------------
@pytest.mark.parametrize("n", [1, 5, 255, 257, 1024, 16385, 65536, 65537])
@pytest.mark.parametrize("kernel", [fl.Stokeslet3D(), fl.WallStokeslet3D(), fl.Brinkmanlet3D(2.5),
                                    fl.Brinkmanlet3D(1 + 2j)], ids=["stokeslet", "wall", "alpha2.5", "complex"])
def test_mixed_sum_of_source_counts(kernel, n):
    """Both plans (one launch up to 65,536 sources), ragged tiles; uneven blob widths, a cluster of
    sources in one cell, targets far outside the box."""
    rng = np.random.default_rng(n)
    m = 333
    X, Y = points(rng, m, n)
    X[:40] = Y[rng.integers(0, n, 40)]
    X[40:50] = [50.0, -30.0, 40.0]
    Y[: n // 50] = Y[0] + 1e-3 * rng.normal(size=(n // 50, 3))
    Y[:, 2] = np.abs(Y[:, 2]) + 1e-3
    e = 0.4 * (8.0 / max(n, 8)) ** (1 / 3) * rng.uniform(0.3, 1.0, n)
    F = rng.normal(size=(n, 3)) + (1j * rng.normal(size=(n, 3)) if n % 2 else 0)
    u, ref = fl.evaluate(kernel, X, Y, F, e, precision="mixed"), fl.evaluate(kernel, X, Y, F, e)
    assert np.linalg.norm(u - ref) <= 2e-6 * np.linalg.norm(ref)
    # where every source is near a target the mixed sum is the FP64 one
    if n <= 257:
        big = np.full(n, 60.0)
        u, ref = (fl.evaluate(kernel, X, Y, F, big, precision=p) for p in ("mixed", "fp64"))
        assert np.linalg.norm(u - ref) <= 1e-13 * np.linalg.norm(ref)
