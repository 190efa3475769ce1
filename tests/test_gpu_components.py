"""FP64 results component by component: what is small beside the other components of its vector, or beside
the distance, keeps its own FP64 precision."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fluidlets_gb300 as fl  # noqa: E402

pytestmark = pytest.mark.gpu

U = 2.0**-53
LD = np.longdouble


def wall_blocks(X, Y, e):
    """The wall kernel's 3 x 3 blocks (pair_math.cuh's header) in extended precision, and the sums of the
    absolute values of their terms."""
    X, Y = X.astype(LD), Y.astype(LD)
    d0, d1 = X[:, None, 0] - Y[None, :, 0], X[:, None, 1] - Y[None, :, 1]
    t, h = X[:, None, 2], Y[None, :, 2]
    dm, dp, e2 = t - h, t + h, LD(e) ** 2
    rq = d0 * d0 + d1 * d1 + e2
    sF, s = 1 / np.sqrt(rq + dm * dm), 1 / np.sqrt(rq + dp * dp)
    Z1 = 2 * sF**2 * s**2 / (sF + s)
    Z3, s5 = Z1 * (sF**2 + sF * s + s**2), 3 * s**5
    G, S = np.zeros(d0.shape + (3, 3), LD), np.zeros(d0.shape + (3, 3), LD)
    for a, da in enumerate((d0, d1)):
        for b, db in enumerate((d0, d1)):
            G[..., a, b], S[..., a, b] = da * db * (Z3 + s5), abs(da * db) * (Z3 + s5)
        G[..., a, a] += Z1 + e2 * Z3 - s**3 + e2 * s5
        S[..., a, a] += Z1 + e2 * Z3 + s**3 + e2 * s5
        G[..., a, 2], G[..., 2, a] = da * (Z3 * dm - s5 * dp), da * (Z3 * dm + s5 * dp)
        S[..., a, 2] = S[..., 2, a] = abs(da) * (Z3 * abs(dm) + s5 * abs(dp))
    G[..., 2, 2] = Z1 + e2 * Z3 - s**3 - e2 * s5 + Z3 * dm**2 - s5 * dp**2
    S[..., 2, 2] = Z1 + e2 * Z3 + s**3 + e2 * s5 + Z3 * dm**2 + s5 * dp**2
    k = (2 * t * h)[..., None, None] / (8 * LD(np.pi))
    return k * G, k * S


@pytest.mark.parametrize("height", [1.0, 1e-3, 1e-6, 1e-9])
def test_wall_matrix_of_low_points(height):
    rng = np.random.default_rng(1)
    X = np.c_[rng.uniform(-1, 1, (40, 2)), height * rng.uniform(0.1, 1.0, 40)]
    Y = np.c_[rng.uniform(-1, 1, (60, 2)), height * rng.uniform(0.1, 1.0, 60)]
    K = fl.assemble(fl.WallStokeslet3D(), X, Y, 0.01)
    B = K.reshape(40, 3, 60, 3).transpose(0, 2, 1, 3)
    G, S = wall_blocks(X, Y, 0.01)
    # a dozen roundings in a coefficient, and those of the displacements, the products and the scale
    assert np.all(abs(B - G) <= 24 * U * S)


# ---- sums -----------------------------------------------------------------------------------------
def radial_blocks(X, Y, e, alpha=None):
    """The blocks A I + B d d^T of a radial kernel in extended precision, and |A| I + |B| |d||d|^T."""
    d = X.astype(LD)[:, None] - Y.astype(LD)[None]
    e2 = np.broadcast_to(np.asarray(e, LD), len(Y))[None] ** 2
    Q = (d * d).sum(-1) + e2
    s = 1 / np.sqrt(Q)
    if alpha is None:
        A, B, k = s + e2 * s**3, s**3, 1 / (8 * LD(np.pi))
    else:
        alpha = np.asarray(alpha, np.clongdouble if isinstance(alpha, complex) else LD)
        z = alpha / s
        E = np.exp(-z)
        f1 = E * (1 + 1 / z + 1 / z**2) - 1 / z**2
        f2 = 3 / z**2 - E * (1 + 3 / z + 3 / z**2)
        A, B, k = s * (f1 + e2 * s**2 * f2), s**3 * f2, 1 / (4 * LD(np.pi))
    dd = d[..., :, None] * d[..., None, :]
    eye = np.eye(3)
    size = abs(A)
    if alpha is not None:  # f1 is a difference
        size = s * (abs(f1) + np.minimum(abs(E * (1 + 1 / z + 1 / z**2)) + abs(1 / z**2), 1) + abs(f2))
    return (k * (A[..., None, None] * eye + B[..., None, None] * dd),
            k * (size[..., None, None] * eye + abs(B)[..., None, None] * abs(dd)))


def check_components(kernel, blocks, X, Y, F, e, precision="fp64"):
    u = fl.evaluate(kernel, X, Y, F, e, precision=precision)
    G, S = blocks
    ref = np.einsum("ijab,jb->ia", G, F.astype(np.clongdouble if np.iscomplexobj(F) else LD))
    size = np.einsum("ijab,jb->ia", S, abs(F.real).astype(LD) + abs(F.imag))
    # thirty roundings in a term, and the sum's (which below 2^-1022 are to multiples of 2^-1074)
    tol = (30 + len(Y)) * (U * size + LD(2.0) ** -1075)
    assert np.all(abs(u.real - ref.real) <= tol)
    if np.iscomplexobj(u):
        assert np.all(abs(u.imag - ref.imag) <= tol)


FREE = [(fl.Stokeslet3D(), None), (fl.Brinkmanlet3D(2.5), 2.5), (fl.Brinkmanlet3D(0.9 + 0.7j), 0.9 + 0.7j)]
FREE_IDS = ["stokeslet", "alpha2.5", "complex"]


@pytest.mark.parametrize("strengths", ["real", "complex"])
@pytest.mark.parametrize("height", [1.0, 1e-3, 1e-6, 1e-9, 1e-12])
@pytest.mark.parametrize("kernel,alpha", FREE, ids=FREE_IDS)
def test_bent_sheet(kernel, alpha, height, strengths):
    rng = np.random.default_rng(2)
    w = np.array([1.0, 1.0, height])
    X, Y = rng.uniform(-1, 1, (50, 3)) * w, rng.uniform(-1, 1, (40, 3)) * w
    F = rng.normal(size=(40, 3)) * w
    if strengths == "complex":
        F = F + 1j * rng.normal(size=(40, 3)) * w
    check_components(kernel, radial_blocks(X, Y, 0.05, alpha), X, Y, F, 0.05)


@pytest.mark.parametrize("height", [1.0, 1e-3, 1e-6, 1e-9])
def test_sheet_on_a_wall(height):
    rng = np.random.default_rng(3)
    X = np.c_[rng.uniform(-1, 1, (50, 2)), height * rng.uniform(0.1, 1.0, 50)]
    Y = np.c_[rng.uniform(-1, 1, (40, 2)), height * rng.uniform(0.1, 1.0, 40)]
    for F in (rng.normal(size=(40, 3)), rng.normal(size=(40, 3)) * [height, height, 1.0]):
        check_components(fl.WallStokeslet3D(), wall_blocks(X, Y, 0.05), X, Y, F, 0.05)


@pytest.mark.parametrize("eps", [1e-3, 1e-6, 1e-9, 1e-12])
@pytest.mark.parametrize("kernel,alpha", FREE, ids=FREE_IDS)
def test_tiny_blobs_push_along_one_axis(kernel, alpha, eps):
    """A target on a source sees a velocity of 1 / eps along that force alone; the other components come
    from the other sources."""
    rng = np.random.default_rng(4)
    Y = rng.uniform(-1, 1, (30, 3))
    e = np.full(30, 0.3)
    e[0] = eps
    F = rng.normal(size=(30, 3))
    F[0] = [1.0, 0.0, 0.0]
    if alpha is None:
        check_components(kernel, radial_blocks(Y, Y, e, alpha), Y, Y, F, e)
    else:  # (the reference's closed form needs |z| above some 1e-3)
        u, v = fl.evaluate(kernel, Y, Y, F, e), fl.evaluate(kernel, Y[:1], Y[1:], F[1:], e[1:])
        assert np.all(abs(u[0, 1:] - v[0, 1:]) <= 60 * U * abs(F).sum() / 0.3)


def test_strengths_of_uneven_components():
    rng = np.random.default_rng(5)
    X, Y = rng.uniform(-1, 1, (20, 3)), rng.uniform(-1, 1, (30, 3))
    X[:, 1] = Y[:, 1] = 0.25  # a plane: u_y comes from f_y alone
    for small in (1e-14, 1e-60, 1e-310):
        F = rng.normal(size=(30, 3)) * [1.0, small, 1.0]
        for kernel, alpha in FREE[:2]:
            check_components(kernel, radial_blocks(X, Y, 0.05, alpha), X, Y, F, 0.05)


@pytest.mark.parametrize("height", [1.0, 1e-6])
def test_near_field_of_a_mixed_sum(height):
    """Every pair near: the mixed sum is the FP64 one."""
    rng = np.random.default_rng(6)
    w = np.array([1.0, 1.0, height])
    X, Y = rng.uniform(-1, 1, (50, 3)) * w, rng.uniform(-1, 1, (40, 3)) * w
    F = rng.normal(size=(40, 3)) * w
    for kernel, alpha in FREE:
        check_components(kernel, radial_blocks(X, Y, 2.0, alpha), X, Y, F, 2.0, precision="mixed")
    X[:, 2], Y[:, 2] = abs(X[:, 2]) + 0.1 * height, abs(Y[:, 2]) + 0.1 * height
    check_components(fl.WallStokeslet3D(), wall_blocks(X, Y, 2.0), X, Y, F, 2.0, precision="mixed")


@pytest.mark.parametrize("scale", [1e-140, 1e-100, 1e-60, 1e60, 1e100, 1e140])
def test_scales_outside_the_fixed_point_ranges(scale):
    """The kernels are homogeneous of degree -1 (alpha L fixed); powers of two scale exactly."""
    c = 2.0 ** round(np.log2(scale))
    rng = np.random.default_rng(7)
    X, Y = rng.uniform(0.1, 1, (20, 3)), rng.uniform(0.1, 1, (30, 3))
    X[:5] = Y[:5]
    F = rng.normal(size=(30, 3))
    for kernel, alpha, scaled in [(fl.Stokeslet3D(), None, fl.Stokeslet3D()),
                                  (fl.Brinkmanlet3D(2.5), 2.5, fl.Brinkmanlet3D(2.5 / c)),
                                  (fl.Brinkmanlet3D(0.9 + 0.7j), 0.9 + 0.7j, fl.Brinkmanlet3D((0.9 + 0.7j) / c))]:
        u = fl.evaluate(scaled, c * X, c * Y, F, c * 0.05) * c
        G, S = radial_blocks(X, Y, 0.05, alpha)
        ref, size = np.einsum("ijab,jb->ia", G, F.astype(LD)), np.einsum("ijab,jb->ia", S, abs(F).astype(LD))
        assert np.all(abs(u - ref) <= 100 * U * size)
    u = fl.evaluate(fl.WallStokeslet3D(), c * X, c * Y, F, c * 0.05) * c
    G, S = wall_blocks(X, Y, 0.05)
    ref, size = np.einsum("ijab,jb->ia", G, F.astype(LD)), np.einsum("ijab,jb->ia", S, abs(F).astype(LD))
    assert np.all(abs(u - ref) <= 100 * U * size)


@pytest.mark.parametrize("strengths", ["real", "complex"])
@pytest.mark.parametrize("order", ["mixed", "sorted", "all below"])
def test_heights_of_both_signs(order, strengths):
    """Targets and sources above and below the wall, alternating within a warp and a tile or in runs."""
    rng = np.random.default_rng(8)
    X, Y = rng.uniform(-1, 1, (300, 3)), rng.uniform(-1, 1, (150, 3))
    if order == "sorted":
        X, Y = X[X[:, 2].argsort()], Y[Y[:, 2].argsort()]
    elif order == "all below":
        X[:, 2], Y[:, 2] = -abs(X[:, 2]), abs(Y[:, 2])
    X[7, 2] = Y[9, 2] = 0.0
    F = rng.normal(size=(150, 3))
    if strengths == "complex":
        F = F + 1j * rng.normal(size=(150, 3))
    u = fl.evaluate(fl.WallStokeslet3D(), X, Y, F, 0.3)
    G, S = wall_blocks(X, Y, 0.3)
    ref = np.einsum("ijab,jb->ia", G, F.astype(np.clongdouble if strengths == "complex" else LD))
    # (the terms of opposite heights do not cancel to the factor 2 t h: each counts by itself)
    size = np.einsum("ijab,jb->ia", abs(S), abs(F.real).astype(LD) + abs(F.imag))
    assert np.all(abs(u - ref) <= (30 + 150) * U * size)
