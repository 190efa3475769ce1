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
