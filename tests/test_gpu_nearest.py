"""Nearest force points with both splits of a query over lanes: the first index on ties, ragged counts."""
import numpy as np
import pytest

pytest.importorskip("torch")

import fluidlets_gb300 as fl  # noqa: E402
import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q", [1, 7, 4863, 4864, 4865, 10001])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 31, 33, 200])
def test_counts_and_ties(q, n):
    rng = np.random.default_rng(q + n)
    X, Y = rng.integers(-3, 4, (q, 3)).astype(float), rng.integers(-3, 4, (n, 3)).astype(float)
    got = fl.nearest_neighbors(X, Y)
    d = ((X[:, None] - Y[None]) ** 2).sum(-1)  # small integers: exact, with many ties
    assert np.array_equal(got, d.argmin(1))
    X, Y = rng.normal(size=(q, 3)), rng.normal(size=(n, 3))
    assert np.array_equal(fl.nearest_neighbors(X, Y), O.nearest_neighbors(X, Y))
