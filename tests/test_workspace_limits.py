"""A workspace that is too small is refused on the host whatever part of it does not fit (no CUDA call is
reached: the pointers here are not device memory)."""
import ctypes

import pytest

from fluidlets_gb300 import _lib, build

P = ctypes.c_void_p(1 << 20)


@pytest.fixture(scope="module")
def L():
    build.build()
    return _lib.load()


def sizes(need):
    """Every size below need by at least the alignment slack, in a few thousand steps, and the smallest ones."""
    step = max(256, need // 3000)
    return [*range(0, min(need - 256, 4096), 64), *range(0, need - 256, step), need - 257]


@pytest.mark.parametrize("m,n,cplx,precision", [(64, 70000, 0, 1), (64, 70000, 1, 1), (40000, 1000, 0, 1), (300, 500, 1, 1),
                                                (300, 500, 1, 0)])
def test_sums(L, m, n, cplx, precision):
    need = L.flg_evaluate_workspace(0, m, n, cplx, 0.0, precision)
    for nb in sizes(need):
        st = L.flg_evaluate(0, 0.0, 0.0, P, m, P, P, n, P, cplx, 1.0, 0.0, P, precision, P, nb, None)
        assert st == _lib.FLG_ERR_INVALID, (nb, need)


@pytest.mark.parametrize("n", [65, 300])
def test_fp64_lu(L, n):
    info = ctypes.c_int(0)
    need = L.flg_lu_factor_f64_workspace(n)
    for nb in sizes(need):
        assert L.flg_lu_factor_f64(n, P, n, P, ctypes.byref(info), P, nb, None) == _lib.FLG_ERR_INVALID, (nb, need)
