"""Low-precision LU at the edges of its diagonal blocks, panels and inverses (lu.cu): sizes around the
128-row blocks and the panels' 32-row groups, few systems (a lane per panel column) and many (two
columns per lane)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from fluidlets_gb300 import _device as dv  # noqa: E402
from fluidlets_gb300 import _lib  # noqa: E402


def _factor_single(L, LU, n, ld, m):
    dinv = torch.full((L.flg_lu_lowp_dinv_elems(n),), float("nan"), dtype=torch.float32, device="cuda")
    flags = torch.full((2,), -1, dtype=torch.int32, device="cuda")
    nb = L.flg_lu_factor_lowp_workspace(n, m)
    ws = dv.workspace(nb)
    _lib.check(L.flg_lu_factor_lowp_async(n, dv.ptr(LU), ld, m, dv.ptr(dinv), dv.ptr(flags), dv.ptr(ws), nb,
                                          dv.stream()), "LU")
    assert torch.all(flags == 0)
    return LU, dinv


@pytest.mark.parametrize("mode", ["fp32", "tf32"])
@pytest.mark.parametrize("n,nbat", [(1, 1), (33, 2), (127, 1), (129, 3), (160, 40), (257, 2), (290, 64), (415, 40)])
def test_lowp_lu_edges(n, nbat, mode):
    """|A - L U| within n u |L||U| (u = 2^-24, all sums in FP32) and, for tf32, the rounding of both
    operands of each rank-128 product (2 x 2^-11 |L||U| of the off-diagonal blocks); the inverses
    within 256 u of each 128-row block, times its condition number (below 8: the diagonal is 4 and
    the rest's norm about 2); every system the same bits as its first run alone."""
    L = _lib.load()
    ld = (n + 31) // 32 * 32
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.zeros((nbat, n, ld), dtype=torch.float32, device="cuda")
    A[:, :, :n] = torch.randn((nbat, n, n), generator=g, device="cuda") / n ** 0.5 + 4.0 * torch.eye(n, device="cuda")
    m = _lib.lu_mode(mode)

    def factor(src, k):
        LU = src.clone()
        dinv = torch.full((k, L.flg_lu_lowp_dinv_elems(n)), float("nan"), dtype=torch.float32, device="cuda")
        flags = torch.full((k, 2), -1, dtype=torch.int32, device="cuda")
        nb = L.flg_lu_factor_lowp_batched_workspace(n, k, m)
        ws = dv.workspace(nb)
        _lib.check(L.flg_lu_factor_lowp_batched_async(n, k, dv.ptr(LU), ld, n * ld, m, dv.ptr(dinv), dv.ptr(flags),
                                                      dv.ptr(ws), nb, dv.stream()), "LU")
        assert torch.all(flags == 0)
        return LU, dinv

    if mode == "fp32":  # the batched entry takes tensor-core modes only
        def factor(src, k):
            out = [_factor_single(L, LU, n, ld, m) for LU in src.clone()]
            return torch.stack([o[0] for o in out]), torch.stack([o[1] for o in out])

    LU, dinv = factor(A, nbat)
    one, done = factor(A[-1:], 1)
    assert torch.equal(one[0], LU[-1]) and torch.equal(done[0], dinv[-1])

    F = LU[:, :, :n].double()
    Lo = torch.tril(F, -1) + torch.eye(n, device="cuda", dtype=torch.float64)
    Up = torch.triu(F)
    blk = torch.arange(n, device="cuda") // 128
    off = torch.minimum(blk[:, None], blk[None, :]) > 0  # entries that a rank-128 product has changed
    bound = n * 2.0 ** -24 * (Lo.abs() @ Up.abs()) + 1e-30
    if mode == "tf32":
        bound = bound + off * 2.0 ** -10 * (Lo.abs() @ Up.abs())
    res = (A[:, :, :n].double() - Lo @ Up).abs()
    assert bool(torch.all(res <= bound)), float((res / bound).max())

    nblk = (n + 127) // 128
    D = dinv.double().reshape(nbat, 2, nblk, 128, 128)
    for k in range(nblk):
        r0, r1 = 128 * k, min(n, 128 * k + 128)
        w = r1 - r0
        for h, T in ((0, Lo), (1, Up)):
            I = torch.eye(128, device="cuda", dtype=torch.float64).repeat(nbat, 1, 1)
            I[:, :w, :w] = T[:, r0:r1, r0:r1]
            err = (D[:, h, k] @ I - torch.eye(128, device="cuda", dtype=torch.float64)).abs().max()
            assert float(err) <= 8 * 256 * 2.0 ** -24, (k, h, float(err))
    assert not np.isnan(dinv.cpu().numpy()).any()


@pytest.mark.parametrize("nr,nc,lds,ldd,off", [(1, 1, 1, 1, 0), (3, 7, 9, 8, 0), (5, 4096, 4096, 4096, 0), (2, 4099, 4100, 4128, 0),
                                               (7, 33, 34, 36, 1), (70000, 5, 6, 8, 0)])
def test_fp32_copies_are_rounded_as_the_conversion(nr, nc, lds, ldd, off):
    """Whole bits: ties, denormals, overflow, infinities and NaN, aligned rows and others."""
    L = _lib.load()
    rng = np.random.default_rng(nc)
    x = rng.normal(size=nr * lds + off) * 10.0 ** rng.integers(-50, 50, nr * lds + off)
    x[::5] = np.ldexp(2.0 * rng.integers(2 ** 23, 2 ** 24, x[::5].size) + 1.0, rng.integers(-160, 110, x[::5].size))  # ties
    x[::11] = np.resize([0.0, -0.0, np.inf, -np.inf, np.nan, 3.4028235677973366e38, 1.1754943e-38, 1e-45, 7e-46, 5e-324],
                        x[::11].size)
    src = torch.from_numpy(x).cuda()[off:].reshape(nr, lds)
    a, b = (torch.full((nr, ldd), 7.0, dtype=torch.float32, device="cuda") for _ in range(2))
    _lib.check(L.flg_convert_f64_f32x2(nr, nc, dv.ptr(src), lds, dv.ptr(a), dv.ptr(b), ldd, dv.stream()))
    ref = src[:, :nc].cpu().float()
    for d in (a, b):
        assert torch.equal(torch.isnan(d[:, :nc].cpu()), torch.isnan(ref)) and torch.all(d[:, nc:] == 7.0)
        assert torch.equal(torch.nan_to_num(d[:, :nc].cpu(), nan=1.0).view(torch.int32),
                           torch.nan_to_num(ref, nan=1.0).view(torch.int32))
