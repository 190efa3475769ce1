"""Mixed-precision dense solves end a step beyond the tolerance where they ended just below it."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import fluidlets_gb300 as fl  # noqa: E402
from fluidlets_gb300.core import IrGraph, _gmres_ir_dense_dev, _lowp_factor_dev  # noqa: E402
from fluidlets_gb300.geometry import biflagellate_shape  # noqa: E402
from fluidlets_gb300.swimming import _system_dev  # noqa: E402

pytestmark = pytest.mark.gpu


def swimmer(body, segments):
    s = biflagellate_shape(0.3, n_body=body, segments=segments, amplitude=0.08)
    A = _system_dev(fl.Stokeslet3D(), s.x, s.X, fl.nearest_neighbors(s.X, s.x), np.zeros(3), 0.02, 1.0)
    b = torch.zeros(A.shape[0], dtype=torch.float64, device="cuda")
    b[:s.v.size] = torch.from_numpy(np.asarray(s.v).ravel()).cuda()
    return A, b


@pytest.mark.parametrize("lu", ["tf32", "bf16"])
@pytest.mark.parametrize("body,segments", [(49, 81), (96, 64), (197, 73), (264, 112)])
def test_swimmer_residuals(body, segments, lu):
    A, b = swimmer(body, segments)
    K32, ld, dinv, A32 = _lowp_factor_dev(A, lu)
    x, _, _, resid = _gmres_ir_dense_dev(A, K32, ld, dinv, b, 1e-12, 60, 200, A32=A32)
    y = torch.empty_like(b)
    with torch.cuda.stream(torch.cuda.Stream()) as _:
        st = torch.cuda.current_stream()
        st.wait_stream(torch.cuda.default_stream())
        ir = IrGraph(A, A32, K32, ld, dinv, b, y, 1e-12, stream=st)
        ir.launch(st)
        status, _, _, resid_graph = ir.result(st)
        ir.close()
    torch.cuda.synchronize()
    assert status == 0
    for v, r in ((x, resid), (y, resid_graph)):
        # a twentieth of the tolerance, and the rounding of the residual's own 1,500-term sums
        assert r <= 0.05e-12
        assert float((b - A @ v).norm() / b.norm()) <= 0.05e-12 + 1e-14
