"""Empty matrices are accepted whatever their pointers."""
import pytest

from fluidlets_gb300 import _lib, build


@pytest.mark.parametrize("rows,cols", [(0, 0), (0, 5), (5, 0)])
def test_conversion_of_an_empty_matrix(rows, cols):
    build.build()
    L = _lib.load()
    assert L.flg_convert_f64_f32(rows, cols, None, cols, None, cols, None) == _lib.FLG_OK
    assert L.flg_convert_f64_f32(rows, cols, None, cols - 1, None, cols, None) == _lib.FLG_ERR_INVALID
