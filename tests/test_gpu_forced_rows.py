"""FV3D_TILE=28xH forces the rows per work item of the mixed 2-D form, with or without its 0 block rows."""
import pytest

import fv3d_gb300 as fv
from fv3d_gb300 import problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile,rows", [("28x5", 5), ("28x16", 16), ("28x7/0", 7)])
def test_forced_rows_are_taken(tile, rows, monkeypatch):
    monkeypatch.setenv("FV3D_TILE", tile)
    pr = problems.sedov(64)
    params = pr.params.copy()
    params.precision = fv._abi.FV_PREC_FP32_MIXED
    b = fv.Batch([params])
    b.set_prim(0, *pr.prim)
    assert b.schedule() == [{"tx": 28, "rows": rows, "block_rows": 0, "split_viscous": 0}]
    b.close()
