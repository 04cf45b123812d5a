"""Work items of the marched mixed 2-D stages by warp number and from the queue.

Where the GPU holds a warp for every item each takes the one of its number,
else the warps pull from the queue counter; which it is must not change a bit.
"""
import numpy as np
import pytest

import fv3d_gb300 as fv
from fv3d_gb300 import problems

pytestmark = pytest.mark.gpu


def run(n, stepping, rows, copies, monkeypatch):
    monkeypatch.setenv("FV3D_TILE", "28x%d" % rows)
    monkeypatch.setenv("FV3D_MULTISTEP", "0")
    pr = problems.random_problem("q", problems._mesh(*n, 1), {"tend": 1.0e30, "boundaries_x": "periodic",
                                                              "boundaries_y": "reflecting"},
                                 {"riemann_solver": "hllc", "reconstruction": "plm", "time_stepping": stepping,
                                  "CFL": 0.4}, {"gamma0": 1.4}, 5, vmag=0.5)
    params = pr.params.copy()
    params.precision = fv._abi.FV_PREC_FP32_MIXED
    b = fv.Batch([params] * copies)
    for i in range(copies):
        b.set_prim(i, *pr.prim)
    b.run(5)
    out = [b.get_prim(i) for i in range(copies)], b.times()
    b.close()
    return out


@pytest.mark.parametrize("stepping", ["euler", "RK2"])
@pytest.mark.parametrize("n,copies", [((140, 900), 1), ((57, 301), 4), ((28, 2432), 1), ((28, 2433), 1)])
def test_same_bits(n, copies, stepping, monkeypatch):
    """One row an item (4,500 and 3,612: queued; about as many as resident warps) against few items."""
    ref, t = run(n, stepping, 64, copies, monkeypatch)
    assert np.isfinite(ref[0]).all()
    got, tg = run(n, stepping, 1, copies, monkeypatch)
    assert list(t) == list(tg)
    for i in range(copies):
        for v in range(5):
            np.testing.assert_array_equal(got[i][v], ref[i][v])
