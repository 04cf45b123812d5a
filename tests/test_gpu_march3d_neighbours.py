"""A mixed 3-D problem beside one that only the block form runs.

Fixed conduction boundaries, the corrected physics and Euler steps without
slopes stay with the block form of the mixed 3-D stage; the other problems of
such a batch keep the z-marched one, and every problem's bits are those it has
alone.
"""
import numpy as np
import pytest

import fv3d_gb300 as fv
from test_gpu_march3d32 import A, P, R, make, run

pytestmark = pytest.mark.gpu


def fixed_temperature(riemann):
    pr = make((20, 12, 9), (P, P, R), riemann, tc=True)
    pr.params.bctc_zmin, pr.params.bctc_zmin_value = fv._abi.FV_BCTC_FIXED_TEMPERATURE, 1.0
    return pr


def corrected(riemann):
    pr = make((20, 12, 9), (P, P, P), riemann, visc=True)
    pr.params.physics = fv._abi.FV_PHYS_CORRECTED
    return pr


def plain(riemann):
    return make((33, 18, 12), (P, R, A), riemann, tc=True, visc=True)


def planar(riemann, plane, visc):
    n, bc = ((40, 30, 1), (P, R, P)) if plane == "xy" else ((40, 1, 30), (P, P, R))
    return make(n, bc, riemann, visc=visc)


@pytest.mark.parametrize("order", [0, 1])
def test_neighbours_do_not_change_a_bit(order, monkeypatch):
    probs = [plain("hllc"), fixed_temperature("hllc"), plain("hllc")]
    if order:
        probs = [probs[1], probs[0], probs[2]]
    (got, times), sched = run(probs, monkeypatch)
    assert sorted(s["tx"] for s in sched) == [16, 30]
    for i, pr in enumerate(probs):
        ((alone,), t), s = run([pr], monkeypatch)
        assert s[0]["tx"] == (16 if pr.params.bctc_zmin else 30)
        assert times[i] == t[0]
        for v in range(5):
            np.testing.assert_array_equal(got[i][v], alone[v], err_msg="%d %d" % (i, v))


def test_every_group_at_once(monkeypatch):
    """All planes, layouts, solvers and forms in one batch: the most groups there can be."""
    probs = [make_one(rs) for rs in ("hll", "hllc") for make_one in (plain, fixed_temperature, corrected)]
    probs += [planar("hllc", plane, visc) for plane in ("xy", "xz") for visc in (False, True)]
    for pr in probs[-4:]:  # no velocity out of the plane without viscosity
        if not pr.params.viscosity_active:
            pr.prim[3 if pr.params.Nz == 1 else 2] = None
    (got, times), sched = run(probs, monkeypatch)
    assert len(sched) == 10
    assert sorted(s["tx"] for s in sched) == [16] * 4 + [28] * 4 + [30] * 2
    for i, pr in enumerate(probs):
        ((alone,), t), _ = run([pr], monkeypatch)
        assert times[i] == t[0]
        for v in range(5):
            np.testing.assert_array_equal(got[i][v], alone[v], err_msg="%d %d" % (i, v))
