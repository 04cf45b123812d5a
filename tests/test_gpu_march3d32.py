"""The z-marched FP32-mixed 3-D kernel (csrc/fv_march3d32.cu).

A CTA owns up to 30 x 15 columns (lanes 1..30 of 15 warps; the rest serve
their neighbours) and a run of layers, so the places to go wrong are sizes
around those, halo cells of every boundary kind, very few layers and runs that
start or end anywhere.  Each case runs a few steps and is held to the mixed
form's bounds against the FP64 form (assert_mixed); the runs of layers and the
group a problem sits in must not change a bit.
"""
import numpy as np
import pytest

import fv3d_gb300 as fv
from fv3d_gb300 import problems
from _helpers import assert_mixed

pytestmark = pytest.mark.gpu

STEPS = 4


def make(n, bc, riemann, recon="plm", stepping="RK2", gravity=False, tc=False, visc=False, seed=11):
    run = {"tend": 1.0e30, **{"boundaries_%s" % a: b for a, b in zip("xyz", bc)}}
    physics = {"gamma0": 1.4}
    if gravity:
        physics.update(gravity=True, g=-0.3)
    extra = {}
    if tc:
        extra["thermal_conduction"] = {"active": True, "kappa": 1e-3}
    if visc:
        extra["viscosity"] = {"active": True, "mu": 1e-3}
    return problems.random_problem("march3", problems._mesh(*n), run,
                                   {"riemann_solver": riemann, "reconstruction": recon, "time_stepping": stepping,
                                    "CFL": 0.4}, physics, seed, extra=extra, wmag=0.6, vmag=0.7)


P, R, A = "periodic", "reflecting", "absorbing"
CASES = [
    lambda: make((30, 15, 5), (P, P, P), "hllc"),
    lambda: make((31, 16, 3), (R, A, P), "hll", tc=True, visc=True),
    lambda: make((29, 14, 33), (A, R, R), "hllc", tc=True, visc=True),
    lambda: make((61, 31, 4), (P, R, A), "hllc", visc=True),
    lambda: make((2, 40, 9), (P, P, R), "hll", gravity=True, tc=True),
    lambda: make((45, 2, 20), (R, P, A), "hllc", stepping="euler"),
    lambda: make((24, 17, 2), (A, A, P), "hll", recon="pcm"),
    lambda: make((33, 46, 7), (P, A, R), "hllc", recon="pcm_wb", gravity=True),
    lambda: make((62, 13, 12), (R, R, P), "hll", stepping="euler", recon="pcm", visc=True),
    lambda: make((40, 33, 1), (P, R, P), "hllc", gravity=True, tc=True),
]


def run(probs, monkeypatch, tile=None):
    if tile:
        monkeypatch.setenv("FV3D_TILE", tile)
    else:
        monkeypatch.delenv("FV3D_TILE", raising=False)
    params = []
    for pr in probs:
        params.append(pr.params.copy())
        params[-1].precision = fv._abi.FV_PREC_FP32_MIXED
    b = fv.Batch(params)
    for i, pr in enumerate(probs):
        b.set_prim(i, *pr.prim)
    sched = b.schedule()
    b.run(STEPS)
    out = [b.get_prim(i) for i in range(len(probs))], b.times()
    b.close()
    return out, sched


@pytest.mark.parametrize("k", range(len(CASES)))
def test_marched_against_fp64(k, monkeypatch):
    pr = CASES[k]()
    s = fv.Simulation(pr.params)
    s.set_prim(*pr.prim)
    t, _ = s.advance(1.0e30, max_steps=STEPS)
    want = s.get_prim()
    s.close()
    ((got,), tm), sched = run([pr], monkeypatch)
    assert sched[0]["tx"] == 30 and sched[0]["block_rows"] == 15
    assert_mixed(got, want, pr.params.gamma0, k)
    assert abs(tm[0] - t) <= 1e-5 * t


@pytest.mark.parametrize("k", range(len(CASES)))
def test_layers_and_group_do_not_change_a_bit(k, monkeypatch):
    pr = CASES[k]()
    ((ref,), t), _ = run([pr], monkeypatch, tile="30x64")
    for probs, tile in (([pr], "30x1"), ([pr], "30x3"), ([pr, pr], "30x5")):
        (got, tg), sched = run(probs, monkeypatch, tile=tile)
        assert sched[0]["tx"] == 30
        for i in range(len(probs)):
            assert tg[i] == t[0]
            for v in range(5):
                np.testing.assert_array_equal(got[i][v], ref[v], err_msg="%s %d" % (tile, v))


def test_what_it_does_not_run_takes_the_block_form(monkeypatch):
    """Fixed conduction boundaries, the corrected physics, and Euler steps without slopes or diffusion."""
    bctc = make((20, 12, 9), (P, P, R), "hllc", tc=True)
    bctc.params.bctc_zmin, bctc.params.bctc_zmin_value = fv._abi.FV_BCTC_FIXED_TEMPERATURE, 1.0
    corrected = make((20, 12, 9), (P, P, P), "hllc", visc=True)
    corrected.params.physics = fv._abi.FV_PHYS_CORRECTED
    euler = make((20, 12, 9), (P, P, P), "hllc", recon="pcm", stepping="euler")
    for pr in (bctc, corrected, euler):
        assert run([pr], monkeypatch)[1][0]["tx"] == 16
    # a group takes the form all of its members have
    other = make((20, 12, 9), (P, P, R), "hllc", tc=True)
    assert run([bctc, other], monkeypatch)[1][0]["tx"] == 16
