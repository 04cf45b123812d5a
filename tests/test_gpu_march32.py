"""The warp-marched FP32-mixed 2-D kernels (csrc/fv_march32.cuh).

A warp owns a strip of 28 columns (lanes 2..29; ghosts on either side) and a
run of rows, so the places to go wrong are widths around multiples of 28,
very few rows, ghost columns and rows of every boundary kind, and runs of
rows that start or end anywhere.  Each case runs a few steps and is held to
the mixed form's bounds against the FP64 form (assert_mixed); the split into
runs of rows and the group a problem sits in must not change a bit.
"""
import numpy as np
import pytest

import fv3d_gb300 as fv
from fv3d_gb300 import problems
from _helpers import assert_mixed

pytestmark = pytest.mark.gpu

STEPS = 4


def make(plane, nx, nb, bc, riemann, recon="plm", stepping="RK2", gravity=False, tc=False, visc=False, wmag=0.0, seed=5):
    mesh = problems._mesh(nx, nb, 1) if plane == "xy" else problems._mesh(nx, 1, nb)
    run = {"tend": 1.0e30, "boundaries_x": bc[0], "boundaries_y": bc[1] if plane == "xy" else "periodic",
           "boundaries_z": "periodic" if plane == "xy" else bc[1]}
    physics = {"gamma0": 1.4}
    if gravity:
        physics.update(gravity=True, g=-0.3)
    extra = {}
    if tc:
        extra["thermal_conduction"] = {"active": True, "kappa": 1e-3}
    if visc:
        extra["viscosity"] = {"active": True, "mu": 1e-3}
    pr = problems.random_problem("march", mesh, run, {"riemann_solver": riemann, "reconstruction": recon,
                                                     "time_stepping": stepping, "CFL": 0.4}, physics, seed,
                                 extra=extra, vmag=0.7)
    w = 0.3 * problems.uniform(seed, 9, nx * nb).reshape(pr.shape) if wmag else None
    out = 3 if plane == "xy" else 2  # the velocity out of the plane
    pr.prim[out] = np.zeros(pr.shape) if w is None else w
    if plane == "xz":
        pr.prim[3] = 0.7 * (2 * problems.uniform(seed, 8, nx * nb).reshape(pr.shape) - 1)
    return pr


CASES = [
    lambda: make("xy", 28, 2, ("periodic", "periodic"), "hllc"),
    lambda: make("xy", 27, 3, ("reflecting", "absorbing"), "hll"),
    lambda: make("xy", 29, 5, ("absorbing", "reflecting"), "hllc", tc=True, visc=True),
    lambda: make("xy", 57, 31, ("periodic", "reflecting"), "hll", tc=True, visc=True, wmag=1),
    lambda: make("xy", 2, 40, ("periodic", "periodic"), "hllc", recon="pcm"),
    lambda: make("xy", 113, 17, ("reflecting", "periodic"), "hllc", stepping="euler"),
    lambda: make("xy", 84, 9, ("absorbing", "absorbing"), "hllc", wmag=1),
    lambda: make("xz", 28, 30, ("periodic", "reflecting"), "hll", gravity=True),
    lambda: make("xz", 55, 2, ("reflecting", "reflecting"), "hllc", gravity=True, tc=True, visc=True),
    lambda: make("xz", 31, 33, ("absorbing", "periodic"), "hll", tc=True, visc=True, wmag=1),
    lambda: make("xz", 40, 21, ("periodic", "absorbing"), "hllc", recon="pcm_wb", gravity=True),
    lambda: make("xz", 86, 13, ("periodic", "periodic"), "hll", stepping="euler", gravity=True, tc=True),
]


def run(probs, monkeypatch, tile=None, multi="0"):
    monkeypatch.setenv("FV3D_MULTISTEP", multi)
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
    b.run(STEPS)
    out = [b.get_prim(i) for i in range(len(probs))], b.times()
    b.close()
    return out


@pytest.mark.parametrize("k", range(len(CASES)))
def test_marched_against_fp64(k, monkeypatch):
    pr = CASES[k]()
    s = fv.Simulation(pr.params)
    s.set_prim(*pr.prim)
    t, _ = s.advance(1.0e30, max_steps=STEPS)
    want = s.get_prim()
    s.close()
    (got,), tm = run([pr], monkeypatch)
    assert_mixed(got, want, pr.params.gamma0, k)
    assert abs(tm[0] - t) <= 1e-5 * t


@pytest.mark.parametrize("k", range(len(CASES)))
def test_rows_and_group_do_not_change_a_bit(k, monkeypatch):
    """Runs of 1, 3 or all rows, several steps per launch, and a neighbour in
    the group (descriptors in shared memory instead of the launch parameters)."""
    pr = CASES[k]()
    (ref,), t = run([pr], monkeypatch, tile="28x64/0")
    for probs, tile, multi in (([pr], "28x1/0", "0"), ([pr], "28x3/0", "0"), ([pr], "28x7/0", "1"),
                               ([pr, pr], "28x5/0", "0"), ([pr, pr], "28x2/0", "1")):
        got, tg = run(probs, monkeypatch, tile=tile, multi=multi)
        for i in range(len(probs)):
            assert tg[i] == t[0]
            for v in range(5):
                np.testing.assert_array_equal(got[i][v], ref[v], err_msg="%s %s %d" % (tile, multi, v))
