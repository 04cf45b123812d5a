"""The FP32-mixed HLLC solver over the range of its quotients.

Densities whose product leaves FP32 (above 9e18) and pressures whose product
with the density does (below 1.2e-38) are within the range of p / rho, on which
the sound speed of a face depends.  Dense states are held to the FP64 form by
the mixed form's bounds (assert_mixed).  Of the thin ones FP32 cannot form
the star pressure in any form of the solver, so there the run has to go on to
a finite state, as the block forms' does.
"""
import numpy as np
import pytest

import fv3d_gb300 as fv
from fv3d_gb300 import problems
from _helpers import assert_mixed

pytestmark = pytest.mark.gpu

STEPS = 4
SHAPES = {"2d": (45, 37, 1), "3d": (33, 18, 9)}
BLOCK = {"2d": "32x16/8", "3d": "16x8"}


def state(shape, rho, p, seed=3):
    """Nearly at rest: densities within 30 %, pressures within 1e-3, velocities of 1e-3 sound speeds."""
    bc = {"tend": 1.0e30, "boundaries_x": "periodic", "boundaries_y": "reflecting", "boundaries_z": "periodic"}
    pr = problems.random_problem("range", problems._mesh(*SHAPES[shape]), bc,
                                 {"riemann_solver": "hllc", "reconstruction": "plm", "time_stepping": "RK2",
                                  "CFL": 0.4}, {"gamma0": 1.4}, seed)
    rng = np.random.default_rng(seed)
    dims = pr.prim[0].shape
    c = np.sqrt(1.4 * p / rho)
    vel = [1e-3 * c * rng.uniform(-1.0, 1.0, dims) for _ in range(3)]
    if shape == "2d":
        vel[2] = None
    pr.prim = [rho * rng.uniform(1.0, 1.3, dims), *vel, p * rng.uniform(1.0, 1.001, dims)]
    return pr


def run(pr, precision, tile, monkeypatch):
    if tile:
        monkeypatch.setenv("FV3D_TILE", tile)
    else:
        monkeypatch.delenv("FV3D_TILE", raising=False)
    params = pr.params.copy()
    params.precision = precision
    b = fv.Batch([params])
    b.set_prim(0, *pr.prim)
    tx = b.schedule()[0]["tx"]
    b.run(STEPS)
    out, t = b.get_prim(0), b.times()[0]
    b.close()
    return out, t, tx


@pytest.mark.parametrize("shape", ["2d", "3d"])
@pytest.mark.parametrize("rho,p", [(1.0e19, 1.0), (1.0e19, 1.0e8), (3.0e24, 1.0e3)])
def test_dense_states(shape, rho, p, monkeypatch):
    pr = state(shape, rho, p)
    want, t, _ = run(pr, fv._abi.FV_PREC_FP64, None, monkeypatch)
    for tile in (None, BLOCK[shape]):
        got, tm, tx = run(pr, fv._abi.FV_PREC_FP32_MIXED, tile, monkeypatch)
        assert tx == {"2d": 28, "3d": 30}[shape] if tile is None else tx in (32, 16)
        assert abs(tm - t) <= 1e-5 * t
        # in units of the state's own scales, as the bounds on velocities are relative to the signal speed
        assert_mixed(got, want, pr.params.gamma0, (shape, rho, p, tile))


@pytest.mark.parametrize("shape", ["2d", "3d"])
@pytest.mark.parametrize("rho,p", [(4.0e-6, 1.0e-33), (1.0e-3, 1.0e-36)])
def test_thin_states_go_on(shape, rho, p, monkeypatch):
    pr = state(shape, rho, p)
    for tile in (None, BLOCK[shape]):
        got, t, _ = run(pr, fv._abi.FV_PREC_FP32_MIXED, tile, monkeypatch)
        assert t > 0.0
        for v in range(5):
            assert np.isfinite(got[v]).all(), (tile, v)
