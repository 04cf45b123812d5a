"""The marched FP32-mixed kernels are as exact as the block forms.

In a stratified layer at near rest every face carries the pressure, and what
is left of it in the flux difference is smaller by orders of magnitude: a flux
rounded once more before the difference, or a diffusive flux added to it,
shows in w at once (1.4 and 1.8 times the block form's error against FP64 were
measured with one and both of these).  The marched forms make the same
roundings per face as the block forms, so the ratio of their errors is about 1
on average; the bound of 1.25 is half-way, in powers, to the smaller of those.
"""
import numpy as np
import pytest

import fv3d_gb300 as fv
from fv3d_gb300 import problems

pytestmark = pytest.mark.gpu

STEPS, SEEDS = 64, 4


def layer2d(seed):
    return problems.rayleigh_taylor(256, 288, kappa=1e-4, mu=1e-4, riemann="hllc", tend=1.0e30, seed=seed)


def layer3d(seed):
    """The same layer in a box, a little noise on every velocity."""
    pr = problems.random_problem(
        "layer3d", problems._mesh(40, 20, 96, xr=(0.0, 0.5), yr=(0.0, 0.25), zr=(0.0, 1.5)),
        {"tend": 1.0e30, "boundaries_x": "periodic", "boundaries_y": "periodic", "boundaries_z": "reflecting"},
        {"riemann_solver": "hllc", "reconstruction": "plm", "time_stepping": "RK2", "CFL": 0.8},
        {"gamma0": 1.4, "gravity": True, "g": "-0.1"}, seed,
        extra={"thermal_conduction": {"active": True, "kappa": "1e-4"}, "viscosity": {"active": True, "mu": "1e-4"}},
        wmag=1.0, vmag=1.0)
    z = ((np.arange(96) + 0.5) * (1.5 / 96)).reshape(96, 1, 1)
    rho = np.where(z > 0.75, 2.0, 1.0) * np.ones_like(pr.prim[0])
    w = 0.01 * (1.0 + np.cos(2 * np.pi * z / 1.5))
    pr.prim = [rho, *(1e-4 * v for v in pr.prim[1:3]), w + 1e-4 * pr.prim[3], 2.5 - 0.1 * rho * (z - 0.75)]
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
    out = b.get_prim(0)
    b.close()
    return out, tx


@pytest.mark.parametrize("make,block,tx,march_tx", [(layer2d, "32x16/8", 32, 28), (layer3d, "16x8", 16, 30)])
def test_no_larger_error_than_the_block_form(make, block, tx, march_tx, monkeypatch):
    logs = []
    for seed in range(SEEDS):
        pr = make(100 + seed)
        want, _ = run(pr, fv._abi.FV_PREC_FP64, None, monkeypatch)
        ref, a = run(pr, fv._abi.FV_PREC_FP32_MIXED, block, monkeypatch)
        got, b = run(pr, fv._abi.FV_PREC_FP32_MIXED, None, monkeypatch)
        assert (a, b) == (tx, march_tx)
        err = [np.linalg.norm(x[3] - want[3]) for x in (ref, got)]
        assert err[0] > 0.0
        logs.append(np.log(err[1] / err[0]))
    assert np.exp(np.mean(logs)) < 1.25, np.exp(logs)
