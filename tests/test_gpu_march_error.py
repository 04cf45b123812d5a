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


@pytest.mark.parametrize("make,block,tx,march_tx", [(layer2d, "32x16/8", 32, 28)])
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
