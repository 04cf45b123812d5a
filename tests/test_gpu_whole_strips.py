"""Small grids whose strips get a whole number of CTAs each (csrc/fv_stage2d.cu).

Sizes whose strips do not divide the CTAs there is room for, so that the
rounded-down count runs, in both planes and with every physical term; two steps
equal the oracle's to the last bit, as at every split.
"""
import pytest

from test_gpu_splits import run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,nx,nb", [(k, nx, nb) for k, (nx, nb) in enumerate(
    [(80, 64), (96, 64), (100, 100), (128, 64), (160, 160), (13, 41), (40, 300), (64, 192)])])
def test_whole_ctas_per_strip(k, nx, nb):
    solver = ("hllc", "hll")[k % 2]
    extra = {"thermal_conduction": {"active": True, "kappa": 0.01}, "viscosity": {"active": True, "mu": 0.01}}
    run_both(nx, nb, 1, 3 * (k // 3), "plm", "RK2", solver)
    run_both(nx, 1, nb, 1 + 3 * (k // 3) + k % 3, "plm", "RK2", solver, extra=extra,
             physics={"gravity": True, "g": -0.4})
