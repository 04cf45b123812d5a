"""FP64 planes of few rows, where a CTA's share can span three strips or more.

The estimate behind the split (csrc/fv_stage2d.cu, split_strips) counts each
strip a CTA's rows touch and may give every strip a CTA, more than fit the GPU
at once; whatever it picks, two steps equal the oracle's to
the last bit.
"""
import pytest

from test_gpu_splits import run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,nx,nb", [(k, nx, nb) for k, (nx, nb) in enumerate(
    [(4000, 3), (2500, 2), (9001, 2), (1200, 4), (20000, 3), (701, 5), (15000, 7), (14700, 8)])])
def test_thin_planes(k, nx, nb):
    extra = {"thermal_conduction": {"active": True, "kappa": 0.01}, "viscosity": {"active": True, "mu": 0.01}}
    run_both(nx, nb, 1, 3 * (k // 3), ("pcm", "plm")[k % 2], ("euler", "RK2")[k % 2], ("hll", "hllc")[k // 2 % 2])
    run_both(nx, 1, nb, 1 + k, "plm", "RK2", "hll", extra=extra, physics={"gravity": True, "g": -0.4})
