"""How the FP64 stage kernels split a grid over the GPU does not show.

The 2-D kernel takes strips of any width up to 32 columns and any run of rows
per CTA, the 3-D kernel blocks of any size up to 16 x 16 columns and any run of
layers, both chosen from the grid's size.  Sizes around those of a strip, a
block and a warp, one-cell-thin remainders and grids smaller than a block
advance two steps and must equal the oracle's to the last bit, with every
reconstruction (PCM reads one cell around a cell, PLM two).
"""
import numpy as np
import pytest

import fv3d_gb300 as fv
from fv3d_gb300 import problems
from oracle import pyoracle

pytestmark = pytest.mark.gpu

BCS = ("absorbing", "reflecting", "periodic")


def run_both(nx, ny, nz, k, recon, stepping, solver, extra=None, physics=None):
    bc = [BCS[(k + a) % 3] for a in range(3)]
    if nz == 1:
        bc[2] = "periodic"
    if ny == 1:
        bc[1] = "periodic"
    run = {"tend": 1.0, **{"boundaries_%s" % a: b for a, b in zip("xyz", bc)}}
    pr = problems.random_problem("split", problems._mesh(nx, ny, nz), run,
                                 {"riemann_solver": solver, "reconstruction": recon, "time_stepping": stepping,
                                  "CFL": 0.3}, dict({"gamma0": 1.4}, **(physics or {})), seed=900 + k, extra=extra,
                                 wmag=0.5 if min(nx, ny, nz) > 1 else 0.0, vmag=0.8)
    sim, ora = fv.Simulation(pr.params), pyoracle.Oracle(pr.params)
    sim.set_prim(*pr.prim)
    ora.set_prim(*pr.prim)
    for _ in range(2):
        dt, want = sim.compute_dt(), ora.compute_dt()
        assert dt == want
        sim.step(dt)
        ora.step(dt)
    for v, (a, b) in enumerate(zip(sim.get_prim(), ora.get_prim())):
        np.testing.assert_array_equal(a, b, err_msg="%dx%dx%d field %d" % (nx, ny, nz, v))
    sim.close()


@pytest.mark.parametrize("k,nx,nb", [(k, nx, nb) for k, (nx, nb) in enumerate(
    [(2, 2), (8, 3), (9, 40), (16, 17), (31, 64), (33, 1), (33, 5), (48, 48), (65, 130), (112, 112), (255, 9),
     (256, 33), (257, 70), (320, 300)]) if nb > 1])
def test_plane_strips(k, nx, nb):
    recon, stepping, solver = ("plm", "pcm", "plm")[k % 3], ("RK2", "euler")[k % 2], ("hllc", "hll")[k // 2 % 2]
    extra = {"thermal_conduction": {"active": True, "kappa": 0.01}, "viscosity": {"active": True, "mu": 0.01}}
    run_both(nx, nb, 1, 3 * (k // 3), recon, stepping, solver)
    run_both(nx, 1, nb, 1 + 3 * (k // 3) + k % 3, recon, stepping, solver,
             extra=extra if k % 2 else None, physics={"gravity": True, "g": -0.4})


@pytest.mark.parametrize("k,n", list(enumerate([(2, 2, 2), (3, 17, 5), (16, 16, 9), (17, 33, 4), (15, 8, 40), (40, 9, 7),
                                           (31, 24, 12), (33, 50, 3), (64, 20, 11), (5, 70, 30)])))
def test_block_columns(k, n):
    recon, stepping, solver = ("plm", "pcm", "pcm_wb")[k % 3], ("RK2", "euler")[k % 2], ("hllc", "hll")[k // 2 % 2]
    extra = {"thermal_conduction": {"active": True, "kappa": 0.01}, "viscosity": {"active": True, "mu": 0.01}}
    run_both(*n, k, recon, stepping, solver, extra=extra if k % 2 else None)
