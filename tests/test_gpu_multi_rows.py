"""The rows per work item of the multi-step launch (mixed 2-D RK2).

Up to 5 rows are taken so that no SM has more than three CTAs of four warps, an
item a warp; longer items use every resident warp.
"""
import os
import re
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CODE = """
import sys
sys.path.insert(0, %r)
import fv3d_gb300 as fv
from fv3d_gb300 import problems
pr = problems.random_problem("m", problems._mesh(%d, %d, 1), {"tend": 1.0e30},
                             {"riemann_solver": "hllc", "reconstruction": "pcm", "time_stepping": "RK2"},
                             {"gamma0": 1.4}, 1)
pr.prim[3] = None
params = pr.params.copy()
params.precision = fv._abi.FV_PREC_FP32_MIXED
b = fv.Batch([params] * %d)
for i in range(%d):
    b.set_prim(i, *pr.prim)
b.run(2)
b.close()
"""


@pytest.mark.parametrize("nx,ny,n", [(30, 1000, 1), (28, 1824, 1), (32, 32, 100), (420, 400, 1), (64, 64, 1)])
def test_short_items_leave_the_fourth_cta(nx, ny, n):
    rows, items, ctas, sms = chosen(nx, ny, n)
    strips = -(-nx // 28) * n
    assert 1 <= rows <= 5 and ctas <= 3 * sms and items == strips * -(-ny // rows)
    assert rows == 1 or strips * -(-ny // (rows - 1)) > 12 * sms  # the fewest


@pytest.mark.parametrize("nx,ny", [(512, 512), (1024, 1024), (28, 30000)])
def test_long_items_take_every_warp(nx, ny):
    rows, items, ctas, sms = chosen(nx, ny, 1)
    assert ctas > 3 * sms and items <= 4 * ctas and -(-nx // 28) * -(-ny // 5) > 12 * sms


def chosen(nx, ny, n):
    import torch
    env = dict(os.environ, FV3D_TILE_LOG="1", FV3D_TILE="28x16")
    for k in ("FV3D_MULTI_ROWS", "FV3D_MULTISTEP"):
        env.pop(k, None)
    r = subprocess.run([sys.executable, "-c", CODE % (ROOT, nx, ny, n, n)], env=env, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    (m,) = re.findall(r"multi-step: (\d+) rows \((\d+) items, (\d+) CTAs\)", r.stderr)
    return (*map(int, m), torch.cuda.get_device_properties(0).multi_processor_count)
