"""The rows per work item that the tuner of the marched mixed 2-D form tries.

An item's first two rows only fill registers, so on small grids items of a few
rows that leave some warps of the GPU idle are faster than the shortest ones
that give every warp one; the tuner has to have such rows among its choices.
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
pr = problems.random_problem("c", problems._mesh(%d, %d, 1), {"tend": 1.0},
                             {"riemann_solver": "hllc", "reconstruction": "pcm", "time_stepping": "%s"},
                             {"gamma0": 1.4}, 1)
pr.prim[3] = None
params = pr.params.copy()
params.precision = fv._abi.FV_PREC_FP32_MIXED
b = fv.Batch([params])
b.set_prim(0, *pr.prim)
print(b.schedule()[0]["rows"])
b.close()
"""


@pytest.mark.parametrize("nx,ny,stepping,wanted", [(256, 256, "euler", {1, 2, 3}), (700, 500, "euler", {3, 5, 8}),
                                                   (700, 500, "RK2", {8})])
def test_rows_tried(nx, ny, stepping, wanted, tmp_path):
    env = dict(os.environ, FV3D_TILE_LOG="1", FV3D_TILE_CACHE=str(tmp_path / "tiles.txt"))
    env.pop("FV3D_TILE", None)
    r = subprocess.run([sys.executable, "-c", CODE % (ROOT, nx, ny, stepping)], env=env, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    tried = {int(m) for m in re.findall(r"candidate 28x(\d+)/0", r.stderr)}
    assert wanted <= tried, tried
    assert int(r.stdout) in tried
