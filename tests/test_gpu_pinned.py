"""States set from and read into pinned host arrays.

Arrays in pinned memory are read and written by the conversion kernels in
place, pageable ones are copied and converted on the GPU: both must give the
same bits, in both precisions, for a handle and in a batch, with and without a
velocity out of the plane and with fields left out.
"""
import ctypes

import numpy as np
import pytest

import fv3d_gb300 as fv
from fv3d_gb300 import problems

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def pinned(a):
    if a is None:
        return None
    h = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    h.copy_(torch.from_numpy(np.ascontiguousarray(a)))
    return h.numpy()


RUN = {"tend": 1.0, "boundaries_x": "periodic", "boundaries_y": "absorbing", "boundaries_z": "periodic"}


def cases():
    xy = problems.random_problem("p", problems._mesh(37, 23, 1), RUN, {"riemann_solver": "hllc"},
                                 {"gamma0": 1.4}, 3)
    xy.prim[3] = None
    w = problems.random_problem("w", problems._mesh(64, 48, 1), RUN, {"time_stepping": "RK2"},
                                {"gamma0": 1.3}, 4, wmag=0.4)
    xz = problems.rayleigh_taylor(40, 120)
    d3 = problems.random_problem("d", problems._mesh(19, 14, 9), RUN, {"time_stepping": "RK2"},
                                 {"gamma0": 1.6}, 5, wmag=0.6)
    rest = problems.sedov(33)
    rest.prim[1:4] = [None, None, None]
    return [xy, w, xz, d3, rest]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("k", range(5))
def test_pinned_equals_pageable(k, precision):
    pr = cases()[k]
    params = pr.params.copy()
    params.precision = precision
    out = []
    for place in (lambda a: a, pinned):
        prim = [place(a) for a in pr.prim]
        sim = fv.Simulation(params)
        # another state first, with a velocity out of the plane: nothing of it may stay
        other = [np.full(pr.shape, x) for x in (1.0, 0.1, 0.2, 0.3, 2.0)]
        sim.set_prim(*[place(a) for a in other])
        sim.set_prim(*prim)
        start = [place(np.full(pr.shape, -1.0)) for _ in range(5)]
        sim.get_prim(start)
        dt = sim.compute_dt()
        sim.advance(1.0e30, max_steps=3)
        end = [place(np.full(pr.shape, -1.0)) for _ in range(5)]
        sim.get_prim(end)
        out.append((dt, start, end, sim.get_prim(), sim.conserved_totals()))
        sim.close()
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][1] + out[0][2], out[1][1] + out[1][2]):
        np.testing.assert_array_equal(a, b)
    for a, b in zip(out[1][2], out[1][3]):  # and the same handle read both ways
        np.testing.assert_array_equal(a, b)
    assert out[0][4] == out[1][4]


@pytest.mark.parametrize("precision", [0, 1])
def test_batch_pinned_equals_pageable(precision):
    probs = cases()[1:4]
    out = []
    for place in (lambda a: a, pinned):
        ps = []
        for pr in probs:
            q = pr.params.copy()
            q.precision, q.time_stepping = precision, fv._abi.FV_TS_RK2
            ps.append(q)
        b = fv.Batch(ps)
        for i, pr in enumerate(probs):
            b.set_prim(i, *[place(a) for a in pr.prim])
        b.run(3)
        dp = ctypes.POINTER(ctypes.c_double)
        got = []
        for i, pr in enumerate(probs):
            f = [place(np.full(pr.shape, -1.0)) for _ in range(5)]
            rc = b.lib.fvgpu_batch_get_prim(b._h, i, *[a.ctypes.data_as(dp) for a in f])
            assert rc == 0, b.last_error()
            got += f
        out.append((b.times().tolist(), got))
        b.close()
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][1], out[1][1]):
        np.testing.assert_array_equal(a, b)


def test_partly_pinned_and_skipped_fields():
    """One pageable field among pinned ones takes the copies; a null output is left out."""
    pr = cases()[1]
    sim = fv.Simulation(pr.params)
    prim = [pinned(a) for a in pr.prim]
    prim[1] = pr.prim[1]
    sim.set_prim(*prim)
    want = sim.get_prim()
    out = [pinned(np.full(pr.shape, -1.0)) for _ in range(5)]
    sim.get_prim([out[0], None, out[2], None, out[4]])
    for v in (0, 2, 4):
        np.testing.assert_array_equal(out[v], want[v])
    assert (out[1] == -1.0).all() and (out[3] == -1.0).all()
    sim.close()
