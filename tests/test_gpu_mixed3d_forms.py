"""The two forms of the FP32-mixed 3-D stage give the same bits.

Groups of problems without z-boundary and corrected physics run z-marched
(blocks of up to 30 x 15 columns) or in 16 x 16 blocks, whichever their sizes
make the faster; fluxes, increments, the state, the time step and with them
every later state must not depend on it.
"""
import numpy as np
import pytest

from test_gpu_march3d32 import A, CASES, P, R, make, run

pytestmark = pytest.mark.gpu

MORE = [
    lambda: make((16, 16, 16), (P, P, P), "hllc", tc=True, visc=True),
    lambda: make((17, 33, 6), (R, A, R), "hll", gravity=True, visc=True),
    lambda: make((50, 18, 11), (A, P, A), "hll", gravity=True, tc=True, visc=True),
    lambda: make((32, 16, 40), (P, P, P), "hllc", recon="pcm", stepping="euler"),
    lambda: make((15, 19, 9), (R, R, R), "hllc", recon="pcm", tc=True, stepping="euler"),
    lambda: make((34, 17, 8), (P, R, R), "hll", recon="pcm_wb", gravity=True, tc=True, visc=True),
]


@pytest.mark.parametrize("k", range(len(CASES) + len(MORE)))
def test_same_bits(k, monkeypatch):
    pr = (CASES + MORE)[k]()
    (ref,), t = run([pr], monkeypatch, tile="30x5")[0]
    assert np.isfinite(ref).all()
    for tile in ("16x64", "16x1", "16x3"):
        ((got,), tg), sched = run([pr], monkeypatch, tile=tile)
        assert sched[0]["tx"] == 16
        assert tg[0] == t[0]
        for v in range(5):
            np.testing.assert_array_equal(got[v], ref[v], err_msg="%s %d" % (tile, v))


def test_same_bits_over_many_steps(monkeypatch):
    """Almost empty cells and the time steps of a flow that grows, 48 steps, two problems in a batch."""
    import test_gpu_march3d32 as m
    monkeypatch.setattr(m, "STEPS", 48)
    probs = [make((24, 20, 18), (P, R, A), "hll", recon="pcm", seed=s) for s in (1, 2)]
    for s, pr in enumerate(probs):
        pr.prim[0] = np.where(np.arange(pr.prim[0].size).reshape(pr.prim[0].shape) % 97 == s, 2e-6, pr.prim[0])
    a, b = (run(probs, monkeypatch, tile=tile)[0] for tile in ("30x6", "16x9"))
    np.testing.assert_array_equal(a[1], b[1])
    for x, y in zip(a[0], b[0]):
        for v in range(5):
            np.testing.assert_array_equal(x[v], y[v])


def test_a_problem_alone_and_in_a_large_batch(monkeypatch):
    """Alone it marches, one of 100 it runs in blocks: the faster form each time, and the same bits."""
    probs = [make((16, 16, 8), (P, R, P), "hllc", tc=True, visc=True, seed=s) for s in range(3)]
    (got, times), sched = run([probs[i % 3] for i in range(100)], monkeypatch)
    assert [s["tx"] for s in sched] == [16]
    for i, pr in enumerate(probs):
        ((alone,), t), s = run([pr], monkeypatch)
        assert s[0]["tx"] == 30
        for k in (i, i + 3, i + 96):
            assert times[k] == t[0]
            for v in range(5):
                np.testing.assert_array_equal(got[k][v], alone[v], err_msg="%d %d" % (k, v))


def test_form_follows_the_plane(monkeypatch):
    """Many columns: blocks of 30 x 15 where they fit the plane, 16 x 16 blocks where those do."""
    for n, tx in (((90, 45, 80), 30), ((64, 64, 64), 16), ((32, 16, 400), 16)):
        assert run([make(n, (P, P, P), "hllc", recon="pcm")], monkeypatch)[1][0]["tx"] == tx, n
