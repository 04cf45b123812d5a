"""A call that CUDA refuses leaves the calls after it alone.

An array whose first page only is registered can be neither read in place nor
copied; the call reports that, and the error must not come up again in the
next launch of any handle.
"""
import mmap

import numpy as np
import pytest

import fv3d_gb300 as fv
from fv3d_gb300 import problems

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("precision", [0, 1])
def test_next_call_after_a_refused_copy(precision):
    pr = problems.sedov(256)
    params = pr.params.copy()
    params.precision = precision
    torch.zeros(1, device="cuda")
    mem = mmap.mmap(-1, 256 * 256 * 8 + mmap.PAGESIZE)
    part = np.frombuffer(mem, np.float64)[:256 * 256].reshape(pr.shape)
    base = part.__array_interface__["data"][0]
    part[...] = pr.prim[0]
    sim, other = fv.Simulation(params), fv.Simulation(params)
    assert int(torch.cuda.cudart().cudaHostRegister(base, mmap.PAGESIZE, 0)) == 0
    try:
        with pytest.raises(fv.FvError):
            sim.set_prim(part, *pr.prim[1:])
        other.set_prim(*pr.prim)
        with pytest.raises(fv.FvError):
            other.get_prim([part, None, None, None, None])
        sim.set_prim(*pr.prim)
        got = sim.get_prim()
    finally:
        torch.cuda.cudart().cudaHostUnregister(base)
        sim.close()
        other.close()
    np.testing.assert_array_equal(got[0], pr.prim[0])
