"""Which host arrays the conversion kernels may read and write in place.

An array counts as pinned when it lies in one pinned allocation or
registration.  One whose ends lie in two, with pageable memory between them,
does not, and takes the copies of pageable arrays.
"""
import ctypes
import mmap

import numpy as np
import pytest

import fv3d_gb300 as fv
from fv3d_gb300 import problems

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MB = 1 << 20


@pytest.fixture
def buffer():
    """8 MB of page-aligned memory and a function that registers a part of it."""
    torch.cuda.init()
    torch.zeros(1, device="cuda")
    mem = mmap.mmap(-1, 8 * MB)
    a = np.frombuffer(mem, np.float64)
    base, done = a.__array_interface__["data"][0], []

    def register(start, size):
        assert int(torch.cuda.cudart().cudaHostRegister(base + start, size, 0)) == 0
        done.append(base + start)

    yield a, register
    for p in done:
        torch.cuda.cudart().cudaHostUnregister(p)


def pinned(*arrays, n):
    """pinned_fields of the library on (up to five) arrays of n values."""
    f = fv.load_library()._ZN2fv13pinned_fieldsEPKPKdxPNS_6FieldsE
    f.restype = ctypes.c_bool
    ptrs = (ctypes.c_void_p * 5)(*[a.__array_interface__["data"][0] for a in arrays])
    view = (ctypes.c_void_p * 5)()
    ok = f(ptrs, ctypes.c_longlong(n), view)
    if ok:
        assert list(view) == list(ptrs)  # GB300: one address for both processors
    return ok


def test_ranges(buffer):
    a, register = buffer
    per = MB // 8
    assert not pinned(a, n=a.size)
    register(0, MB)
    register(4 * MB, MB)
    assert pinned(a, n=per) and pinned(a[4 * per:], n=per) and pinned(a[4 * per + 3:], n=per - 3)
    assert not pinned(a, n=5 * per)  # both ends pinned, the middle not
    assert not pinned(a, n=per + 1) and not pinned(a[1:], n=per) and not pinned(a[2 * per:], n=2 * per + 1)
    assert pinned(a, a[4 * per:], n=per) and not pinned(a, a[per:], n=per)


def test_allocations():
    t = torch.empty(3 * MB // 8, dtype=torch.float64, pin_memory=True).numpy()
    assert pinned(t, n=t.size) and pinned(t[17:], t[1:], n=t.size - 17)
    assert not pinned(np.zeros(100), n=100)
    d = torch.zeros(100, dtype=torch.float64, device="cuda")

    class Device:
        __array_interface__ = {"data": (d.data_ptr(), False)}

    assert not pinned(Device(), n=100)


@pytest.mark.parametrize("precision", [0, 1])
def test_states_across_two_registrations_are_refused(buffer, precision):
    """CUDA copies no array that begins in one registration and ends in another; the call says so."""
    a, register = buffer
    pr = problems.random_problem("r", problems._mesh(256, 200, 1), {"tend": 1.0}, {"riemann_solver": "hllc"},
                                 {"gamma0": 1.4}, 7)
    pr.prim[3] = None
    n, per = 256 * 200, MB // 8
    assert n * 8 > 4 * mmap.PAGESIZE
    for k in range(5):
        register(k * MB, mmap.PAGESIZE)
        register(k * MB + (n * 8 - 1) // mmap.PAGESIZE * mmap.PAGESIZE, mmap.PAGESIZE)
    fields = [a[k * per:k * per + n].reshape(pr.shape) for k in range(5)]
    for k in (0, 1, 2, 4):
        fields[k][...] = pr.prim[k]
    params = pr.params.copy()
    params.precision = precision
    sim = fv.Simulation(params)
    with pytest.raises(fv.FvError):
        sim.set_prim(*[None if k == 3 else f for k, f in enumerate(fields)])
    sim.close()
    sim = fv.Simulation(params)
    sim.set_prim(*pr.prim)
    with pytest.raises(fv.FvError):
        sim.get_prim(fields)
    sim.close()
