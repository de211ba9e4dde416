"""populate_pages (csrc/mfc_launch.h), which makes the destination of a download
resident: pinned arrays, large arrays and everything on a machine without a
device keep what they hold, fresh pages become resident, and a download gives
the same values wherever it goes."""
import ctypes
import mmap

import numpy as np
import pytest

BIG = 300 * mmap.PAGESIZE


def _populate():
    from microfc_gb300 import _lib
    f = _lib.load()._ZN3mfc14populate_pagesEPvm
    f.argtypes = [ctypes.c_void_p, ctypes.c_size_t]
    f.restype = None
    return f


def _stays(a):
    f = _populate()
    a[:] = np.arange(len(a), dtype=np.uint32).astype(np.uint8) | 1
    want = a.copy()
    f(a.ctypes.data + 1, len(a) - 1)
    f(None, 100)
    assert np.array_equal(a, want)


def test_contents_stay_without_a_device():
    import torch
    if torch.cuda.is_available():
        pytest.skip("there is a device")
    for n in (2, 4097, 1 << 20, BIG + 5):
        _stays(np.empty(n, dtype=np.uint8))


@pytest.mark.gpu
def test_contents_of_large_and_pinned_arrays_stay():
    import torch
    torch.zeros(1, device="cuda")
    _stays(np.empty(BIG + 5, dtype=np.uint8))
    for n in (4097, BIG + 5):
        _stays(torch.empty(n, dtype=torch.uint8, pin_memory=True).numpy())


@pytest.mark.gpu
@pytest.mark.parametrize("pages", [3, 300])
def test_fresh_pages_become_resident(pages):
    import torch
    torch.zeros(1, device="cuda")
    f = _populate()
    libc = ctypes.CDLL(None, use_errno=True)
    with mmap.mmap(-1, pages * mmap.PAGESIZE, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS) as m:
        view = (ctypes.c_char * len(m)).from_buffer(m)
        at = ctypes.c_void_p(ctypes.addressof(view))
        f(at, len(m))
        vec = (ctypes.c_ubyte * pages)()
        assert libc.mincore(at, ctypes.c_size_t(len(m)), vec) == 0
        del view
    assert all(v & 1 for v in vec)


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(40, 26), (900, 500)])
def test_downloads_agree_wherever_they_go(nx, ny):
    import torch
    from microfc_gb300 import Simulation, cases, preprocess
    c = cases.shock_droplet_2d(nx=64, ny=32, steps=2, dt=1e-9).replace(m=nx - 1, n=ny - 1)
    x, y, z, q = preprocess.generate(c)
    n = q.nbytes
    with Simulation(c, x, y, z, q_cons=q) as sim:
        fresh = np.frombuffer(mmap.mmap(-1, n, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS), dtype=np.float64)
        for out in (np.full(c.shape, 7.0), fresh.reshape(c.shape),
                    torch.full(c.shape, 7.0, dtype=torch.float64, pin_memory=True).numpy()):
            assert np.array_equal(sim.download(out), q)
