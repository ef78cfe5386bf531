"""Large fields read into host memory of every kind: the pages of a destination of 32 MB or more are made
present before the copy, which must change neither what is copied nor anything beside it, and must not
matter where the system refuses it."""
import ctypes as C
import mmap

import numpy as np
import pytest

from conftest import seeded_vorticity
from fsibe_2d_gb300 import make_params, FSIBE_FP32C

pytestmark = pytest.mark.gpu
NX, NY = 4096, 1024                                     # 32 MB a field: the least that is populated
BYTES = 8 * NX * NY


@pytest.fixture(scope="module")
def run():
    import fsibe_2d_gb300 as F
    r = F.Run(make_params(nx=NX, ny=NY, ns=16, xl=4.0, yl=1.0, x0=1.0, y0=0.5, precision=FSIBE_FP32C))
    r.init_fields(seeded_vorticity(NX, ny=NY, seed=3))
    yield r, r.vort().copy()
    r.close()


def _read(r, address):
    r._call("download_vort", C.cast(C.c_void_p(address), C.POINTER(C.c_double)))


@pytest.mark.parametrize("offset", [0, 8, 4096 - 8, 4096, 65536 + 24])
def test_unaligned_and_reused_destinations(run, offset):
    r, want = run
    m = mmap.mmap(-1, BYTES + 4 * 65536)                # fresh pages
    a = np.frombuffer(m, dtype=np.uint8)
    a[:] = 0x5a
    for _ in range(2):                                  # and the same memory again
        _read(r, a.ctypes.data + offset)
        got = np.frombuffer(m, dtype=np.float64, offset=offset, count=NX * NY)
        assert np.array_equal(got, want.ravel())
        assert (a[:offset] == 0x5a).all() and (a[offset + BYTES:] == 0x5a).all()
        got[:] = 0.0
    fresh = mmap.mmap(-1, BYTES + 4 * 65536)            # not touched before the copy
    _read(r, np.frombuffer(fresh, dtype=np.uint8).ctypes.data + offset)
    assert np.array_equal(np.frombuffer(fresh, dtype=np.float64, offset=offset, count=NX * NY), want.ravel())


def test_neighbours_without_write_access(run):
    r, want = run
    pg = mmap.PAGESIZE
    m = mmap.mmap(-1, BYTES + 2 * pg)
    a = np.frombuffer(m, dtype=np.uint8)
    a[:] = 0x33
    libc = C.CDLL(None, use_errno=True)
    base = a.ctypes.data
    for p in (base, base + pg + BYTES):
        assert libc.mprotect(C.c_void_p(p), C.c_size_t(pg), mmap.PROT_READ) == 0
    _read(r, base + pg)
    assert np.array_equal(np.frombuffer(m, dtype=np.float64, offset=pg, count=NX * NY), want.ravel())
    assert (a[:pg] == 0x33).all() and (a[pg + BYTES:] == 0x33).all()
    for p in (base, base + pg + BYTES):
        assert libc.mprotect(C.c_void_p(p), C.c_size_t(pg), mmap.PROT_READ | mmap.PROT_WRITE) == 0


def test_destinations_that_cannot_be_populated(run):
    """Page-locked memory, which the system may refuse to populate."""
    torch = pytest.importorskip("torch")
    r, want = run
    t = torch.zeros(NX * NY, dtype=torch.float64).pin_memory()
    _read(r, t.data_ptr())
    assert np.array_equal(t.numpy(), want.ravel())
