"""ResultPages (ep_hostmem.h): the pages of a result array are made resident
ahead of its download without a store to them, so that an array which overlaps
an input, or belongs to a call that fails later, keeps its contents."""
import ctypes
import mmap

import numpy as np
import pytest

MB = 1 << 20
SLAB = 8 * MB


def _pages(native, addr, n):
    """Constructs ResultPages(addr, n), waits for every slab, destroys it."""
    sym = lambda s, *a: ctypes.CFUNCTYPE(None, ctypes.c_void_p, *a)((s, native))  # noqa: E731
    ctor = sym("_ZN2ep11ResultPagesC1EPvm", ctypes.c_void_p, ctypes.c_size_t)
    wait = sym("_ZN2ep11ResultPages4waitEm", ctypes.c_size_t)
    dtor = sym("_ZN2ep11ResultPagesD1Ev")
    obj = ctypes.create_string_buffer(512)          # larger than the object
    at = ctypes.c_void_p((ctypes.addressof(obj) + 63) // 64 * 64)
    ctor(at, addr, n)
    for i in range((n + SLAB - 1) // SLAB):
        wait(at, i)
    dtor(at)


@pytest.mark.parametrize("n", [0, 1, 4095, 70_001, 9 * MB + 3, 32 * MB - 1, 32 * MB, 70 * MB + 5])
@pytest.mark.parametrize("offset", [0, 13])
def test_contents_are_kept(native, n, offset):
    a = np.random.default_rng(n).integers(1, 256, n + offset + 64, dtype=np.uint8)
    want = a.copy()
    _pages(native, a.ctypes.data + offset, n)
    assert np.array_equal(a, want)


@pytest.mark.parametrize("n", [20 * MB, 80 * MB])
def test_fresh_pages_are_resident_and_zero(native, n):
    libc = ctypes.CDLL(None, use_errno=True)
    m = mmap.mmap(-1, n)
    view = ctypes.c_char.from_buffer(m)
    addr = ctypes.addressof(view)
    if libc.madvise(ctypes.c_void_p(addr), ctypes.c_size_t(mmap.PAGESIZE), 23):
        pytest.skip("this kernel has no MADV_POPULATE_WRITE")
    _pages(native, addr, n)
    vec = (ctypes.c_ubyte * (n // mmap.PAGESIZE))()
    assert libc.mincore(ctypes.c_void_p(addr), ctypes.c_size_t(n), vec) == 0
    assert all(v & 1 for v in vec)
    assert not np.frombuffer(m, np.uint8).any()
    del view


def test_read_only_pages_are_left_alone(native):
    # the advice fails there; the copy that follows reports the error
    m = mmap.mmap(-1, 64 * MB, prot=mmap.PROT_READ)
    a = np.frombuffer(m, np.uint8)
    _pages(native, a.ctypes.data, a.nbytes)
    assert not a.any()
