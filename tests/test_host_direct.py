"""frg_update_host's choice between a kernel's own stores and a copy, on the host:
stores only where the whole state lies in one pinned range that the device may
write.  (A state that runs past the end of its range would fault the device.)"""
import ctypes as C

import pytest

HOST, DEVICE, RW, RO = 1, 2, 3, 1
BASE, SIZE = 0x10000, 0x3000


def _target(host, nbytes, mem_type=HOST, access=RW, dev=None, start=BASE, size=SIZE):
    from fr_learn_b200.solver import lib

    f = lib().frg_direct_target
    f.argtypes = [C.c_void_p, C.c_ulonglong, C.c_uint, C.c_uint] + [C.c_ulonglong] * 3
    f.restype = C.c_void_p
    return f(host, nbytes, mem_type, access, host if dev is None else dev, start, size)


@pytest.mark.parametrize("off, nbytes", [(0, SIZE), (0, 8), (SIZE - 8, 8), (0x1000, 0x2000)])
def test_inside_one_writable_range_is_stored_to(off, nbytes):
    assert _target(BASE + off, nbytes) == BASE + off
    assert _target(BASE + off, nbytes, dev=0x7F0000000000 + off) == 0x7F0000000000 + off


@pytest.mark.parametrize("off, nbytes", [(0, SIZE + 8), (8, SIZE), (SIZE - 8, 16), (SIZE, 8), (-8, 16), (0, 1 << 63)])
def test_past_the_range_is_copied(off, nbytes):
    assert _target(BASE + off, nbytes) is None


@pytest.mark.parametrize("kw", [dict(mem_type=0), dict(mem_type=DEVICE), dict(access=RO), dict(access=0), dict(dev=0)])
def test_pageable_device_and_read_only_memory_is_copied(kw):
    assert _target(BASE, 64, **kw) is None


@pytest.mark.parametrize("off", [1, 4])
def test_a_misaligned_state_is_copied(off):
    assert _target(BASE + off, 64) is None
    assert _target(BASE, 64, dev=BASE + off) is None
