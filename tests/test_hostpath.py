"""The native marshaller of run_vectors (spoc_b200/csrc/hostpath.c) against a recording stand-in for the launch call: what it
hands over, which arguments it leaves to the interpreted path, and how it marks the vectors.  Needs no GPU."""
import ctypes as C

import numpy as np
import pytest

from spoc_b200 import Backend, Vector, _lib as L, dims1d, plugin


class Calls:
    """Stands in for sb200_kernel_launch and records every call."""

    TYPE = C.CFUNCTYPE(C.c_int, C.c_uint64, C.POINTER(L.Arg), C.c_int, C.POINTER(C.c_uint32), C.POINTER(C.c_uint32), C.c_uint32,
                       C.c_uint64)

    def __init__(self):
        self.rc, self.seen = 0, []
        self.fn = Calls.TYPE(self.call)

    def call(self, handle, args, n, grid, block, shared, stream):
        field = {L.ARG_BUFFER: "buffer", L.ARG_I32: "i32", L.ARG_I64: "i64", L.ARG_F32: "f32", L.ARG_F64: "f64"}
        self.seen.append((handle, [(args[i].tag, getattr(args[i].v, field[args[i].tag])) for i in range(n)], list(grid[:3]),
                          list(block[:3]), shared, stream))
        return self.rc


@pytest.fixture
def calls():
    hp = plugin._hostpath()
    c = Calls()
    hp.bind(C.cast(c.fn, C.c_void_p).value, Vector)
    yield c
    hp.bind(C.cast(L.load().sb200_kernel_launch, C.c_void_p).value, Vector)


def _vector(n, location, address=0x1000):
    b = Backend()
    v = Vector(b, np.zeros(n, np.float32))
    v.buffer = b.Memory.Buffer(0, address, n, 4)
    v.location = location
    return v


def test_vectors_on_the_device_are_expanded_and_marked_stale(calls):
    a, b = _vector(5, Vector.BOTH), _vector(0, Vector.STALE_CPU, 0xFFFF000000000000)
    args = [a, ("float32", 1.5), b, ("int32", -7), ("int64", 1 << 40), ("float64", 0.1)]
    assert plugin._hostpath().launch(9, args, dims1d(256), dims1d(3), 64) == 0
    (handle, got, grid, block, shared, stream), = calls.seen
    assert (handle, grid, block, shared, stream) == (9, [3, 1, 1], [256, 1, 1], 64, 0)
    assert got == [(L.ARG_BUFFER, 0x1000), (L.ARG_I32, 5), (L.ARG_F32, 1.5), (L.ARG_BUFFER, 0xFFFF000000000000), (L.ARG_I32, 0),
                   (L.ARG_I32, -7), (L.ARG_I64, 1 << 40), (L.ARG_F64, 0.1)]
    assert a.location == Vector.STALE_CPU and b.location == Vector.STALE_CPU


def test_a_small_pinned_vector_is_launched_on(calls):
    v = _vector(Vector.PIN_MIN_BYTES // 4 - 1, Vector.STALE_CPU)
    v._pinned = True
    try:
        assert plugin._hostpath().launch(9, [v], dims1d(1), dims1d(1), 0) == 0
        assert len(calls.seen) == 1
    finally:
        v._pinned, v.buffer = False, None


def test_a_failed_launch_leaves_the_locations(calls):
    calls.rc = L.ERR_BOUNDS
    a = _vector(5, Vector.BOTH)
    assert plugin._hostpath().launch(9, (a,), dims1d(1), dims1d(1), 0) == L.ERR_BOUNDS
    assert a.location == Vector.BOTH


def _pinned():
    v = _vector(Vector.PIN_MIN_BYTES // 4, Vector.BOTH)     # its result would be sent back behind the launch
    v._pinned = True
    return v


def _coming_back():
    v = _vector(4, Vector.STALE_CPU)
    v._prefetch_dev = 0
    return v


def _unallocated():
    v = _vector(4, Vector.BOTH)
    v.buffer = None
    return v


@pytest.mark.parametrize("arg", [lambda: _vector(4, Vector.CPU), _pinned, _coming_back, _unallocated, lambda: ("int32", 1 << 31),
                                 lambda: ("int32", np.int32(3)), lambda: ("float32", 3), lambda: ("int16", 3), lambda: ["int32", 3],
                                 lambda: 3])
def test_everything_else_is_left_to_the_interpreted_path(calls, arg):
    first = _vector(5, Vector.BOTH)
    a = arg()
    assert plugin._hostpath().launch(9, [first, a], dims1d(1), dims1d(1), 0) is None
    assert calls.seen == [] and first.location == Vector.BOTH
    if isinstance(a, Vector):   # nothing here has a device or a registration behind it
        a._pinned, a._prefetch_dev, a.buffer = False, None, None
