"""What a caller's streams promise to the calls enqueued on them: a call starts
after everything in front of it, whatever the caller's own kernels wait for;
the legacy default stream is ordered with the caller's blocking streams; and
the calls can be captured into a graph.  Every point is compared with the
oracle's checksum of the scalars that the call must have read."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import synth
from conftest import NATIVE

pytestmark = pytest.mark.gpu

DELAY_US = 3000  # of the caller's producer: several times what a call's launches take


@pytest.fixture(scope="module")
def caller():
    out = os.path.join(NATIVE, "_build")
    os.makedirs(out, exist_ok=True)
    so, src = os.path.join(out, "libcaller_streams.so"), os.path.join(NATIVE, "caller_streams.cu")
    subprocess.run(["nvcc", "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC", "-shared", "-cudart", "static",
                    "-o", so, src], check=True)
    lib = ctypes.CDLL(so)

    handle, size, delay = ctypes.c_void_p, ctypes.c_ulonglong, ctypes.c_uint
    for name, types in {"delayed_copy": [handle, handle, handle, size, delay], "passing": [handle], "blocking_stream": [handle],
                        "stream_destroy": [handle], "capture_begin": [handle], "capture_end": [handle, handle],
                        "graph_launch": [handle, handle], "graph_destroy": [handle]}.items():
        getattr(lib, "caller_" + name).argtypes = types

    class Caller:
        def __getattr__(self, name):
            def call(*args):
                assert getattr(lib, "caller_" + name)(*args) == 0, name
            return call
    return Caller()


class Work:
    """Bases, the scalars a call must read, and others that it must not."""

    def __init__(self, n, seed):
        import bellman_cuda as bcm
        self.bcm, self.n = bcm, n
        bc = self.bc = bcm.BellmanCuda()
        bc.set_device(0)
        bc.msm_set_up()
        self.pool, self.stream = bc.mem_pool_create(0), bc.stream_create(True)
        self.scalars, self.k = synth.workload("uniform", n, seed)
        self.stale = synth.uniform_scalars(seed + 1, n)
        kd = bc.to_device(self.k)
        self.bases = bc.malloc(n * 64)
        bc.generator_multiples(kd, self.bases, n, self.stream)
        bc.stream_synchronize(self.stream)
        bc.free(kd)
        self.source, self.read = bc.to_device(self.scalars), bc.to_device(self.stale)
        self.results, self.copied = bc.malloc(254 * 96), bc.malloc(254 * 96)
        self.point = bc.malloc(ctypes.sizeof(bcm.AffinePoint))
        bc.memcpy(self.copied, np.zeros((254, 24), np.uint32), 254 * 96)

    def warm(self):
        """Every kernel loaded, so that the launches below follow each other closely."""
        assert self.bc.msm_any(self.pool, self.stream, self.bases, self.source, self.results, self.n) == 0
        assert self.bc.final_sum_async(self.results, self.point, self.stream) == 0
        self.bc.stream_synchronize(self.stream)

    def tuple(self):
        return self.bcm.AffinePoint.from_buffer_copy(self.bc.from_device(self.point, (20,)).tobytes()).as_tuple()

    def close(self):
        for p in (self.bases, self.source, self.read, self.results, self.copied, self.point):
            self.bc.free(p)
        self.bc.stream_destroy(self.stream)
        self.bc.mem_pool_destroy(self.pool)


@pytest.mark.parametrize("path,n", [("pool", 300), ("pool", 30000), ("pool", (1 << 19) + 5), ("no_alloc", 300), ("no_alloc", 40000)])
def test_behind_a_kernel_that_waited_for_nothing(caller, oracle, path, n):
    """The scalars are written by a slow kernel; between it and the MSM the
    caller has launched one early that ends without waiting for it.  The MSM,
    and behind another such pair the final sum, still start after the writes."""
    w = Work(n, 61)
    w.warm()
    s = w.stream.handle
    caller.delayed_copy(s, w.source, w.read, n * 32, DELAY_US)
    caller.passing(s)
    if path == "pool":
        assert w.bc.msm_any(w.pool, w.stream, w.bases, w.read, w.results, n) == 0
    else:
        assert w.bc.msm_no_alloc(w.stream, w.bases, w.read, w.results, n) == 0
    caller.delayed_copy(s, w.results, w.copied, 254 * 96, DELAY_US)
    caller.passing(s)
    assert w.bc.final_sum_async(w.copied, w.point, w.stream) == 0
    w.bc.stream_synchronize(w.stream)
    got = w.tuple()
    w.close()
    assert got == oracle.msm_checksum(w.k, w.scalars)


@pytest.mark.parametrize("n", [300, (1 << 19) + 5])
def test_legacy_stream_between_blocking_streams(caller, oracle, n):
    """MSM and final sum on the legacy default stream, between a blocking
    stream's producer of the scalars and its later overwriting of them."""
    w = Work(n, 71)
    w.warm()
    blocking = ctypes.c_void_p()
    caller.blocking_stream(ctypes.byref(blocking))
    legacy = w.bcm.Handle()
    stale = w.bc.to_device(w.stale)
    caller.delayed_copy(blocking, w.source, w.read, n * 32, DELAY_US)
    assert w.bc.msm_any(w.pool, legacy, w.bases, w.read, w.results, n) == 0
    assert w.bc.final_sum_async(w.results, w.point, legacy) == 0
    caller.delayed_copy(blocking, stale, w.read, n * 32, 0)
    w.bc.stream_synchronize(w.bcm.Handle(blocking.value))
    w.bc.stream_synchronize(legacy)
    got = w.tuple()
    caller.stream_destroy(blocking)
    w.bc.free(stale)
    w.close()
    assert got == oracle.msm_checksum(w.k, w.scalars)


@pytest.mark.parametrize("path,n", [("pool", 300), ("pool", (1 << 19) + 5), ("no_alloc", 300), ("no_alloc", 40000)])
def test_captured(caller, oracle, path, n):
    """MSM and final sum captured into a graph and replayed, the second time
    with other scalars in the same buffer."""
    w = Work(n, 81)
    w.warm()
    s = w.stream.handle
    if path == "no_alloc":
        assert w.bc.msm_no_alloc(w.stream, w.bases, w.read, w.results, n) == 0
        w.bc.stream_synchronize(w.stream)
    graph = ctypes.c_void_p()
    caller.capture_begin(s)
    if path == "pool":
        assert w.bc.msm_any(w.pool, w.stream, w.bases, w.read, w.results, n) == 0
    else:
        assert w.bc.msm_no_alloc(w.stream, w.bases, w.read, w.results, n) == 0
    assert w.bc.final_sum_async(w.results, w.point, w.stream) == 0
    caller.capture_end(s, ctypes.byref(graph))
    got = []
    for scalars in (w.stale, w.scalars):
        w.bc.memcpy(w.read, scalars, n * 32)
        w.bc.stream_synchronize(w.bcm.Handle())
        caller.graph_launch(graph, s)
        w.bc.stream_synchronize(w.stream)
        got.append(w.tuple())
    caller.graph_destroy(graph)
    w.close()
    assert got == [oracle.msm_checksum(w.k, w.stale), oracle.msm_checksum(w.k, w.scalars)]
