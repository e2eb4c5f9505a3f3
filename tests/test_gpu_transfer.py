"""Page-locked rings and recycled device blocks: what else the process is doing meanwhile."""
import ctypes as C
import threading
import time

import numpy as np
import pytest
import torch

from alsparse_b200 import capi, spblas, synth
from gpu_util import check_mv, make_handle

pytestmark = pytest.mark.gpu


class Capture:
    """Captures what the library puts on a stream of its own; the graph is thrown away."""

    def __enter__(self):
        self.cu, self.stream = C.CDLL("libcuda.so.1"), torch.cuda.Stream()
        self.stream.wait_stream(torch.cuda.current_stream())
        spblas.set_stream(self.stream.cuda_stream)
        assert self.cu.cuStreamBeginCapture_v2(C.c_void_p(self.stream.cuda_stream), 2) == 0  # relaxed
        return self

    def __exit__(self, *_):
        graph = C.c_void_p()
        self.cu.cuStreamEndCapture(C.c_void_p(self.stream.cuda_stream), C.byref(graph))
        if graph.value:
            self.cu.cuGraphDestroy(graph)
        spblas.set_stream(None)
        torch.cuda.synchronize()


def triples(nnz, rows):
    rng = np.random.default_rng(nnz)
    return rng.integers(rows, size=nnz, dtype=np.int32), rng.integers(rows, size=nnz, dtype=np.int32), rng.random(nnz)


def test_copies_refused_inside_a_capture_leave_later_ones_alone():
    """Host vectors and conversions wait for the device, so a capture ends with an error; the calls behind it do not."""
    m = synth.zipf("d", 5, 200000, 200000, 1.8, 1, 100000)
    A = make_handle("d", m)
    x, y = synth.vector("d", 1, 1, m.cols), synth.vector("d", 1, 2, m.nrows)  # (1.6 MB: more than a small block)
    dx, dy = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    ri, ci, v = triples(300000, 20000)
    st, coo = spblas.create_coo("d", capi.BASE_ZERO, 20000, 20000, len(v), ri, ci, v)
    assert st == capi.SUCCESS
    for vectors in ((x, dy), (dx, y), (x, y)):
        assert spblas.mv("d", 0, 1.0, A, spblas.descr(), vectors[0], 0.5, vectors[1]) == capi.SUCCESS  # (staging buffers)
    for vectors in ((x, dy), (dx, y), (x, y)) * 5:
        with Capture():
            assert spblas.mv("d", 0, 1.0, A, spblas.descr(), vectors[0], 0.5, vectors[1]) != capi.SUCCESS
    with Capture():
        status, B = spblas.convert_csr(coo)
        assert status != capi.SUCCESS
    check_mv("d", m, 1.5, 0.5, A=A)
    spblas.destroy(A)
    large = synth.poisson("d", 6, 300000, 300000, 9.0)  # 21 MB of values: every chunk of the ring more than once
    check_mv("d", large, 1.5, 0.5)
    status, B = spblas.convert_csr(coo)
    assert status == capi.SUCCESS, spblas.last_error()
    for h in (coo, B):
        spblas.destroy(h)


@pytest.mark.parametrize("mode", [1, 2])  # thread-local, relaxed: what other threads do is no part of the capture
def test_assembly_in_another_thread_leaves_a_capture_alone(mode):
    """A program that records a graph in one thread and converts and destroys matrices in another."""
    ri, ci, v = triples(300000, 20000)

    def assemble():
        st, coo = spblas.create_coo("d", capi.BASE_ZERO, 20000, 20000, len(v), ri, ci, v)
        st2, A = spblas.convert_csr(coo)
        assert st == st2 == capi.SUCCESS, spblas.last_error()
        spblas.destroy(coo)
        return A

    handles = [assemble() for _ in range(3)]
    cu, stream, done = C.CDLL("libcuda.so.1"), torch.cuda.Stream(), []
    x, y = torch.ones(20000, dtype=torch.float64, device="cuda"), torch.zeros(20000, dtype=torch.float64, device="cuda")
    assert spblas.mv("d", 0, 1.0, handles[1], spblas.descr(), x, 0.0, y) == capi.SUCCESS  # queued, not waited for
    assert cu.cuStreamBeginCapture_v2(C.c_void_p(stream.cuda_stream), mode) == 0

    def work():
        torch.cuda.set_device(0)
        for A in handles:
            spblas.destroy(A)
        spblas.destroy(assemble())
        done.append(True)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    graph = C.c_void_p()
    ended = cu.cuStreamEndCapture(C.c_void_p(stream.cuda_stream), C.byref(graph))
    if graph.value:
        cu.cuGraphDestroy(graph)
    assert done and ended == 0


def test_memory_of_a_destroyed_handle_is_not_handed_out_under_its_products():
    """A product still queued when its handle is destroyed, and a conversion of the same size right behind it."""
    ri, ci, v = triples(300000, 20000)

    def assemble(values):
        st, coo = spblas.create_coo("d", capi.BASE_ZERO, 20000, 20000, len(v), ri, ci, values)
        st2, A = spblas.convert_csr(coo)
        assert st == st2 == capi.SUCCESS, spblas.last_error()
        spblas.destroy(coo)
        return A

    x = torch.ones(20000, dtype=torch.float64, device="cuda")
    want, got = (torch.zeros(20000, dtype=torch.float64, device="cuda") for _ in range(2))
    side = torch.cuda.Stream()
    A = assemble(v)
    assert spblas.mv("d", 0, 1.0, A, spblas.descr(), x, 0.0, want) == capi.SUCCESS
    torch.cuda.synchronize()
    for stream in (None, side.cuda_stream):
        got.zero_()
        torch.cuda.synchronize()
        spblas.set_stream(stream)
        try:
            with torch.cuda.stream(side if stream else torch.cuda.default_stream()):
                torch.cuda._sleep(100_000_000)  # about 50 ms in front of the product
                assert spblas.mv("d", 0, 1.0, A, spblas.descr(), x, 0.0, got) == capi.SUCCESS
        finally:
            spblas.set_stream(None)
        spblas.destroy(A)
        A = assemble(-v)
        torch.cuda.synchronize()
        assert torch.equal(got, want)
        spblas.destroy(A)
        A = assemble(v)
    spblas.destroy(A)


@pytest.mark.parametrize("way", ["up", "down"])
def test_copies_do_not_wait_for_another_thread(way):
    """A product behind a long queue on one stream, and one with vectors as large on an idle stream from another thread."""
    m = synth.poisson("d", 7, 900000, 3300000, 3.0)  # x 26 MB, more than a ring holds; y 7 MB
    x = synth.vector("d", 7, 1, m.cols)
    dx = torch.from_numpy(x).cuda()
    streams, handles = [torch.cuda.Stream() for _ in range(2)], [make_handle("d", m) for _ in range(2)]
    ys = [np.zeros(m.nrows) if way == "down" else torch.zeros(m.nrows, dtype=torch.float64, device="cuda") for _ in range(2)]

    def call(i):
        assert spblas.mv("d", 0, 1.0, handles[i], spblas.descr(), dx if way == "down" else x, 0.0, ys[i]) == capi.SUCCESS

    try:
        for i in range(2):  # (staging buffers and, once, the answer)
            spblas.set_stream(streams[i].cuda_stream)
            call(i)
            torch.cuda.synchronize()
        want = ys[0].copy() if way == "down" else ys[0].clone()
        with torch.cuda.stream(streams[0]):
            torch.cuda._sleep(2_000_000_000)  # about a second
            queued = torch.cuda.Event()
            queued.record()
        spblas.set_stream(streams[0].cuda_stream)  # (read when a call begins)
        first = threading.Thread(target=call, args=(0,))
        first.start()
        time.sleep(0.2)
        spblas.set_stream(streams[1].cuda_stream)
        call(1)
        assert not queued.query(), "the call waited for the other thread's"
        first.join()
    finally:
        spblas.set_stream(None)
    torch.cuda.synchronize()
    for y in ys:
        assert (y == want).all()
    for A in handles:
        spblas.destroy(A)


def test_kept_memory_is_reported_and_given_back():
    """What conversions leave in the cache can be had back, and a handle reports the block it really holds."""
    def assemble(nnz):
        rng = np.random.default_rng(nnz)
        ri, ci = rng.integers(50000, size=nnz, dtype=np.int32), rng.integers(50000, size=nnz, dtype=np.int32)
        st, coo = spblas.create_coo("d", capi.BASE_ZERO, 50000, 50000, nnz, ri, ci, np.ones(nnz))
        st2, A = spblas.convert_csr(coo)
        assert st == st2 == capi.SUCCESS, spblas.last_error()
        spblas.destroy(coo)
        return A

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    spblas.destroy(assemble(3000000))  # (kernels loaded)
    assert spblas.release_cached_memory() == capi.SUCCESS
    base = free()
    spblas.destroy(assemble(3000000))
    assert free() < base - (30 << 20)  # kept for the next conversion
    A = assemble(1700000)  # its arrays take a little more than half of the block that lies there
    spblas.release_cached_memory()
    held, reported = base - free(), spblas.mat_info(A)[1].device_bytes
    assert abs(held - reported) <= 6 << 20  # CUDA hands memory out in pieces of 2 MB
    assert reported <= 1.3 * 1700000 * 12 + (1 << 20)
    check_mv("d", synth.poisson("d", 6, 300000, 300000, 9.0), 1.5, 0.5)  # rings made anew
    spblas.destroy(A)
    spblas.release_cached_memory()
    assert abs(base - free()) <= 2 << 20
