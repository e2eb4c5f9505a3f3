"""Copies between pageable host memory and the device through the page-locked rings: what else the process is doing."""
import ctypes as C

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
