"""mv with host vectors: the sizes at which the way they travel changes, and more callers than page-locked blocks."""
import threading

import numpy as np
import pytest

import oracle
from alsparse_b200 import capi, spblas, synth
from gpu_util import check_mv, make_handle
from helpers import NP, assert_rows_close, row_scale

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["s", "d"])
@pytest.mark.parametrize("rows_bytes", [8, 64 << 10, (64 << 10) + 8, 250 << 10, 256 << 10, (256 << 10) + 8])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_sizes_around_the_limits(kind, rows_bytes, beta):
    # up to 64 KB of y the kernel works on the block, up to 512 KB together the vectors are packed, above they are copied
    n = rows_bytes // np.dtype(NP[kind]).itemsize
    for m in (synth.poisson(kind, 3, n, n, 9.0), synth.poisson(kind, 4, n, max(1, n // 3), 3.0)):
        check_mv(kind, m, 1.5, beta)


@pytest.mark.parametrize("make", [lambda k: synth.zipf(k, 5, 3000, 3000, 1.8, 1, 1500), lambda k: synth.stencil27(k, 12),
                                  lambda k: synth.from_lengths(k, 5, np.zeros(300, np.int32), 200)])
@pytest.mark.parametrize("kind", ["s", "d"])
def test_every_kernel_family(kind, make):
    m = make(kind)
    for beta in (0.0, 0.5):
        check_mv(kind, m, -1.0, beta)
    A, x = make_handle(kind, m), synth.vector(kind, 1, 1, m.cols)
    y = np.full(m.nrows, np.nan, NP[kind])  # beta == 0: what y held does not matter
    assert spblas.mv(kind, 0, 1.0, A, spblas.descr(), x, 0.0, y) == capi.SUCCESS and np.isfinite(y).all()
    spblas.destroy(A)


@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_large_pageable_vectors_in_windows(beta):
    rows = (1 << 20) + 777
    check_mv("s", synth.poisson("s", 6, rows, 3001, 2.0), 1.5, beta)


def test_more_callers_than_blocks():
    m = synth.poisson("d", 7, 4000, 4000, 8.0)
    x, y0 = synth.vector("d", 7, 1, m.cols), synth.vector("d", 7, 2, m.nrows)
    ref = oracle.gemv("d", m.rows_start, m.rows_end, m.col, m.val, 1.5, x, 0.5, y0.copy())
    scale = row_scale(m.ptr, m.col, m.val, x, 1.5, 0.5, y0)
    handles = [make_handle("d", m) for _ in range(12)]
    results = [None] * len(handles)

    def work(i):
        for _ in range(20):
            y = y0.copy()
            assert spblas.mv("d", 0, 1.5, handles[i], spblas.descr(), x, 0.5, y) == capi.SUCCESS
        results[i] = y

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(handles))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for y in results:
        assert y is not None
        assert_rows_close("d", y, ref, scale, "concurrent callers")
    for A in handles:
        spblas.destroy(A)
