"""The row-major dense-block product's element-stream kernel: edges of its batches and segments, rows cut over segments,
more column slices than one grid holds, and the calls that may not allocate."""
import numpy as np
import pytest
import torch

import oracle
from alsparse_b200 import capi, spblas, synth
from gpu_util import TORCH, make_handle
from helpers import assert_rows_close, mm_scale

pytestmark = pytest.mark.gpu


def lengths(shape):
    if shape == "even":  # whole rows per warp, empty ones among them
        lens = synth.rowlen_poisson(21, 9001, 6.0, 900).copy()
        lens[::13] = 0
        return lens
    # rows around the lengths at which a row may be cut, long rows side by side, runs of empty rows at both ends
    rng = np.random.default_rng(3)
    lens = rng.choice([0, 0, 1, 2, 7, 31, 32, 33, 63, 64, 65, 66, 127], 4000).astype(np.int32)
    lens[:40] = 0
    lens[-50:] = 0
    lens[[40, 41, 1000, 1001, 3949]] = [900, 257, 2000, 256, 1999]
    return lens


def multiply(kind, A, alpha, X, columns, ldx, beta, Y, ldy):
    assert spblas.mm(kind, 0, alpha, A, spblas.descr(), capi.ROW_MAJOR, X, columns, ldx, beta, Y, ldy) == capi.SUCCESS, \
        spblas.last_error()


def check(kind, m, A, columns, pad=0, alpha=1.5, beta=0.5, call=multiply):
    ldx, ldy = columns + pad, columns + pad
    X, Y0 = synth.vector(kind, 5, 3, m.cols * ldx), synth.vector(kind, 5, 4, m.nrows * ldy)
    # (long fp32 rows: the oracle in double precision spends no tolerance on its own rounding)
    f = np.float64
    ref = oracle.gemm("d", "row", m.rows_start, m.rows_end, m.col, m.val.astype(f), alpha, X.astype(f), columns, ldx, beta,
                      Y0.astype(f), ldy)
    dX, dY = torch.from_numpy(X).cuda(), torch.from_numpy(Y0).cuda()
    call(kind, A, alpha, dX, columns, ldx, beta, dY, ldy)
    torch.cuda.synchronize()
    scale = mm_scale(m.ptr, m.col, m.val, X, columns, ldx, alpha, beta, Y0, ldy)
    shape = (m.nrows, ldy)
    assert_rows_close(kind, dY.cpu().numpy().reshape(shape)[:, :columns].reshape(-1),
                      ref.reshape(shape)[:, :columns].reshape(-1), scale.reshape(-1), f"{columns} columns")


@pytest.mark.parametrize("kind", ["s", "d"])
@pytest.mark.parametrize("shape", ["even", "skewed"])
def test_batches_segments_and_cut_rows(kind, shape):
    m = synth.from_lengths(kind, 21, lengths(shape), 2500)
    A = make_handle(kind, m)
    for columns, pad in ((9, 0), (12, 0), (16, 0), (20, 3), (33, 0), (64, 0), (130, 2)):
        check(kind, m, A, columns, pad)
    check(kind, m, A, 24, beta=0.0)
    spblas.destroy(A)


def test_more_column_slices_than_a_grid_is_high():
    columns = 65535 * 32 + 1  # odd: single elements, 32 lanes wide
    lens = np.array([2, 0, 3], np.int32)
    m = synth.from_lengths("s", 4, lens, 3)
    A = make_handle("s", m)
    X = torch.rand(3, columns, device="cuda")
    Y = torch.zeros(3, columns, device="cuda")
    multiply("s", A, 1.0, X, columns, columns, 0.0, Y, columns)
    dense = np.zeros((3, 3))
    np.add.at(dense, (np.repeat(np.arange(3), lens), m.col), m.val)
    ref = torch.from_numpy(dense).cuda() @ X.double()
    assert float((Y - ref).abs().max()) <= 1e-5 * 3
    spblas.destroy(A)


@pytest.mark.parametrize("kind", ["s", "d"])
def test_products_that_may_not_allocate(kind):
    """A capture before and after the segment table exists, a wider product behind a recorded one, a refused allocation."""
    m = synth.from_lengths(kind, 21, lengths("skewed"), 2500)
    lib = capi.load()
    side = torch.cuda.Stream()

    def captured(*args):
        side.wait_stream(torch.cuda.current_stream())
        graph = torch.cuda.CUDAGraph()
        spblas.set_stream(side.cuda_stream)
        try:
            with torch.cuda.stream(side), torch.cuda.graph(graph, stream=side):
                multiply(*args)
            graph.replay()
        finally:
            spblas.set_stream(None)
        torch.cuda.synchronize()

    def denied(*args):
        lib.alphasparse_cuda_debug_fail_alloc(1)
        try:
            multiply(*args)
        finally:
            lib.alphasparse_cuda_debug_fail_alloc(0)

    even = synth.from_lengths(kind, 21, lengths("even"), 2500)
    A = make_handle(kind, even)
    for columns in (24, 40):
        check(kind, even, A, columns)  # (loads the kernels)
    spblas.destroy(A)
    A = make_handle(kind, m)
    check(kind, m, A, 24, call=captured)
    check(kind, m, A, 24, call=denied)
    spblas.set_stream(side.cuda_stream)
    try:
        check(kind, m, A, 24)  # the table, and room for 24 columns on this stream
    finally:
        spblas.set_stream(None)
    check(kind, m, A, 24, call=captured)
    check(kind, m, A, 40, call=captured)  # no room for 40

    # a recorded product stays usable behind a wider one
    x, y, z = (torch.rand(n, dtype=TORCH[kind], device="cuda") for n in (m.cols * 24, m.nrows * 24, m.cols * 128))
    want = torch.zeros_like(y)
    graph = torch.cuda.CUDAGraph()
    side.wait_stream(torch.cuda.current_stream())
    spblas.set_stream(side.cuda_stream)
    try:
        with torch.cuda.stream(side):
            multiply(kind, A, 1.0, x, 24, 24, 0.0, want, 24)
            with torch.cuda.graph(graph, stream=side):
                multiply(kind, A, 1.0, x, 24, 24, 0.0, y, 24)
            multiply(kind, A, 1.0, z, 128, 128, 0.0, torch.zeros(m.nrows * 128, dtype=TORCH[kind], device="cuda"), 128)
            graph.replay()
            side.synchronize()
    finally:
        spblas.set_stream(None)
    assert torch.equal(y, want)
    spblas.destroy(A)


@pytest.mark.parametrize("longest,blocks_run", [(90, True), (900, True), (1500, False)])
def test_column_blocks_where_they_are_asked_for(longest, blocks_run):
    """Mean 12: even rows, a row that the segment table would cut, and one too long for a lane group (one pass then)."""
    lens = synth.rowlen_poisson(13, 4000, 12.0, 60).copy()
    lens[11] = longest
    m = synth.from_lengths("s", 13, lens, 3000)
    A = make_handle("s", m)
    try:
        for blocks in (2, 5, 1):
            assert spblas.set_option("spmm_col_blocks", blocks) == capi.SUCCESS
            check("s", m, A, 24)  # (the table)
            before = spblas.launch_count()
            check("s", m, A, 24)
            launches, reported = spblas.launch_count() - before, spblas.mat_info(A)[1].spmm_col_blocks
            if blocks_run and blocks > 1:
                assert launches == blocks and reported == blocks
            else:
                assert launches <= 2 and reported == 1
    finally:
        spblas.set_option("spmm_col_blocks", -1)
        spblas.destroy(A)


@pytest.mark.parametrize("shape", ["skewed", "thirty"])
def test_rows_of_x_that_no_element_names_are_dropped(shape):
    """The kernel reads row 0 of X behind the end of a segment: what it holds must not reach Y."""
    lens = lengths("skewed") if shape == "skewed" else np.full(3001, 30, np.int32)
    m = synth.from_lengths("s", 21, lens, 2500)
    m = synth.Csr(m.nrows, m.cols + 1, 0, m.ptr, m.col + 1, m.val)  # column 0 is in no row
    A = make_handle("s", m)
    for columns in (12, 33, 64):
        X = torch.rand(m.cols, columns, device="cuda")
        Y = torch.empty(2, m.nrows, columns, device="cuda")
        for y, worst in zip(Y, (0.0, float("nan"))):
            X[0] = worst
            multiply("s", A, 1.5, X, columns, columns, 0.0, y, columns)
        torch.cuda.synchronize()
        assert torch.equal(Y[0], Y[1])
        X[0] = float("inf")
        multiply("s", A, 1.5, X, columns, columns, 0.0, Y[1], columns)
        torch.cuda.synchronize()
        assert torch.equal(Y[0], Y[1])
    spblas.destroy(A)


def test_two_streams_of_one_handle_at_once():
    """Each stream has partial sums of its own for the rows that are cut over segments."""
    m = synth.from_lengths("d", 21, lengths("skewed"), 2500)
    A = make_handle("d", m)
    columns, streams = 64, [torch.cuda.Stream() for _ in range(2)]
    xs = [torch.rand(m.cols, columns, dtype=torch.float64, device="cuda") for _ in streams]
    ys = [torch.zeros(m.nrows, columns, dtype=torch.float64, device="cuda") for _ in streams]
    want = [torch.zeros_like(y) for y in ys]
    for x, y in zip(xs, want):
        multiply("d", A, 1.0, x, columns, columns, 0.0, y, columns)
    torch.cuda.synchronize()
    try:
        for _ in range(50):  # products of the two streams run side by side
            for s, x, y in zip(streams, xs, ys):
                spblas.set_stream(s.cuda_stream)
                multiply("d", A, 1.0, x, columns, columns, 0.0, y, columns)
    finally:
        spblas.set_stream(None)
    torch.cuda.synchronize()
    for y, w in zip(ys, want):
        assert torch.equal(y, w)
    spblas.destroy(A)
