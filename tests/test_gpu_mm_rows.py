"""Row-major dense-block products on rows of few elements (a lane group per row) and of many (element stream): every width of
load, lane group and remainder on both sides of the line between the two."""
import numpy as np
import pytest
import torch

import oracle
from alsparse_b200 import capi, spblas, synth
from gpu_util import TORCH, make_handle
from helpers import assert_rows_close, mm_scale

pytestmark = pytest.mark.gpu


def product(kind, A, X, columns, ldx, alpha, beta, Y, ldy):
    st = spblas.mm(kind, 0, alpha, A, spblas.descr(), capi.ROW_MAJOR, X, columns, ldx, beta, Y, ldy)
    assert st == capi.SUCCESS, spblas.last_error()
    torch.cuda.synchronize()


def lengths(shape):
    rng = np.random.default_rng(9)
    if shape == "short":  # empty rows among them, and one wave of them only
        return rng.integers(0, 6, 4001).astype(np.int32)
    if shape == "short, more rows":
        return rng.integers(0, 4, 50021).astype(np.int32)
    if shape == "short, one of 70":  # uneven, and short enough to be walked beside the others
        lens = rng.integers(0, 3, 900001).astype(np.int32)
        lens[3] = 70
        return lens
    return rng.integers(28, 33, 3001).astype(np.int32)  # "even"


@pytest.mark.parametrize("kind", ["s", "d"])
@pytest.mark.parametrize("shape", ["short", "short, more rows", "short, one of 70", "even"])
def test_widths_and_remainders(kind, shape):
    m = synth.from_lengths(kind, 21, lengths(shape), 2500)
    A = make_handle(kind, m)
    widths = ((12, 0, 0.5), (33, 1, 0.0)) if m.nrows > 100000 else \
        ((9, 0, 0.5), (10, 0, 0.0), (12, 4, 0.5), (15, 0, 0.5), (20, 0, 0.0), (34, 0, 0.5), (40, 1, 0.5), (64, 0, 0.0), (132, 0, 0.5))
    for columns, pad, beta in widths:
        ld = columns + pad
        X, Y0 = synth.vector(kind, 5, 3, m.cols * ld), synth.vector(kind, 5, 4, m.nrows * ld)
        ref = oracle.gemm(kind, "row", m.rows_start, m.rows_end, m.col, m.val, 1.5, X, columns, ld, beta, Y0.copy(), ld)
        dX, dY = torch.from_numpy(X).cuda(), torch.from_numpy(Y0).cuda()
        product(kind, A, dX, columns, ld, 1.5, beta, dY, ld)
        scale = mm_scale(m.ptr, m.col, m.val, X, columns, ld, 1.5, beta, Y0, ld)
        Y = dY.cpu().numpy().reshape(m.nrows, ld)
        assert np.array_equal(Y[:, columns:], Y0.reshape(m.nrows, ld)[:, columns:]), "padding written"
        assert_rows_close(kind, Y[:, :columns].reshape(-1), ref.reshape(m.nrows, ld)[:, :columns].reshape(-1), scale.reshape(-1),
                          f"{columns} columns")
    spblas.destroy(A)


@pytest.mark.parametrize("rows", [300, 20000, 60000])
@pytest.mark.parametrize("columns", [12, 24, 33])
def test_short_rows_are_summed_element_after_element(rows, columns):
    """Told apart by rounding: 2^24 + 1 + 1 + 1 - 2^24 is 0 in single precision in this order, and 2 in pairs."""
    m = synth.Csr(rows, 5, 0, np.arange(0, 5 * rows + 1, 5, dtype=np.int32), np.tile(np.arange(5, dtype=np.int32), rows),
                  np.tile(np.array([2.0 ** 24, 1, 1, 1, -2.0 ** 24], np.float32), rows))
    A = make_handle("s", m)
    X, Y = torch.ones(5, columns, device="cuda"), torch.ones(rows, columns, device="cuda")
    product("s", A, X, columns, columns, 1.0, 1.0, Y, columns)
    assert bool((Y == 1.0).all())
    spblas.destroy(A)


@pytest.mark.parametrize("kind", ["s", "d"])
def test_host_operands_in_row_windows(kind):
    """Short rows in the eight windows of a product with host operands."""
    columns = 40
    m = synth.from_lengths(kind, 21, np.random.default_rng(1).integers(0, 4, 250001).astype(np.int32), 1200)
    A = make_handle(kind, m)
    X, Y0 = synth.vector(kind, 5, 3, m.cols * columns), synth.vector(kind, 5, 4, m.nrows * columns)
    dX, dY, Y = torch.from_numpy(X).cuda(), torch.from_numpy(Y0).cuda(), Y0.copy()
    product(kind, A, dX, columns, columns, 1.5, 0.5, dY, columns)
    product(kind, A, X, columns, columns, 1.5, 0.5, Y, columns)
    assert torch.equal(torch.from_numpy(Y).to(TORCH[kind]), dY.cpu())
    spblas.destroy(A)
