"""Column-major dense-block product of a banded matrix (a lane per row, no transposes): edges of its row tiles and of its
groups of dense columns."""
import numpy as np
import pytest
import torch

import oracle
from alsparse_b200 import capi, spblas, synth
from gpu_util import make_handle
from helpers import assert_rows_close, mm_scale

pytestmark = pytest.mark.gpu


def banded(kind, rows, offsets, empty=None):
    """Row r holds the columns r + offsets that lie inside the matrix; the rows of `empty` hold none."""
    col = np.arange(rows)[:, None] + np.asarray(offsets)[None, :]
    inside = (col >= 0) & (col < rows)
    if empty is not None:
        inside[empty] = False
    ptr = np.concatenate([[0], np.cumsum(inside.sum(1))]).astype(np.int32)
    return synth.Csr(rows, rows, 0, ptr, col[inside].astype(np.int32), synth.vector(kind, 3, 1, int(ptr[-1])))


@pytest.mark.parametrize("kind", ["s", "d"])
@pytest.mark.parametrize("make", [lambda k: synth.stencil27(k, 9), lambda k: banded(k, 33, (-1, 0, 1)),
                                  lambda k: banded(k, 1000, (-40, -1, 0, 1, 40)), lambda k: banded(k, 31, range(0, 8)),
                                  lambda k: banded(k, 4097, (-2, 5)),
                                  lambda k: banded(k, 2000, (-1, 0, 1, 7), slice(320, 400)),  # whole tiles and a part of one
                                  lambda k: banded(k, 1001, (0, 1, 2), slice(990, None))])
def test_tiles_and_column_groups(kind, make):
    m = make(kind)
    A = make_handle(kind, m)
    for columns, pad, alpha, beta in ((1, 0, 1.0, 0.0), (2, 3, 1.5, 0.5), (3, 0, -1.0, 1.0), (4, 1, 1.5, 0.5), (5, 0, 1.0, 0.0),
                                      (8, 2, 1.5, 0.5), (9, 0, 1.5, 0.5), (19, 1, 1.0, 0.0), (33, 0, 1.5, 0.5)):
        ldx, ldy = m.cols + pad, m.nrows + 2 * pad
        X, Y0 = synth.vector(kind, 5, 3, columns * ldx), synth.vector(kind, 5, 4, columns * ldy)
        ref = oracle.gemm(kind, "col", m.rows_start, m.rows_end, m.col, m.val, alpha, X, columns, ldx, beta, Y0.copy(), ldy)
        dX, dY = torch.from_numpy(X).cuda(), torch.from_numpy(Y0).cuda()
        before = spblas.launch_count()
        assert spblas.mm(kind, 0, alpha, A, spblas.descr(), capi.COLUMN_MAJOR, dX, columns, ldx, beta, dY, ldy) == capi.SUCCESS
        torch.cuda.synchronize()
        assert spblas.launch_count() == before + 1  # one kernel: this path
        Y = dY.cpu().numpy().reshape(columns, ldy)
        assert np.array_equal(Y[:, m.nrows:], Y0.reshape(columns, ldy)[:, m.nrows:]), "padding written"
        rows_of = lambda v, ld, n: np.ascontiguousarray(v.reshape(columns, ld)[:, :n].T).reshape(-1)
        scale = mm_scale(m.ptr, m.col, m.val, rows_of(X, ldx, m.cols), columns, columns, alpha, beta,
                         rows_of(Y0, ldy, m.nrows), columns)
        assert_rows_close(kind, rows_of(Y, ldy, m.nrows), rows_of(ref, ldy, m.nrows), scale.reshape(-1), f"{columns} columns")
    spblas.destroy(A)
