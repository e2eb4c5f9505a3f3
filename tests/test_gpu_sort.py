"""Triples to CSR at the edges of the device sort: tile remainders, 32- and 64-bit keys, one pass and many, against the
oracle's conversion (bit-exact, equal pairs in input order), and the recycled memory behind repeated conversions."""
import numpy as np
import pytest

import oracle
from alsparse_b200 import capi, spblas
from gpu_util import download
from helpers import NP

pytestmark = pytest.mark.gpu

TILE = 4096  # elements per block of the sort; conversions of 2 * TILE elements and more run on the device


@pytest.mark.parametrize("kind", ["s", "d"])
@pytest.mark.parametrize("rows,cols", [(2, 1), (3, 700), (65536, 65536), (65537, 65536), (100003, 200003)])
@pytest.mark.parametrize("nnz", [2 * TILE, 2 * TILE + 1, 5 * TILE - 1, 70001])
def test_conversion_at_tile_and_key_edges(kind, rows, cols, nnz):
    rng = np.random.default_rng(nnz + rows)
    ri, ci = rng.integers(rows, size=nnz, dtype=np.int32), rng.integers(cols, size=nnz, dtype=np.int32)
    v = rng.uniform(-1, 1, nnz).astype(NP[kind])
    ri[-1], ci[-1] = rows - 1, cols - 1
    st, coo = spblas.create_coo(kind, capi.BASE_ZERO, rows, cols, nnz, ri, ci, v)
    assert st == capi.SUCCESS
    st, A = spblas.convert_csr(coo)
    assert st == capi.SUCCESS, spblas.last_error()
    optr, ocol, oval = oracle.coo_to_csr(kind, 0, rows, ri, ci, v)
    st, _, _, _, start, end, col, val = spblas.export_csr(kind, A)
    assert st == capi.SUCCESS
    assert (start == optr[:-1]).all() and (end == optr[1:]).all() and (col == ocol).all() and (val == oval).all()
    import torch
    st, d_ptr, d_col, d_val = spblas.device_csr(A)   # the device copy is made separately from the host arrays
    assert (download(d_ptr, rows + 1, torch.int32) == optr).all() and (download(d_col, nnz, torch.int32) == ocol).all()
    assert (download(d_val, nnz, torch.float32 if kind == "s" else torch.float64) == oval).all()
    for h in (coo, A):
        spblas.destroy(h)


def test_repeated_conversions_do_not_share_memory():
    # two live handles and a stream of short-lived ones of changing size through the recycled blocks
    rng = np.random.default_rng(5)
    live = []
    for step, nnz in enumerate([300000, 20000, 300001, 9000, 290000, 310000]):
        rows = 5000 + step
        ri, ci = rng.integers(rows, size=nnz, dtype=np.int32), rng.integers(rows, size=nnz, dtype=np.int32)
        v = rng.uniform(-1, 1, nnz)
        st, coo = spblas.create_coo("d", capi.BASE_ONE, rows, rows, nnz, ri + 1, ci + 1, v)
        st2, A = spblas.convert_csr(coo)
        assert st == st2 == capi.SUCCESS
        spblas.destroy(coo)
        live.append((A, oracle.coo_to_csr("d", 0, rows, ri, ci, v)))
        if len(live) > 2:
            spblas.destroy(live.pop(0)[0])
        for A, (optr, ocol, oval) in live:
            st, _, _, _, start, end, col, val = spblas.export_csr("d", A)
            assert (end == optr[1:]).all() and (col == ocol).all() and (val == oval).all()
            x, y = np.ones(len(optr) - 1), np.zeros(len(optr) - 1)
            assert spblas.mv("d", 0, 1.0, A, spblas.descr(), x, 0.0, y) == capi.SUCCESS
            want = np.add.reduceat(np.append(oval, 0.0), optr[:-1]) * (np.diff(optr) > 0)
            # sums of at most 100-odd terms below one: well inside 1e-12 of the sum of magnitudes
            assert (np.abs(y - want) <= 1e-12 * (1 + np.diff(optr))).all()
    for A, _ in live:
        spblas.destroy(A)
