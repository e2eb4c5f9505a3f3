"""Copies by all cores: create_coo copies its three arrays into the handle."""
import ctypes as C
import os

import numpy as np

from alsparse_b200 import capi, spblas


class CooRecord(C.Structure):
    """The leading members of spmat_coo_{s,d}_t."""
    _fields_ = [("values", C.c_void_p), ("row_indx", C.c_void_p), ("col_indx", C.c_void_p)]


def threads():
    return set(os.listdir("/proc/self/task"))


def copied(nnz):
    ri, ci = np.arange(nnz, dtype=np.int32), np.arange(nnz, dtype=np.int32)[::-1].copy()
    v = np.arange(nnz, dtype=np.float64)
    st, A = spblas.create_coo("d", capi.BASE_ZERO, nnz, nnz, nnz, ri, ci, v)
    assert st == capi.SUCCESS
    st = spblas.destroy(A)
    assert st == capi.SUCCESS


def test_copies_of_changing_size_keep_their_threads():
    """Large pieces are copied by the whole team, smaller ones by a few of it: none is ended and started again."""
    copied(1 << 20)
    before = threads()
    for nnz in (1 << 20, 50000, 1 << 20, 70000, 100, 1 << 20, 40000, 300000, 1 << 20):
        copied(nnz)
    assert threads() == before


def test_contents_at_the_edges_of_pieces():
    """Sizes around those at which one more thread takes part, from aligned and unaligned sources."""
    piece = (128 << 10) // 8
    for nnz in [1, 7, piece - 1, piece, 2 * piece - 1, 2 * piece, 2 * piece + 1, 5 * piece + 13, 40 * piece + 3]:
        for shift in (0, 1):
            ri, ci = (np.arange(nnz + 1, dtype=np.int32)[shift:shift + nnz] for _ in range(2))
            v = np.random.default_rng(nnz).random(nnz + 1)[shift:shift + nnz]
            st, A = spblas.create_coo("d", capi.BASE_ZERO, nnz + 1, nnz + 1, nnz, ri, ci, v)
            assert st == capi.SUCCESS
            record = C.cast(C.cast(A, C.POINTER(capi.Matrix)).contents.mat, C.POINTER(CooRecord)).contents
            for pointer, want in ((record.row_indx, ri), (record.col_indx, ci), (record.values, v)):
                kind = C.c_int32 if want.dtype == np.int32 else C.c_double
                got = np.ctypeslib.as_array(C.cast(pointer, C.POINTER(kind)), shape=(nnz,))
                assert np.array_equal(got, want)
            spblas.destroy(A)
