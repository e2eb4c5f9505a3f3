"""Row tiles around 48 KB of shared memory, the most a launch may use before its limit is raised.  The limit stays raised
for the rest of the process, so the sizes are taken in ascending order in a process of their own."""
import os
import subprocess
import sys

import pytest

from helpers import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import sys
import numpy as np
import torch
from alsparse_b200 import capi, spblas, synth

kind, call = sys.argv[1:3]
dtype, size = (np.float32, 4) if kind == "s" else (np.float64, 8)
tol = 1e-5 if kind == "s" else 1e-12
most = (48 << 10) // (size + 4)  # elements of a tile whose values and columns take 48 KB
ran = 0
for span in range(most - 48, most + 52, 4):
    rows = 24  # one tile: its elements are all the matrix has
    lens = np.full(rows, span // rows, np.int64)
    lens[:span % rows] += 1
    ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = np.concatenate([r + np.arange(n) for r, n in enumerate(lens)]).astype(np.int32)
    cols = int(col.max()) + 1
    val = synth.vector(kind, 1, 1, span)
    st, A = spblas.create_csr(kind, 0, rows, cols, ptr[:-1], ptr[1:], col, val)
    assert st == capi.SUCCESS, spblas.last_error()
    assert spblas.mat_info(A)[1].algorithm == capi.ALG_ROWTILE
    x = synth.vector(kind, 1, 2, 3 * cols).reshape(3, cols)
    dense = np.zeros((rows, cols))
    dense[np.repeat(np.arange(rows), lens), col] = val
    dx, dy = torch.from_numpy(x.copy()).cuda(), torch.ones(3, rows, dtype=torch.float32 if kind == "s" else torch.float64, device="cuda")
    n = 1 if call == "mv" else 3
    for beta in (0.0, 0.5):
        before = dy.cpu().numpy().astype(float)
        if call == "mv":
            st = spblas.mv(kind, 0, 1.5, A, spblas.descr(), dx, beta, dy)
        else:
            st = spblas.mm(kind, 0, 1.5, A, spblas.descr(), capi.COLUMN_MAJOR, dx, 3, cols, beta, dy, rows)
        assert st == capi.SUCCESS, (span, capi.STATUS_NAMES[st], spblas.last_error())
        torch.cuda.synchronize()
        want = 1.5 * x[:n].astype(float) @ dense.T + beta * before[:n]
        scale = 1.5 * np.abs(x[:n]).astype(float) @ np.abs(dense).T + np.abs(beta * before[:n])
        assert (np.abs(dy.cpu().numpy()[:n] - want) <= tol * scale).all(), span
        ran += 1
    spblas.destroy(A)
print("ran", ran)
"""


@pytest.mark.parametrize("kind", ["s", "d"])
@pytest.mark.parametrize("call", ["mv", "mm"])
def test_tiles_around_the_launch_limit(kind, call):
    out = subprocess.run([sys.executable, "-c", CHILD, kind, call], cwd=ROOT, capture_output=True, text=True, timeout=300,
                         env=dict(os.environ, PYTHONPATH=ROOT))
    assert out.returncode == 0, out.stdout + out.stderr
    assert "ran 50" in out.stdout
