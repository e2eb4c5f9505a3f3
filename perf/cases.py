"""The workloads by which changes to the library are timed.

A case is a dict of plain values: a matrix (shape and distribution of the stored elements), an operation and where
its operands live.  ``prepare`` makes the matrix handle and the vectors a program holds before the call, ``run`` makes
one call through ``alsparse_b200.spblas`` (the C entry points of the same names), ``work`` counts what the operation
cannot do without.  Row lengths, columns and values follow the distributions of the repository's generators
(``alsparse_b200/synth``), drawn on the device so that a large matrix takes a fraction of a second.
"""
import math
import weakref

import numpy as np
import torch

from alsparse_b200 import capi, spblas

NUMPY = {"s": np.float32, "d": np.float64}
TORCH = {"s": torch.float32, "d": torch.float64}
BYTES = {"s": 4, "d": 8}

# Row lengths of the power-law matrices: P(n) ~ n^-1.8 for 1 <= n <= the longest row.
ZIPF_S, ZIPF_MAX = 1.8, 200000


def _mv(name, matrix, kind, rows, mean, **more):
    case = {"op": "mv", "matrix": matrix, "kind": kind, "rows": rows, "cols": more.pop("cols", rows), "mean": mean,
            "trans": False, "where": "device", "alpha": 1.0, "beta": 0.0}
    return dict({"name": name} if name else {}, **{**case, **more})


def _mm(name, matrix, kind, rows, mean, columns, layout, **more):
    return dict(_mv(name, matrix, kind, rows, mean, **more), op="mm", columns=columns, layout=layout)


def listed():
    return [
        # The smallest calls.  A product of a few thousand elements inside a solver whose vectors stay on the device:
        # what counts is what one call costs the host and the device.
        _mv("mv_tiny_device", "poisson", "s", 1000, 5),
        # ... and the same product called as the CPU library was: host vectors in, host vector complete on return.
        _mv("mv_tiny_host", "poisson", "d", 1500, 7, where="host", alpha=2.0, beta=2.0),
        # Stencils of structured grids, the inner product of an iterative solver: an ordinary grid whose matrix fits
        # L2, and the benchmark's large one that has to stream from HBM.
        _mv("mv_stencil_mid", "stencil27", "d", 61 ** 3, 27, beta=0.5),
        _mv("mv_stencil_large", "stencil27", "d", 160 ** 3, 27),
        # Unstructured columns, rows of one length (finite elements in a poor ordering, k-nearest-neighbour graphs).
        _mv("mv_uniform_large", "uniform", "s", 1 << 23, 16, alpha=1.5, beta=0.5),
        # Graph matrices: half the rows hold one or two elements, a few hundred hold 200,000.
        _mv("mv_powerlaw", "powerlaw", "d", 1 << 21, 37),
        # The product by the transpose of a rectangular matrix of ragged size (least squares: every step multiplies by
        # A and by A^T); the transpose is formed by the library at the first call and stays with the handle.
        _mv("mv_transposed", "poisson", "d", 1500007, 12, cols=700001, trans=True, alpha=-1.0, beta=1.0),
        # Host vectors of a large matrix, page-locked as a program that cares would have them: copies and kernel overlap.
        _mv("mv_host_large", "uniform", "s", 1 << 22, 16, where="pinned", alpha=1.5, beta=0.5),
        # Dense blocks.  Feature propagation: 64 features, and 24 features over a power-law graph.
        _mm("mm_row_64", "poisson", "s", 1 << 20, 32, 64, "row"),
        _mm("mm_row_powerlaw_24", "powerlaw", "s", 400009, 37, 24, "row", beta=1.0),
        # A block solver with several right-hand sides, stored one after the other.
        _mm("mm_col_stencil_6", "stencil27", "d", 80 ** 3, 27, 6, "col"),
        # Assembly: unordered triples to a handle that can be multiplied by, and its CSR arrays.  Programs whose
        # coefficients change do this at every step.
        _mv("assemble", "poisson", "d", 250007, 16, op="assemble", where="host"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["small", "stencil", "uniform", "powerlaw", "transposed", "host", "mm_row", "mm_skew", "mm_col",
                       "assemble"])
    kind = rng.choice("sd")
    scale = rng.choice([dict(alpha=1.0, beta=0.0), dict(alpha=1.5, beta=0.5), dict(alpha=-1.0, beta=1.0)])
    if what == "small":
        rows = _log(rng, 500, 30000)
        return _mv(None, rng.choice(["poisson", "powerlaw", "uniform"]), kind, rows, rng.randint(3, 20),
                   where=rng.choice(["device", "host"]), **scale)
    if what == "stencil":
        return _mv(None, "stencil27", kind, _log(rng, 20, 155) ** 3, 27, **scale)
    if what == "uniform":
        mean = rng.randint(4, 40)
        return _mv(None, rng.choice(["uniform", "poisson"]), kind, _log(rng, 30000, min(1 << 23, (1 << 26) // mean)), mean,
                   **scale)
    if what == "powerlaw":
        return _mv(None, "powerlaw", kind, _log(rng, 30000, 1 << 21), 37, **scale)
    if what == "transposed":
        mean = rng.randint(4, 24)
        return _mv(None, rng.choice(["uniform", "poisson", "powerlaw"]), kind, _log(rng, 20000, 1500000), mean,
                   cols=_log(rng, 20000, 1500000), trans=True, **scale)
    if what == "host":
        return _mv(None, rng.choice(["uniform", "poisson"]), kind, _log(rng, 30000, 1 << 22), rng.randint(4, 16),
                   where=rng.choice(["host", "pinned"]), **scale)
    if what == "mm_row":
        columns = _log(rng, 2, 128)
        return _mm(None, rng.choice(["uniform", "poisson", "stencil27"]), kind, _log(rng, 20, 78) ** 3, 27, columns, "row",
                   **scale)
    if what == "mm_skew":
        return _mm(None, "powerlaw", kind, _log(rng, 20000, 400009), 37, _log(rng, 2, 64), rng.choice(["row", "col"]),
                   **scale)
    if what == "mm_col":
        return _mm(None, rng.choice(["poisson", "stencil27"]), kind, _log(rng, 20, 80) ** 3, 27, _log(rng, 2, 32), "col",
                   **scale)
    return _mv(None, rng.choice(["poisson", "uniform"]), kind, _log(rng, 4000, 250007), 16, op="assemble", where="host")


# ---- matrices ----------------------------------------------------------------------------------------------------


def _zipf_lengths(rows, cols, gen):
    longest = min(ZIPF_MAX, max(2, cols // 8))
    cdf = torch.arange(1, longest + 1, device="cuda", dtype=torch.float64).pow_(-ZIPF_S).cumsum_(0)
    at = torch.rand(rows, generator=gen, device="cuda", dtype=torch.float64) * cdf[-1]
    return torch.searchsorted(cdf, at).clamp_(max=longest - 1) + 1


def _pattern(case, gen):
    """(row of every stored element or None, row offsets, columns) on the device, ordered by row and column."""
    rows, cols = case["rows"], case["cols"]
    if case["matrix"] == "stencil27":
        n = round(rows ** (1 / 3))
        at = torch.arange(rows, device="cuda", dtype=torch.int32)
        z, y, x = at // (n * n), at // n % n, at % n
        step = [(dz, dy, dx) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
        inside = torch.stack([(z + dz >= 0) & (z + dz < n) & (y + dy >= 0) & (y + dy < n) & (x + dx >= 0) & (x + dx < n)
                              for dz, dy, dx in step], 1)
        shift = torch.tensor([(dz * n + dy) * n + dx for dz, dy, dx in step], device="cuda", dtype=torch.int32)
        col = (at[:, None] + shift)[inside]
        lens = inside.sum(1)
    else:
        if case["matrix"] == "uniform":
            lens = torch.full((rows,), case["mean"], device="cuda", dtype=torch.int64)
        elif case["matrix"] == "poisson":
            lens = torch.poisson(torch.full((rows,), float(case["mean"]), device="cuda"), generator=gen).long()
        else:
            lens = _zipf_lengths(rows, cols, gen)
        key = torch.repeat_interleave(torch.arange(rows, device="cuda"), lens) << 32
        key |= torch.randint(cols, key.shape, generator=gen, device="cuda")
        key = torch.unique_consecutive(key.sort().values)  # the few columns drawn twice for one row are stored once
        lens = torch.bincount(key >> 32, minlength=rows)
        col = (key & 0xffffffff).int()
    ptr = torch.zeros(rows + 1, device="cuda", dtype=torch.int32)
    ptr[1:] = lens.cumsum(0)
    return lens, ptr, col


def _values(case, lens, ptr, col, gen):
    if case["matrix"] == "stencil27":
        row = torch.repeat_interleave(torch.arange(case["rows"], device="cuda", dtype=torch.int32), lens)
        return torch.where(col == row, 26.0, -1.0).to(TORCH[case["kind"]])
    return _uniform(col.numel(), case, gen)


def _uniform(n, case, gen):
    return torch.rand(n, generator=gen, device="cuda", dtype=TORCH[case["kind"]]).mul_(2).sub_(1)


class State:
    """A matrix handle (released with the state) and the operands of the call."""

    def __init__(self, case):
        self.case, self.kind = case, case["kind"]
        self.descr = spblas.descr(capi.GENERAL)
        self.operation = capi.TRANSPOSE if case["trans"] else capi.NON_TRANSPOSE
        self.release = lambda: None

    def hold(self, handle):
        self.handle = handle
        self.release = weakref.finalize(self, spblas.destroy, handle)


class Borrowed(np.ndarray):
    """An array inside a handle: keeps the state that holds the handle."""

    @classmethod
    def of(cls, array, state):
        array = array.view(cls)
        array.state = state
        return array


def _done(status):
    if status != capi.SUCCESS:
        raise RuntimeError("%s %s" % (capi.STATUS_NAMES[status], spblas.last_error()))


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    s = State(case)
    rows, cols = case["rows"], case["cols"]
    lens, ptr, col = _pattern(case, gen)
    val = _values(case, lens, ptr, col, gen)
    if case["op"] == "assemble":
        row = torch.repeat_interleave(torch.arange(rows, device="cuda", dtype=torch.int32), lens)
        order = torch.rand(col.numel(), generator=gen, device="cuda", dtype=torch.float64).argsort()[:_elements(case)]
        assert len(order) == _elements(case)
        s.triples = [t[order].cpu().numpy() for t in (row, col, val)]
        return s
    ptr = ptr.cpu().numpy()
    status, handle = spblas.create_csr(case["kind"], capi.BASE_ZERO, rows, cols, ptr[:-1], ptr[1:], col.cpu().numpy(),
                                       val.cpu().numpy())
    _done(status)
    s.hold(handle)
    n_in, n_out = (rows, cols) if case["trans"] else (cols, rows)
    width = case.get("columns", 1)
    s.x, s.y = _uniform(n_in * width, case, gen), _uniform(n_out * width, case, gen)
    if case["op"] == "mm":
        row_major = case["layout"] == "row"
        s.layout = capi.ROW_MAJOR if row_major else capi.COLUMN_MAJOR
        s.ldx, s.ldy = (width, width) if row_major else (n_in, n_out)
    if case["where"] == "host":
        s.x, s.y = s.x.cpu().numpy(), s.y.cpu().numpy()
    elif case["where"] == "pinned":
        s.x, s.y = s.x.cpu().pin_memory(), s.y.cpu().pin_memory()
    return s


def run(s):
    case = s.case
    if case["op"] == "mv":
        _done(spblas.mv(s.kind, s.operation, case["alpha"], s.handle, s.descr, s.x, case["beta"], s.y))
        return s.y
    if case["op"] == "mm":
        _done(spblas.mm(s.kind, s.operation, case["alpha"], s.handle, s.descr, s.layout, s.x, case["columns"], s.ldx,
                        case["beta"], s.y, s.ldy))
        return s.y
    s.release()  # the handle of the step before
    row, col, val = s.triples
    status, coo = spblas.create_coo(s.kind, capi.BASE_ZERO, case["rows"], case["cols"], len(val), row, col, val)
    _done(status)
    status, handle = spblas.convert_csr(coo)
    spblas.destroy(coo)
    _done(status)
    s.hold(handle)
    status, _, _, _, *arrays = spblas.export_csr(s.kind, handle)
    _done(status)
    return [Borrowed.of(a, s) for a in arrays]


# ---- what an operation cannot do without ---------------------------------------------------------------------------


def _elements(case):
    """Stored elements, up to the spread of the random row lengths."""
    rows, cols = case["rows"], case["cols"]
    if case["matrix"] == "stencil27":
        return (3 * round(rows ** (1 / 3)) - 2) ** 3
    if case["matrix"] == "powerlaw":
        longest = min(ZIPF_MAX, max(2, cols // 8))
        n = np.arange(1, longest + 1, dtype=np.float64)
        return int(rows * (n ** (1 - ZIPF_S)).sum() / (n ** -ZIPF_S).sum())
    if case["op"] == "assemble":  # always the same number of triples: a little less than the random lengths add up to
        return rows * case["mean"] * 15 // 16
    return rows * case["mean"]


def work(case):
    nnz, rows, cols, size = _elements(case), case["rows"], case["cols"], BYTES[case["kind"]]
    csr = nnz * (size + 4) + (rows + 1) * 4
    if case["op"] == "assemble":
        return {"bytes": nnz * (size + 8) + csr, "flops": 0}
    width = case.get("columns", 1)
    n_in, n_out = (rows, cols) if case["trans"] else (cols, rows)
    return {"bytes": csr + (n_in + n_out * (2 if case["beta"] else 1)) * width * size, "flops": 2 * nnz * width}


def tolerance(case):
    # an assembly moves values and counts; a product is a sum of products, formed in any order
    if case["op"] == "assemble":
        return "exact"
    return {"rel": 1e-5 if case["kind"] == "s" else 1e-13}
