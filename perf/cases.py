"""Performance cases of the B200 SpGEMM backend, as a user's program runs them.

Every case is one call sequence through the library's public entry points
(the ctypes binding rvsp_b200 of include/rv_sparse.h and include/rvsp_cuda.h)
on seeded synthetic operands made on the GPU. Kinds:

* oneshot   C = A * B, device CSR in and out (rvsp_cuda_spgemm_f32), exact or learned
* host      C = A * A, host CSR in and out (rvsp_spgemm_csr)
* first     a descriptor's first product: work estimation, then the compute that fills C
* reuse     a descriptor's later products: new values on the structure it already filled
* batched   many independent products in one call (rvsp_cuda_spgemm_batched_f32)
* f64, i8   the FP64 and INT8 -> INT32 products (rvsp_cuda_spgemm_f64 / _i8)
* coo       COO with repeats -> canonical CSR (rvsp_cuda_coo_to_csr)

Matrices: uniform (a fixed number of distinct uniform columns per row),
poisson (5-point Laplacian of a grid), rmat (R-MAT graph, quadrant
probabilities .57 .19 .19 .05, repeats merged, optionally one row panel of at
most 2^31 - 1 products), tall (geometric row lengths times a power-law B).
A case fixes the pattern of its matrices ("pattern" seeds it); a seed gives
the values, and the order of a COO list.
"""

import ctypes as C
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "rv-sparse_b200"))
import rvsp_b200 as rv  # noqa: E402

INT32_MAX = 2 ** 31 - 1


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # the smallest calls: a coarse-grid or test-sized product, all latency
        {"name": "uniform_512_exact", "kind": "oneshot", "algo": "exact", "matrix": "uniform",
         "rows": 512, "cols": 512, "per_row": 16, "pattern": 0},
        # an ordinary one-shot product of a small uniform matrix (benchmark's plain 4096^2)
        {"name": "uniform_4096_exact", "kind": "oneshot", "algo": "exact", "matrix": "uniform",
         "rows": 4096, "cols": 4096, "per_row": 16, "pattern": 0},
        # the same through the reference's own C API on host arrays, as code
        # ported from the reference calls it
        {"name": "uniform_4096_host", "kind": "host", "algo": "exact", "matrix": "uniform",
         "rows": 4096, "cols": 4096, "per_row": 16, "pattern": 0},
        # a large sparse product with short, uneven rows (a restriction or a
        # feature join): tall A times power-law B
        {"name": "tall_2m_exact", "kind": "oneshot", "algo": "exact", "matrix": "tall",
         "rows": 2000000, "cols": 100000, "pattern": 0},
        # a solver's setup: structure analysis and first product of a stencil
        # matrix, ragged grid
        {"name": "poisson_1023x1025_first", "kind": "first", "algo": "exact", "matrix": "poisson",
         "nx": 1023, "ny": 1025, "pattern": 0},
        # a solver's every later step: new values on that structure
        {"name": "poisson_1024_reuse", "kind": "reuse", "algo": "exact", "matrix": "poisson",
         "nx": 1024, "ny": 1024, "pattern": 0},
        # the same for a graph, whose rows run from empty to very long
        {"name": "rmat16_reuse", "kind": "reuse", "algo": "exact", "matrix": "rmat", "scale": 16,
         "edge_factor": 16, "panel": -1, "pattern": 0},
        # a whole graph product (two-hop neighbours), exact sizing
        {"name": "rmat17_exact", "kind": "oneshot", "algo": "exact", "matrix": "rmat", "scale": 17,
         "edge_factor": 16, "panel": -1, "pattern": 0},
        # the headline workload: one row panel of the 2^20 graph's product,
        # learned sizing, the largest call one int32 C allows
        {"name": "rmat20_panel_learned", "kind": "oneshot", "algo": "learned", "matrix": "rmat",
         "scale": 20, "edge_factor": 16, "panel": 4, "pattern": 0},
        # many uneven products at once (blocks of a domain decomposition)
        {"name": "batched_128_learned", "kind": "batched", "algo": "learned", "count": 128,
         "lo": 256, "hi": 65536, "pattern": 0},
        # the reference's FP64 product
        {"name": "uniform_100k_f64", "kind": "f64", "matrix": "uniform", "rows": 100000,
         "cols": 100000, "per_row": 12, "pattern": 0},
        # loading: an edge list with repeats to canonical CSR
        {"name": "coo_rmat20", "kind": "coo", "scale": 20, "edge_factor": 16,
         "symmetric": False, "pattern": 0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["oneshot", "oneshot", "oneshot", "host", "first", "reuse", "batched",
                       "f64", "i8", "coo"])
    c = {"kind": kind, "pattern": rng.randrange(1 << 30)}
    if kind == "coo":
        return c | {"scale": rng.randint(12, 20), "edge_factor": rng.randint(5, 16),
                    "symmetric": rng.random() < 0.3}
    if kind in ("oneshot", "host", "batched"):
        c["algo"] = rng.choice(["exact", "learned"])
    elif kind in ("first", "reuse"):
        c["algo"] = "exact"
    if kind == "batched":
        return c | {"count": _log(rng, 8, 128), "lo": 256, "hi": 65536}
    matrix = "uniform" if kind in ("host", "f64", "i8") else rng.choice(
        ["uniform", "poisson", "rmat", "tall" if kind == "oneshot" else "rmat"])
    c["matrix"] = matrix
    if matrix == "uniform":
        n = _log(rng, 300, 20000 if kind == "host" else 200000)
        c |= {"rows": n, "cols": max(200, int(n * rng.uniform(0.5, 1.0))),
              "per_row": rng.randint(3, 24)}
    elif matrix == "poisson":
        c |= {"nx": _log(rng, 60, 1100), "ny": _log(rng, 60, 1100)}
    elif matrix == "rmat":
        c |= {"scale": rng.randint(11, 17 if kind == "oneshot" else 16),
              "edge_factor": rng.randint(6, 16), "panel": -1}
    else:
        c |= {"rows": _log(rng, 60000, 2000000), "cols": _log(rng, 20000, 150000)}
    return c


# ---------------------------------------------------------------------------
# operands
# ---------------------------------------------------------------------------

class Csr:
    """A device CSR matrix. A row panel's row pointer is a view into the whole
    one, so its offsets index the whole column and value arrays."""

    def __init__(self, rows, cols, nnz, row_ptr, col_idx, values):
        self.rows, self.cols, self.nnz = rows, cols, nnz
        self.row_ptr, self.col_idx, self.values = row_ptr, col_idx, values

    def struct(self):
        return rv.csr_struct(self.rows, self.cols, self.nnz, self.row_ptr, self.col_idx,
                             self.values)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _values(n, g, kind):
    if kind == "i8":
        return torch.randint(-127, 128, (n,), generator=g, device="cuda").to(torch.int8)
    dt = torch.float64 if kind == "f64" else torch.float32
    return torch.rand(n, generator=g, device="cuda", dtype=dt) * 2 - 1


def _from_keys(rows, cols, keys, values=None):
    r = torch.div(keys, cols, rounding_mode="floor")
    rp = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(torch.bincount(r, minlength=rows), 0)
    ci = (keys - r * cols).to(torch.int32)
    return Csr(rows, cols, int(keys.numel()), rp.to(torch.int32), ci, values)


def _uniform(rows, cols, per_row, g):
    extra = per_row + 8  # enough candidates that per_row of them are distinct
    c = torch.randint(0, cols, (rows, extra), generator=g, device="cuda").sort(1).values
    pick = torch.rand(rows, extra, generator=g, device="cuda")
    pick[:, 1:][c[:, 1:] == c[:, :-1]] = 2.0  # repeats go last
    keep = pick.argsort(1)[:, :per_row]
    c, pick = c.gather(1, keep), pick.gather(1, keep)
    r = torch.arange(rows, device="cuda")[:, None]
    keys = (r * cols + c)[pick < 2.0].sort().values
    return _from_keys(rows, cols, keys)


def _poisson(nx, ny):
    n = nx * ny
    idx = torch.arange(n, device="cuda")
    i, j = torch.div(idx, ny, rounding_mode="floor"), idx % ny
    keys = []
    for di, dj in ((-1, 0), (0, -1), (0, 0), (0, 1), (1, 0)):
        ok = (i + di >= 0) & (i + di < nx) & (j + dj >= 0) & (j + dj < ny)
        keys.append((idx * n + idx + di * ny + dj)[ok])
    keys = torch.cat(keys).sort().values
    diag = torch.div(keys, n, rounding_mode="floor") == keys % n
    return _from_keys(n, n, keys, torch.where(diag, 4.0, -1.0))


def _rmat_edges(scale, edge_factor, g):
    n = edge_factor << scale
    r = torch.zeros(n, dtype=torch.int64, device="cuda")
    c = torch.zeros(n, dtype=torch.int64, device="cuda")
    for bit in range(scale):
        u = torch.rand(n, generator=g, device="cuda")
        r |= (u >= 0.76).long() << bit
        c |= (((u >= 0.57) & (u < 0.76)) | (u >= 0.95)).long() << bit
    return r, c


def _row_products(A, B):
    blen = (B.row_ptr[1:] - B.row_ptr[:-1]).long()
    cum = torch.zeros(A.nnz + 1, dtype=torch.int64, device="cuda")
    cum[1:] = torch.cumsum(blen[A.col_idx.long()], 0)
    return cum[A.row_ptr.long()]  # products before each row


def _rmat(scale, edge_factor, panel, g):
    n = 1 << scale
    r, c = _rmat_edges(scale, edge_factor, g)
    keys = torch.unique(r * n + c)
    M = _from_keys(n, n, keys)
    if panel < 0:
        return M, M
    # the panel's rows: contiguous panels of at most 2^31 - 1 products each
    before = _row_products(M, M)
    r0 = 0
    for _ in range(panel + 1):
        r1 = int(torch.searchsorted(before, before[r0] + INT32_MAX, right=True)) - 1
        r1 = max(r0 + 1, min(r1, n))
        first, r0 = r0, (r1 if r1 < n else r0)
    view = M.row_ptr[first:r1 + 1]
    return Csr(r1 - first, n, int(view[-1]), view, M.col_idx, None), M


def _counted(counts, cols, g):
    """Sorted keys row * cols + column, about counts[row] distinct uniform columns a row."""
    rows = torch.repeat_interleave(torch.arange(counts.numel(), device="cuda"), counts)
    c = torch.randint(0, cols, (rows.numel(),), generator=g, device="cuda")
    return torch.unique(rows * cols + c)


def _tall(rows, n, g):
    u = torch.rand(rows, generator=g, device="cuda", dtype=torch.float64).clamp_min(1e-12)
    a_counts = (u.log() / math.log(1 - 1 / 8.0)).floor().long() + 1  # geometric, mean 8
    ka = _counted(a_counts, n, g)
    A = _from_keys(rows, n, ka)
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64).clamp_min(1e-12)
    b_counts = (4.1 * u ** (-1 / 1.1)).floor().clamp(1, min(20000, n)).long()  # mean about 24
    kb = _counted(b_counts, n, g)
    return A, _from_keys(n, n, kb)


def _sizes(case):
    r = random.Random(case["pattern"])
    return [(_log(r, case["lo"], case["hi"]), r.uniform(4.0, 32.0)) for _ in range(case["count"])]


def _block(sizes, g, gv):
    """One stacked random matrix per list of sizes, cut into the products' own CSR arrays."""
    n = torch.tensor([s for s, _ in sizes], device="cuda")
    lam = torch.tensor([x for _, x in sizes], device="cuda", dtype=torch.float32)
    counts = torch.poisson(lam.repeat_interleave(n), generator=g).long()
    width = n.repeat_interleave(n)  # columns of each row's matrix
    rows = torch.repeat_interleave(torch.arange(counts.numel(), device="cuda"), counts)
    c = (torch.rand(rows.numel(), generator=g, device="cuda", dtype=torch.float64) *
         width[rows]).long()
    big = 1 << 20
    M = _from_keys(counts.numel(), big, torch.unique(rows * big + c))
    M.values = _values(M.nnz, gv, "f32")
    out, r0 = [], 0
    ends = [0] + torch.cumsum(n, 0).tolist()
    bounds = M.row_ptr[torch.tensor(ends, device="cuda")].tolist()
    for i, (s, _) in enumerate(sizes):
        a, b = bounds[i], bounds[i + 1]
        rp = M.row_ptr[ends[i]:ends[i + 1] + 1] - a
        out.append(Csr(s, s, b - a, rp, M.col_idx[a:b].clone(), M.values[a:b].clone()))
    return out


def _operands(case, seed):
    """A and B: the pattern is the case's own, the values are the seed's."""
    g, gv = _gen(case["pattern"]), _gen(seed)
    m = case["matrix"]
    if m == "uniform":
        A = B = _uniform(case["rows"], case["cols"], case["per_row"], g)
        if case["rows"] != case["cols"]:
            B = _uniform(case["cols"], case["rows"], case["per_row"], g)
    elif m == "poisson":
        A = B = _poisson(case["nx"], case["ny"])
    elif m == "rmat":
        A, B = _rmat(case["scale"], case["edge_factor"], case["panel"], g)
    else:
        A, B = _tall(case["rows"], case["cols"], g)
    if case["kind"] == "i8":
        # entries that sum to zero are not stored: the values are the case's
        # own, with each row of A's sign the seed's, so every seed's C has
        # the same pattern
        B.values = _values(B.nnz, g, "i8")
        sign = torch.randint(0, 2, (A.rows,), generator=gv, device="cuda").to(torch.int8) * 2 - 1
        lens = (A.row_ptr[1:] - A.row_ptr[:-1]).long()
        v = B.values if A is B else _values(A.nnz, g, "i8")
        A = Csr(A.rows, A.cols, A.nnz, A.row_ptr, A.col_idx, v * sign.repeat_interleave(lens))
        return A, B
    if m == "poisson":
        B.values = (B.values * (torch.rand(B.nnz, generator=gv, device="cuda") + 0.5)).float()
    else:
        B.values = _values(B.nnz, gv, case["kind"])
    if A.col_idx is B.col_idx:
        A.values = B.values
    else:
        A.values = _values(A.nnz, gv, case["kind"])
    return A, B


def _pairs(case, seed):
    g, gv, sizes = _gen(case["pattern"]), _gen(seed), _sizes(case)
    return list(zip(_block(sizes, g, gv), _block(sizes, g, gv)))


def _edges(case, seed):
    """The case's edges in the seed's order, with the seed's values."""
    gv = _gen(seed)
    r, c = _rmat_edges(case["scale"], case["edge_factor"], _gen(case["pattern"]))
    order = torch.randperm(r.numel(), generator=gv, device="cuda")
    return r[order].int(), c[order].int(), _values(r.numel(), gv, "f32")


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------

class _Owned:
    """A library-owned device array: released when its tensor goes."""

    def __init__(self, p, n, typestr):
        self.p = p
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (p, False),
                                         "version": 3}

    def __del__(self):
        rv.free_device(self.p)


_TYPESTR = {torch.int32: "<i4", torch.float32: "<f4", torch.float64: "<f8"}


def _tensor(p, n, dtype):
    if n == 0:
        rv.free_device(p)
        return torch.zeros(0, dtype=dtype, device="cuda")
    return torch.as_tensor(_Owned(p, n, _TYPESTR[dtype]), device="cuda")


def _csr_out(rows, nnz, prp, pci, pv, dtype):
    return {"row_ptr": _tensor(prp, rows + 1, torch.int32),
            "col_idx": _tensor(pci, nnz, torch.int32), "values": _tensor(pv, nnz, dtype)}


class _HostOwned:
    """A host CSR result: released with rvsp_csr_destroy when its arrays go."""

    def __init__(self, c):
        self.c = c

    def __del__(self):
        rv.lib().rvsp_csr_destroy(C.byref(self.c))

    def array(self, p, n, typestr):
        a = _HostView(self, p, n, typestr)
        return np.asarray(a)


class _HostView:
    def __init__(self, owner, p, n, typestr):
        self.owner = owner
        self.__array_interface__ = {"shape": (n,), "typestr": typestr, "data": (p, False),
                                    "version": 3}


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "batched":
        s["pairs"] = _pairs(case, seed)
        return s
    if kind == "coo":
        s["r"], s["c"], s["v"] = _edges(case, seed)
        return s
    A, B = _operands(case, seed)
    s["A"], s["B"] = A, B
    if kind == "host":
        def host(M):
            return Csr(M.rows, M.cols, M.nnz, M.row_ptr.cpu().numpy(), M.col_idx.cpu().numpy(),
                       M.values.cpu().numpy())
        s["A"] = host(A)
        s["B"] = s["A"] if B is A else host(B)
    if kind in ("first", "reuse"):
        s["d"] = rv.Descriptor(rv.RVSP_SPGEMM_ALGO_CUDA)
        s["ws"] = torch.empty(4096, dtype=torch.uint8, device="cuda")
    if kind == "reuse":  # the structure analysed and filled by an earlier product
        _first(s)
    return s


def _first(s):
    A, B, d = s["A"], s["B"], s["d"]
    a, b = A.struct(), B.struct()
    st, _, nnz = d.work_estimation(a, b)
    rv.check(st, "work_estimation")
    s["out"] = {"row_ptr": torch.empty(A.rows + 1, dtype=torch.int32, device="cuda"),
                "col_idx": torch.empty(nnz, dtype=torch.int32, device="cuda"),
                "values": torch.empty(nnz, dtype=torch.float32, device="cuda")}
    s["c"] = rv.csr_struct(A.rows, B.cols, nnz, s["out"]["row_ptr"], s["out"]["col_idx"],
                           s["out"]["values"])
    rv.check(d.compute(a, b, s["c"], s["ws"]), "compute")
    return s["out"]


def run(state):
    case = state["case"]
    kind = case["kind"]
    L = rv.lib()
    algo = rv.RVSP_CUDA_ALGO_LEARNED if case.get("algo") == "learned" else rv.RVSP_CUDA_ALGO_EXACT
    if kind == "first":
        return _first(state)
    if kind == "reuse":
        rv.check(state["d"].compute(state["A"].struct(), state["B"].struct(), state["c"],
                                    state["ws"]), "compute")
        return state["out"]
    if kind == "batched":
        (prp, pci, pv), nnz, rows, entries = rv.spgemm_batched(state["pairs"], algo)
        out = _csr_out(int(rows[-1]) + len(state["pairs"]) - 1, nnz, prp, pci, pv, torch.float32)
        return out | {"row_offsets": rows, "entry_offsets": entries}
    if kind == "host":
        A, B = state["A"], state["B"]
        a, b, c = rv.from_csr(A), rv.from_csr(B), rv.CsrMatrix()
        opts = rv.SpgemmOptions(rv.RVSP_BACKEND_CUDA_LEARNED if case["algo"] == "learned"
                                else rv.RVSP_BACKEND_CUDA, rv.RVSP_DTYPE_FP32, rv.RVSP_DTYPE_FP32)
        rv.check(L.rvsp_spgemm_csr(C.byref(a), C.byref(b), C.byref(c), C.byref(opts)),
                 "rvsp_spgemm_csr")
        o = _HostOwned(c)
        return {"row_ptr": o.array(c.row_ptr, A.rows + 1, "<i4"),
                "col_idx": o.array(c.col_idx, c.nnz, "<i4"),
                "values": o.array(c.values, c.nnz, "<f4")}
    prp, pci, pv, nnz = C.c_void_p(), C.c_void_p(), C.c_void_p(), C.c_int32()
    if kind == "coo":
        n = 1 << case["scale"]
        rv.check(L.rvsp_cuda_coo_to_csr(n, n, state["r"].numel(), rv.ptr(state["r"]),
                                        rv.ptr(state["c"]), rv.ptr(state["v"]),
                                        1 if case["symmetric"] else 0, 1, C.byref(prp),
                                        C.byref(pci), C.byref(pv), C.byref(nnz)), "coo_to_csr")
        return _csr_out(n, nnz.value, prp.value, pci.value, pv.value, torch.float32)
    A, B = state["A"], state["B"]
    ops = [rv.ptr(x) for x in (A.row_ptr, A.col_idx, A.values, B.row_ptr, B.col_idx, B.values)]
    outs = [C.byref(x) for x in (prp, pci, pv, nnz)]
    if kind == "f64":
        rv.check(L.rvsp_cuda_spgemm_f64(A.rows, A.cols, B.cols, *ops, *outs), "spgemm_f64")
    elif kind == "i8":
        rv.check(L.rvsp_cuda_spgemm_i8(A.rows, A.cols, B.cols, *ops, *outs), "spgemm_i8")
    else:
        rv.check(L.rvsp_cuda_spgemm_f32(algo, A.rows, A.cols, B.cols, *ops, *outs, None),
                 "spgemm_f32")
    dtype = {"f64": torch.float64, "i8": torch.int32}.get(kind, torch.float32)
    return _csr_out(A.rows, nnz.value, prp.value, pci.value, pv.value, dtype)


# ---------------------------------------------------------------------------
# work: operands read once, C written once; expected sizes of the seeded matrices
# ---------------------------------------------------------------------------

def _csr_bytes(rows, nnz, vbytes=4):
    return 4 * (rows + 1) + (4 + vbytes) * nnz


def work(case):
    kind = case["kind"]
    if kind == "batched":
        b = f = 0.0
        for n, lam in _sizes(case):
            p = n * lam * lam
            nnz_c = n * n * (1 - math.exp(-lam * lam / n))
            b += 2 * _csr_bytes(n, n * lam) + _csr_bytes(n, nnz_c)
            f += 2 * p
        return {"bytes": b, "flops": f}
    if kind == "coo":
        n = case["edge_factor"] << case["scale"]
        out = 0.96 * n * (2 if case["symmetric"] else 1)
        return {"bytes": 12 * n + _csr_bytes(1 << case["scale"], out),
                "flops": 0.04 * n}
    vb, ob = {"f64": (8, 8), "i8": (1, 4)}.get(kind, (4, 4))
    m = case["matrix"]
    if m == "uniform":
        rows, cols, k = case["rows"], case["cols"], case["per_row"]
        n_b, p = rows if rows != cols else cols, rows * k * k
        nnz_a, nnz_b = rows * k, cols * k
        nnz_c = rows * n_b * (1 - math.exp(-k * k / n_b))
        rows_b = cols
    elif m == "poisson":
        rows = rows_b = case["nx"] * case["ny"]
        nnz_a = nnz_b = 5 * rows - 2 * (case["nx"] + case["ny"])
        p, nnz_c = 25 * rows, 13 * rows
    elif m == "rmat":
        s, ef = case["scale"], case["edge_factor"]
        rows = rows_b = 1 << s
        nnz_a = nnz_b = 0.9 * ef * rows
        p = 400.8e6 * 7.3 ** ((s - 16) / 2) * (ef / 16) ** 1.75
        if case["panel"] >= 0:  # nine full panels and a rest
            share = min(1.0, INT32_MAX / p)
            rows, nnz_a, p = rows * share, nnz_a * share, p * share
        nnz_c = 0.46 * p
    else:
        rows, rows_b = case["rows"], case["cols"]
        nnz_a, nnz_b = 8 * rows, 24 * rows_b
        p = nnz_c = 190 * rows
    return {"bytes": _csr_bytes(rows, nnz_a, vb) + _csr_bytes(rows_b, nnz_b, vb) +
            _csr_bytes(rows, nnz_c, ob), "flops": 2 * p}


# ---------------------------------------------------------------------------
# exact: the values in 64 bits, by expanding and sorting the products
# ---------------------------------------------------------------------------

def _exact_rows(A, B, before, r0, r1):
    """Values of rows [r0, r1) in row then column order, summed in FP64."""
    lo, hi = int(A.row_ptr[r0]), int(A.row_ptr[r1])
    if hi == lo:
        return torch.zeros(0, dtype=torch.float64, device="cuda")
    k = A.col_idx[lo:hi].long()
    lens = (B.row_ptr[1:] - B.row_ptr[:-1]).long()[k]
    rows = torch.repeat_interleave(torch.arange(r1 - r0, device="cuda"),
                                   (A.row_ptr[r0 + 1:r1 + 1] - A.row_ptr[r0:r1]).long())
    ends = torch.cumsum(lens, 0)
    e = torch.repeat_interleave(torch.arange(hi - lo, device="cuda"), lens)
    q = torch.arange(int(ends[-1]), device="cuda") - (ends - lens)[e] + B.row_ptr.long()[k][e]
    prod = A.values[lo:hi].double()[e] * B.values[q].double()
    key, order = (rows[e] * B.cols + B.col_idx[q].long()).sort()
    del e, q
    _, where = torch.unique_consecutive(key, return_inverse=True)
    n = int(where[-1]) + 1 if where.numel() else 0
    return torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, where, prod[order])


def _exact_values(A, B):
    shift = int(A.row_ptr[0])
    if shift:  # a row panel: its own entries, from 0
        A = Csr(A.rows, A.cols, A.nnz - shift, A.row_ptr - shift, A.col_idx[shift:A.nnz],
                A.values[shift:A.nnz])
    before = _row_products(A, B)
    parts, r0 = [], 0
    while r0 < A.rows:
        r1 = int(torch.searchsorted(before, before[r0] + 100_000_000, right=True)) - 1
        r1 = max(r0 + 1, min(r1, A.rows))
        parts.append(_exact_rows(A, B, before, r0, r1))
        r0 = r1
    return torch.cat(parts)


def exact(case, seed):
    kind = case["kind"]
    if kind == "i8":  # whole numbers
        return None
    if kind == "batched":
        return {"row_ptr": None, "col_idx": None, "row_offsets": None, "entry_offsets": None,
                "values": torch.cat([_exact_values(A, B) for A, B in _pairs(case, seed)])}
    if kind == "coo":
        n = 1 << case["scale"]
        r, c, v = _edges(case, seed)
        r, c, v = r.long(), c.long(), v.double()
        if case["symmetric"]:
            off = r != c
            r, c, v = (torch.cat([r, c[off]]), torch.cat([c, r[off]]), torch.cat([v, v[off]]))
        key, order = (r * n + c).sort(stable=True)
        _, where = torch.unique_consecutive(key, return_inverse=True)
        out = torch.zeros(int(where[-1]) + 1, dtype=torch.float64, device="cuda")
        return {"row_ptr": None, "col_idx": None, "values": out.index_add_(0, where, v[order])}
    A, B = _operands(case, seed)
    v = _exact_values(A, B)
    return {"row_ptr": None, "col_idx": None, "values": v.cpu().numpy() if kind == "host" else v}
