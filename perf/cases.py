"""Performance cases: the work a user's program has this library do.

Each case is one call sequence through the public entry points on matrices of the kinds
the benchmark (bench.py) and the tests use: grid Laplacians, Zipf-row graphs, 27-point
stencils, 3x3-block FEM-like matrices and mixed batches.  Matrices and vectors are made
from the seed on the GPU; a program hands the library host structs once (the handle), then
calls it many times.  A pass sets the result buffer to its starting value y0 (the library
computes y += A x) and runs the operation on the program's stream.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from clspmv_b200 import (COO, CSP_FLAG_ADJOINT, CSP_FLAG_BF16, CSP_FLAG_GRAPH, CSP_METH_XPANEL, Batch, Cocktail, Handle,
                         capi, lib)
from clspmv_b200.batch import CSP_BATCH_ADJ, CSP_BATCH_FWD, CSP_BATCH_TUNE_MODEL

ELL_4ROW, CSR_ADAPTIVE, CSR_GROUP, DIA_4ROW, BDIA_STAGED = 1, 2, 3, 1, 1


# --------------------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------------------
def listed():
    return [
        # The smallest call: one SpMV of a 128 x 128 grid Laplacian inside a host-driven solver; launch-bound.
        {"name": "laplacian_128_csr", "family": "laplacian", "nx": 128, "ny": 128, "format": "csr",
         "method": CSR_ADAPTIVE, "bf16": False},
        # An explicit time stepper that stays on the device: u += A u, 64 steps in one call, as captured graphs.
        {"name": "heat_511x517_dia_64steps", "family": "heat", "nx": 511, "ny": 517, "format": "dia",
         "method": DIA_4ROW, "steps": 64},
        # A large irregular graph (one power-iteration step) in the layout for columns without locality.
        {"name": "zipf_1m_xpanel", "family": "zipf", "rows": 1_000_000, "format": "csr", "method": CSP_METH_XPANEL,
         "op": "spmv", "bf16": False},
        # A smaller graph whose arrays the program already holds on the device, in entry (COO) order.
        {"name": "zipf_300k_coo_device", "family": "zipf", "rows": 300_007, "format": "noalloc", "method": 0,
         "op": "spmv", "bf16": False},
        # A training step over an irregular matrix in CSR: forward, transposed product and value gradients.
        {"name": "zipf_200k_csr_step", "family": "zipf", "rows": 200_003, "format": "csr", "method": CSR_ADAPTIVE,
         "op": "step", "bf16": False},
        # A large structured-grid operator, forward only: the largest stencil the benchmark runs.
        {"name": "stencil_160_bdia", "family": "stencil", "g": 160, "format": "bdia", "method": BDIA_STAGED,
         "op": "spmv", "bf16": False},
        # A mid-size stencil with an odd grid: forward, transposed product and value gradients.
        {"name": "stencil_97_dia_step", "family": "stencil", "g": 97, "format": "dia", "method": DIA_4ROW,
         "op": "step", "bf16": False},
        # A FEM-like 3x3-block matrix, one right-hand side: the inner product of an iterative solver.
        {"name": "fem_500k_k1", "family": "fem", "block_rows": 500_000, "k": 1, "bf16": False},
        # The same with eight right-hand sides and values stored as BF16 (a block solver that saves memory).
        {"name": "fem_500k_k8_bf16", "family": "fem", "block_rows": 500_000, "k": 8, "bf16": True},
        # The same with 32 right-hand sides in FP32: the largest call.
        {"name": "fem_500k_k32", "family": "fem", "block_rows": 500_000, "k": 32, "bf16": False},
        # A few small matrices of mixed structure, forward only: an inference request.
        {"name": "batch_24_small_fwd", "family": "batch", "count": 24, "lo": 1_000, "hi": 8_000, "op": "spmv",
         "bf16": False},
        # A batch of uneven matrices of all three structures, forward + adjoint + value gradients: a training step.
        {"name": "batch_128_step", "family": "batch", "count": 128, "lo": 1_000, "hi": 200_000, "op": "step",
         "bf16": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    family = rng.choice(("laplacian", "heat", "zipf", "zipf", "stencil", "stencil", "fem", "fem", "fem", "batch", "batch"))
    if family == "laplacian":
        fmt, method = rng.choice((("csr", CSR_ADAPTIVE), ("csr", CSR_GROUP), ("ell", ELL_4ROW), ("dia", DIA_4ROW)))
        return {"family": family, "nx": _log_int(rng, 40, 900), "ny": _log_int(rng, 40, 900), "format": fmt,
                "method": method, "bf16": rng.random() < 0.25}
    if family == "heat":
        fmt, method = rng.choice((("csr", CSR_ADAPTIVE), ("ell", ELL_4ROW), ("dia", DIA_4ROW)))
        return {"family": family, "nx": _log_int(rng, 64, 700), "ny": _log_int(rng, 64, 700), "format": fmt,
                "method": method, "steps": rng.randint(8, 100)}
    if family == "zipf":
        fmt, method, op = rng.choice((("csr", CSP_METH_XPANEL, "spmv"), ("csr", CSR_ADAPTIVE, "spmv"), ("coo", 0, "spmv"),
                                      ("noalloc", 0, "spmv"), ("csr", CSR_ADAPTIVE, "step")))
        return {"family": family, "rows": _log_int(rng, 5_000, 1_000_000 if op == "spmv" else 300_000), "format": fmt,
                "method": method, "op": op, "bf16": fmt != "noalloc" and op == "spmv" and rng.random() < 0.25}
    if family == "stencil":
        fmt, method = rng.choice((("bdia", BDIA_STAGED), ("dia", DIA_4ROW)))
        op = rng.choice(("spmv", "step"))
        return {"family": family, "g": _log_int(rng, 20, 150 if op == "spmv" else 110), "format": fmt, "method": method,
                "op": op, "bf16": op == "spmv" and rng.random() < 0.3}
    if family == "fem":
        return {"family": family, "block_rows": _log_int(rng, 3_000, 400_000),
                "k": rng.choice((1, 1, 1, 3, 4, 8, 8, 16, 20, 32, 32)), "bf16": rng.random() < 0.4}
    lo = _log_int(rng, 500, 4_000)
    return {"family": family, "count": _log_int(rng, 4, 40), "lo": lo, "hi": lo * rng.randint(2, 40),
            "op": rng.choice(("spmv", "step", "step")), "bf16": rng.random() < 0.25}


# --------------------------------------------------------------------------------------
# inputs, made on the GPU from the seed
# --------------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform(gen, n, low=-1.0, high=1.0):
    return torch.rand(n, generator=gen, device="cuda") * (high - low) + low


def _stored(val, bf16):
    """The values the library works with: rounded to BF16 where they are stored so."""
    return val.to(torch.bfloat16).to(torch.float32) if bf16 else val


def _grid5(nx, ny, diag, off):
    """5-point operator on an nx-by-ny grid: diagonal-major (offsets, columns, values), -1 where outside."""
    n = nx * ny
    k = torch.arange(n, device="cuda")
    i, j = k // nx, k % nx
    offs = [-nx, -1, 0, 1, nx]
    ok = torch.stack([i > 0, j > 0, k >= 0, j < nx - 1, i < ny - 1])
    col = torch.where(ok, k[None, :] + torch.tensor(offs, device="cuda")[:, None], -1)
    val = torch.full((5, n), off, device="cuda")
    val[2] = diag
    return offs, col, torch.where(ok, val, torch.zeros_like(val))


def _grid27(g, gen):
    """27-point stencil on a g^3 grid, values U(0.5, 1.5): (offsets, in-grid mask, values), diagonal-major."""
    n = g ** 3
    k = torch.arange(n, device="cuda")
    z, y, x = k // (g * g), (k // g) % g, k % g
    offs, val = [], torch.empty((27, n), device="cuda")
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                ok = ((z + dz >= 0) & (z + dz < g) & (y + dy >= 0) & (y + dy < g) & (x + dx >= 0) & (x + dx < g))
                val[len(offs)] = _uniform(gen, n, 0.5, 1.5) * ok
                offs.append(dz * g * g + dy * g + dx)
    return offs, val


def _distinct(gen, row, lo, hi, width):
    """Columns in [lo, hi) per entry, distinct inside each row, sorted by (row, column)."""
    col = lo + (torch.rand(row.numel(), generator=gen, device="cuda", dtype=torch.float64) * (hi - lo)).long()
    key = torch.sort(row * width + col).values
    while True:
        again = torch.zeros_like(key, dtype=torch.bool)
        again[1:] = key[1:] == key[:-1]
        count = int(again.sum())
        if not count:
            return key // width, key % width
        r, l, h = key[again] // width, lo[again], hi[again]   # row order keeps every row's bounds in place
        key[again] = r * width + l + (torch.rand(count, generator=gen, device="cuda", dtype=torch.float64) * (h - l)).long()
        key = torch.sort(key).values


def _zipf(n, seed, s=2.0, max_len=10_000):
    """n-by-n, Zipf(s) row lengths clipped to [1, max_len], uniform distinct columns, values N(0, 1).
    The size fixes the lengths (so every seed has the same number of entries), the seed their order."""
    gen = _generator(seed)
    lens = np.clip(np.random.default_rng(n).zipf(s, n), 1, min(max_len, max(1, n // 4))).astype(np.int64)
    lens = torch.from_numpy(lens).cuda()[torch.randperm(n, generator=gen, device="cuda")]
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), lens)
    zero, full = torch.zeros_like(row), torch.full_like(row, n)
    row, col = _distinct(gen, row, zero, full, n)
    return row, col, torch.randn(row.numel(), generator=gen, device="cuda")


def _blocks(nbr, gen, deg, band=2000):
    """Block columns of an nbr-by-nbr block matrix: degree uniform in deg (the size fixes the degrees, the seed
    their order), columns uniform within +-band."""
    i = torch.arange(nbr, device="cuda")
    lo, hi = (i - band).clamp(min=0), (i + band).clamp(max=nbr - 1) + 1
    d = torch.randint(deg[0], deg[1] + 1, (nbr,), generator=_generator(nbr), device="cuda")
    d = torch.minimum(d[torch.randperm(nbr, generator=gen, device="cuda")], hi - lo)
    brow = torch.repeat_interleave(i, d)
    return _distinct(gen, brow, lo[brow], hi[brow], nbr)


def _fem(nbr, gen):
    """3x3-block FEM-like matrix: block rows, block columns, values (9, blocks)."""
    brow, bcol = _blocks(nbr, gen, (10, 30))
    return brow, bcol, torch.randn((9, brow.numel()), generator=gen, device="cuda")


def _entries(kind, rows, seed):
    """One matrix of a mixed batch at about 12 nonzeros per row: (n, row, col, val)."""
    gen = _generator(seed)
    if kind == "laplacian":   # the squared 5-point Laplacian: 13 points
        nx = max(3, int(math.sqrt(rows)))
        ny = max(3, rows // nx)
        k = torch.arange(nx * ny, device="cuda")
        i, j = k // nx, k % nx
        points = [(0, 0, 20.0)] + [(a, b, -8.0) for a, b in ((0, 1), (0, -1), (1, 0), (-1, 0))]
        points += [(a, b, 2.0) for a in (-1, 1) for b in (-1, 1)] + [(a, b, 1.0) for a, b in ((0, 2), (0, -2), (2, 0), (-2, 0))]
        points.sort()
        col = torch.stack([torch.where((i + a >= 0) & (i + a < ny) & (j + b >= 0) & (j + b < nx), k + a * nx + b, -1)
                           for a, b, _ in points], 1)
        val = torch.tensor([v for _, _, v in points], device="cuda").expand(nx * ny, -1)
        val = val * _uniform(gen, nx * ny, 0.5, 1.5)[:, None]   # a coefficient per cell
        ok = col >= 0
        return nx * ny, k[:, None].expand(-1, len(points))[ok], col[ok], val[ok]
    if kind == "zipf":
        return (rows,) + _zipf(rows, seed, s=1.85)
    nbr = max(2, rows // 3)
    brow, bcol = _blocks(nbr, gen, (2, 6))
    a = torch.arange(3, device="cuda")
    row = (3 * brow[:, None, None] + a[None, :, None]).expand(-1, 3, 3).reshape(-1)
    col = (3 * bcol[:, None, None] + a[None, None, :]).expand(-1, 3, 3).reshape(-1)
    order = torch.argsort(row * (3 * nbr) + col)
    return 3 * nbr, row[order], col[order], torch.randn(row.numel(), generator=gen, device="cuda")


def _batch_shapes(case, seed):
    """(kind, rows, seed) of every matrix; sizes are the case's, not the seed's."""
    rng = np.random.default_rng(case["count"] * 1_000_003 + case["lo"])
    out = []
    for i in range(case["count"]):
        rows = int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        out.append((("laplacian", "zipf", "block")[i % 3], rows, int(seed) * 1009 + i))
    return out


def _host(t, dtype):
    return np.ascontiguousarray(t.to(dtype).cpu().numpy())


_I32, _F32 = torch.int32, torch.float32


def _coo(n, row, col, val):
    return COO(n, n, _host(row, _I32), _host(col, _I32), _host(val, _F32))


def _diagonals(n, offs, val):
    """A Cocktail of one DIA or BDIA part over arrays this module keeps."""
    aligned = (n + 31) // 32 * 32
    data = torch.zeros((len(offs), aligned), device="cuda")
    data[:, :n] = val
    return aligned, _host(data.reshape(-1), _F32)


def _diagonal_mat(fmt, method, n, offs, val):
    mat = Cocktail(n, n, int((val != 0).sum()))
    mat._owned = False   # the arrays below are numpy's, not the library's
    aligned, data = _diagonals(n, offs, val)
    o = np.array(offs, np.int32)
    keep = [o, data]
    if fmt == "dia":
        d = mat.s.dia
        d.dia_num, d.dia_length, d.dia_length_aligned = len(offs), n, aligned
        d.dia_offsets, d.dia_data = capi.as_ptr(o, C.c_int), capi.as_ptr(data, C.c_float)
        mat.s.ifusedia, mat.s.dia_meth_num = True, method
    else:
        first = [i for i in range(len(offs)) if i == 0 or offs[i] != offs[i - 1] + 1]
        bo, bp = o[first].copy(), np.array(first + [len(offs)], np.int32)
        keep += [bo, bp]
        d = mat.s.bdia
        d.bdia_band_num, d.bdia_length, d.bdia_length_aligned = len(first), n, aligned
        d.bdia_offsets, d.bdia_bptr = capi.as_ptr(bo, C.c_int), capi.as_ptr(bp, C.c_int)
        d.bdia_data = capi.as_ptr(data, C.c_float)
        mat.s.ifusebdia, mat.s.bdia_meth_num = True, method
    d.matinfo.width, d.matinfo.height, d.matinfo.nnz = n, n, mat.s.mat_nnz
    mat._keep = keep
    return mat


# --------------------------------------------------------------------------------------
# one matrix per case: (n, k, ...) as 64-bit exact() and the handles both need it
# --------------------------------------------------------------------------------------
def _vectors(case, seed, n, k=1):
    gen = _generator(int(seed) + 77_777)
    return [_uniform(gen, n * k) for _ in range(4)]   # x, y0, ybar, xbar0


class _View:
    """A device buffer of `owner` (a Handle or Batch), as an array torch can wrap; a tensor over it keeps the owner."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "data": (ptr, False), "version": 3}


def _view(owner, ptr, n):
    return torch.as_tensor(_View(owner, ptr, n), device="cuda")


_STREAM = []


def _stream():
    """The program's stream, torch's current one: every handle runs on it too."""
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
        _STREAM[0].wait_stream(torch.cuda.current_stream())
        torch.cuda.set_stream(_STREAM[0])
    return _STREAM[0]


def _flat_case(case, seed):
    """laplacian, heat, zipf: (n, row, col, val) in row order."""
    if case["family"] == "zipf":
        return (case["rows"],) + _zipf(case["rows"], seed)
    heat = case["family"] == "heat"
    _, col, val = _grid5(case["nx"], case["ny"], -0.8 if heat else 4.0, 0.2 if heat else -1.0)
    n = case["nx"] * case["ny"]
    ok = (col >= 0).t()
    row = torch.arange(n, device="cuda")[:, None].expand(-1, 5)[ok]
    return n, row, col.t()[ok], val.t()[ok].contiguous()


def prepare(case, seed):
    _stream()
    family = case["family"]
    flags = CSP_FLAG_BF16 if case.get("bf16") else 0
    if family == "batch":
        return _prepare_batch(case, seed, flags)
    state = {"case": case, "op": case.get("op", "spmv")}
    if state["op"] == "step":
        flags |= CSP_FLAG_ADJOINT
    if family == "fem":
        k, nbr = case["k"], case["block_rows"]
        n = 3 * nbr
        gen = _generator(seed)
        brow, bcol, val = _fem(nbr, gen)
        blocks = brow.numel()
        aligned = (blocks + 31) // 32 * 32
        data = torch.zeros((9, aligned), device="cuda")
        data[:, :blocks] = val
        rp = torch.zeros(nbr + 1, dtype=_I32, device="cuda")
        rp[1:] = torch.cumsum(torch.bincount(brow, minlength=nbr), 0)
        arrays = [_host(rp, _I32), _host(3 * bcol, _I32), _host(data.reshape(-1), _F32)]
        b = capi.bcsr_matrix()
        b.matinfo.width, b.matinfo.height, b.matinfo.nnz = n, n, 9 * blocks
        b.bcsr_bwidth, b.bcsr_bheight, b.bcsr_row_num = 3, 3, nbr
        b.bcsr_aligned_size, b.bcsr_block_num = aligned, blocks
        b.bcsr_row_ptr, b.bcsr_col_id = capi.as_ptr(arrays[0], C.c_int), capi.as_ptr(arrays[1], C.c_int)
        b.bcsr_data = capi.as_ptr(arrays[2], C.c_float)
        x, y0, _, _ = _vectors(case, seed, n, k)
        h = Handle(None, _host(x, _F32), None, flags, nrhs=k, bcsr=b)
    else:
        k = 1
        if family == "stencil":
            n = case["g"] ** 3
            offs, val = _grid27(case["g"], _generator(seed))
            mat = _diagonal_mat(case["format"], case["method"], n, offs, val)
        elif case["format"] == "noalloc":
            n, row, col, val = _flat_case(case, seed)
            x, y0, _, _ = _vectors(case, seed, n)
            state.update(n=n, row=row.to(_I32), col=col.to(_I32), val=val.contiguous(), x=x, y0=y0, y=y0.clone())
            return state
        elif case["format"] == "dia":
            offs, _, val = _grid5(case["nx"], case["ny"], *((-0.8, 0.2) if family == "heat" else (4.0, -1.0)))
            n = case["nx"] * case["ny"]
            mat = _diagonal_mat("dia", case["method"], n, offs, val)
        else:
            n, row, col, val = _flat_case(case, seed)
            mat = Cocktail.single(case["format"], _coo(n, row, col, val), case["method"])
        x, y0, ybar, xbar0 = _vectors(case, seed, n)
        if family == "heat":
            flags |= CSP_FLAG_GRAPH
            y0 = x
        h = Handle(mat, _host(x, _F32), None, flags)
        mat.free()
        if state["op"] == "step":
            state.update(ybar=ybar, xbar0=xbar0, xbar=xbar0.clone(),
                         abar=torch.zeros(h.adjoint_slots, device="cuda"))
    h.set_stream(_stream().cuda_stream)
    state.update(n=n, count=n * k, handle=h, x=x, y0=y0, y=_view(h, h.res_ptr, n * k))
    return state


def _prepare_batch(case, seed, flags):
    step = case["op"] == "step"
    mats = [_coo(*_entries(*shape)) for shape in _batch_shapes(case, seed)]
    b = Batch(mats, flags=flags | CSP_FLAG_GRAPH | (CSP_FLAG_ADJOINT if step else 0), tune=CSP_BATCH_TUNE_MODEL)
    b.mats = []   # the batch holds its own copies
    b.set_stream(_stream().cuda_stream)
    nx, ny, na = int(b.x_off[-1]), int(b.y_off[-1]), int(b.abar_off[-1])
    x, y0, ybar, xbar0 = _vectors(case, seed, nx)
    p = b.device_ptrs()
    _view(b, p["x"], nx).copy_(x)
    state = {"case": case, "op": case["op"], "batch": b, "y0": y0, "y": _view(b, p["y"], ny)}
    if step:
        _view(b, p["ybar"], ny).copy_(ybar)
        state.update(xbar0=xbar0, xbar=_view(b, p["xbar"], nx), abar=_view(b, p["abar"], na))
    torch.cuda.synchronize()
    return state


# --------------------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------------------
def run(state):
    op = state["op"]
    if "batch" in state:
        state["y"].copy_(state["y0"])
        if op == "step":
            state["xbar"].copy_(state["xbar0"])
        state["batch"].run(CSP_BATCH_FWD | CSP_BATCH_ADJ if op == "step" else CSP_BATCH_FWD)
        return {"y": state["y"], "xbar": state["xbar"], "abar": state["abar"]} if op == "step" else {"y": state["y"]}
    if "handle" not in state:   # COO arrays held by the program
        y, n = state["y"], state["n"]
        y.copy_(state["y0"])
        capi.check(lib().csp_coo_spmv_noalloc(n, n, state["row"].numel(), state["row"].data_ptr(), state["col"].data_ptr(),
                                              state["val"].data_ptr(), state["x"].data_ptr(), y.data_ptr(),
                                              _stream().cuda_stream), "coo_spmv_noalloc")
        return {"y": y}
    h = state["handle"]
    h.cpy_result_from_gpu(state["y0"].data_ptr(), state["count"])
    if state["case"]["family"] == "heat":
        h.cpy_vector_from_gpu(state["x"].data_ptr(), state["count"])
        h.iterate(state["case"]["steps"])
        return {"y": state["y"]}
    h.do_spmv(1)
    if op != "step":
        return {"y": state["y"]}
    state["xbar"].copy_(state["xbar0"])
    h.spmv_adjoint(state["ybar"].data_ptr(), state["xbar"].data_ptr(), state["abar"].data_ptr())
    return {"y": state["y"], "xbar": state["xbar"], "abar": state["abar"]}


# --------------------------------------------------------------------------------------
# what a pass cannot do without, and its results in 64 bits
# --------------------------------------------------------------------------------------
def _spmv_bytes(matrix, n, k=1):
    return matrix + 12 * n * k   # x and y0 read, y written


def work(case):
    family, vb = case["family"], 2 if case.get("bf16") else 4
    step = case.get("op") == "step"
    if family in ("laplacian", "heat"):
        nx, ny = case["nx"], case["ny"]
        n, nnz, steps = nx * ny, 5 * nx * ny - 2 * nx - 2 * ny, case.get("steps", 1)
        matrix = {"dia": vb * 5 * n, "ell": (vb + 4) * 5 * n, "csr": (vb + 4) * nnz + 4 * n}[case["format"]]
        return {"bytes": steps * _spmv_bytes(matrix, n), "flops": 2 * nnz * steps}
    if family == "zipf":
        # the mean of the clipped Zipf row lengths
        n = case["rows"]
        lim = min(10_000, max(1, n // 4))
        zeta = math.pi ** 2 / 6
        nnz = int(n * (sum(1.0 / l for l in range(1, lim)) / zeta + lim * (1 - sum(1.0 / l ** 2 for l in range(1, lim)) / zeta)))
        matrix = (vb + 8) * nnz if case["format"] in ("coo", "noalloc") else (vb + 4) * nnz + 4 * n
    elif family == "stencil":
        n = case["g"] ** 3
        nnz = (3 * case["g"] - 2) ** 3
        matrix = vb * 27 * n
        if step:   # forward, transposed product, one gradient per slot
            return {"bytes": 2 * _spmv_bytes(matrix, n) + 4 * 27 * n, "flops": 5 * nnz}
    elif family == "fem":
        n, k, blocks = 3 * case["block_rows"], case["k"], 20 * case["block_rows"]
        return {"bytes": _spmv_bytes((9 * vb + 4) * blocks + 4 * case["block_rows"], n, k), "flops": 18 * blocks * k}
    else:
        n = nnz = matrix = 0
        for kind, rows, _ in _batch_shapes(case, 0):
            n += rows
            if kind == "laplacian":
                nnz, matrix = nnz + 13 * rows, matrix + 13 * vb * rows
            elif kind == "zipf":
                lim = min(10_000, max(1, rows // 4))
                zeta = sum(l ** -1.85 for l in range(1, 20_000)) + 20_000 ** -0.85 / 0.85
                head = sum(l ** -1.85 for l in range(1, lim)) / zeta
                z = int(rows * (sum(l ** -0.85 for l in range(1, lim)) / zeta + lim * (1 - head)))
                nnz, matrix = nnz + z, matrix + (vb + 4) * z + 4 * rows
            else:
                nnz, matrix = nnz + 12 * rows, matrix + (9 * vb + 4) * (4 * rows // 3) + 4 * rows // 3
    if step:
        return {"bytes": 2 * _spmv_bytes(matrix, n) + 4 * nnz, "flops": 5 * nnz}
    return {"bytes": _spmv_bytes(matrix, n), "flops": 2 * nnz}


def _product(row, col, val, x, y0):
    return y0.double().index_add(0, row, val.double() * x.double()[col])


def exact(case, seed):
    family, bf16 = case["family"], bool(case.get("bf16"))
    if family == "batch":
        mats = [_entries(*shape) for shape in _batch_shapes(case, seed)]
        total = sum(m[0] for m in mats)
        x, y0, ybar, xbar0 = _vectors(case, seed, total)
        y, xbar, at = y0.double(), xbar0.double(), 0
        for n, row, col, val in mats:
            val, part = _stored(val, bf16), slice(at, at + n)
            y[part] = _product(row, col, val, x[part], y0[part])
            xbar[part] = _product(col, row, val, ybar[part], xbar0[part])
            at += n
        return {"y": y, "xbar": xbar, "abar": None} if case["op"] == "step" else {"y": y}
    if family == "fem":
        nbr, k = case["block_rows"], case["k"]
        brow, bcol, val = _fem(nbr, _generator(seed))
        val = _stored(val, bf16)
        x, y0, _, _ = _vectors(case, seed, 3 * nbr, k)
        y, xd = y0.double().view(nbr, 3, k), x.double().view(nbr, 3, k)
        step = max(1, 60_000_000 // (3 * k))
        for a in range(0, brow.numel(), step):
            part = slice(a, a + step)
            p = torch.einsum("ebi,bik->bek", val[:, part].double().view(3, 3, -1).permute(0, 2, 1), xd[bcol[part]])
            y.index_add_(0, brow[part], p)
        return {"y": y.reshape(-1)}
    if family == "stencil" or case["format"] == "dia":
        if family == "stencil":
            n = case["g"] ** 3
            offs, val = _grid27(case["g"], _generator(seed))
        else:
            n = case["nx"] * case["ny"]
            offs, _, val = _grid5(case["nx"], case["ny"], *((-0.8, 0.2) if family == "heat" else (4.0, -1.0)))
        val = _stored(val, bf16).double()
        x, y0, ybar, xbar0 = _vectors(case, seed, n)

        def apply(u, out):
            for d, o in enumerate(offs):
                a, b = max(0, -o), min(n, n - o)
                out[a:b] += val[d, a:b] * u[a + o:b + o]
            return out

        if family == "heat":
            u = x.double()
            for _ in range(case["steps"]):
                u = apply(u, u.clone())
            return {"y": u}
        y = apply(x.double(), y0.double())
        if case.get("op") != "step":
            return {"y": y}
        aligned = (n + 31) // 32 * 32
        xbar, abar = xbar0.double(), torch.zeros((27, aligned), dtype=torch.float64, device="cuda")
        for d, o in enumerate(offs):
            a, b = max(0, -o), min(n, n - o)
            xbar[a + o:b + o] += val[d, a:b] * ybar[a:b].double()
            abar[d, a:b] = ybar[a:b].double() * x[a + o:b + o].double()
        return {"y": y, "xbar": xbar, "abar": abar.reshape(-1)}
    n, row, col, val = _flat_case(case, seed)
    val = _stored(val, bf16)
    x, y0, ybar, xbar0 = _vectors(case, seed, n)
    if family == "heat":
        u = x.double()
        for _ in range(case["steps"]):
            u = _product(row, col, val, u, u)
        return {"y": u}
    y = _product(row, col, val, x, y0)
    if case.get("op") != "step":
        return {"y": y}
    return {"y": y, "xbar": _product(col, row, val, ybar, xbar0), "abar": ybar.double()[row] * x.double()[col]}
