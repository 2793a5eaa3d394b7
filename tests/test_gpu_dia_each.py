"""Diagonals that mostly stand alone (the kernel that takes them one by one) around the rule that
chooses it, at row counts off every unit, rectangular shapes and x / y at 4-byte alignment,
against the FP64 oracle; the same steps as csp_iterate; and enough bytes in flight."""
import ctypes as C

import numpy as np
import pytest
import torch

from clspmv_b200 import CSP_FLAG_ADJOINT, CSP_FLAG_BF16, CSP_FLAG_GRAPH, Cocktail, Handle, capi
from clspmv_b200.matrices import csr_from_coo, vector
from tests import _oracle
from tests.gpu_timing import spmv_us
from tests.gpu_util import TOL, coo_of
from tests.test_gpu_bf16 import bf16_round
from tests.test_gpu_dia_rows import _banded
from tests.test_gpu_iterate import _iterated, _manual, _scaled

pytestmark = pytest.mark.gpu

BANDS = {
    "two": [-7, 5],
    "seven_in_five": [-90, -20, -1, 0, 1, 20, 90],
    "five_in_three": [-20, -1, 0, 1, 20],        # the other kernel's side of the rule
    "nine": [-1003, -502, -51, -9, 0, 6, 53, 604, 1005],
    "unsorted_twelve": [30 * i for i in range(-6, 6)],
}


@pytest.mark.parametrize("band", sorted(BANDS))
@pytest.mark.parametrize("size", [(331, 331), (1025, 1025), (5003, 5003), (3002, 6001), (4010, 4003)])
@pytest.mark.parametrize("fmt", ["dia", "bdia"])
@pytest.mark.parametrize("bf16", [False, True])
def test_dia_each(band, size, fmt, bf16):
    case = _banded(*size, [o for o in BANDS[band] if -size[0] < o < size[1]] or [0], 195)
    h, w, r, c, v = case
    x, y0 = vector(w, seed=96), vector(h, seed=97)
    hd = Handle(Cocktail.single(fmt, coo_of(case), 1), x, y0, CSP_FLAG_BF16 if bf16 else 0)
    hd.do_spmv(1)
    y = hd.cpy_result_to_cpu()
    hd.free()
    yhat, bound = _oracle.fp64_spmv(h, w, csr_from_coo(h, r), c, bf16_round(v) if bf16 else v, x, y0)
    err, row = _oracle.max_rel_err(y, yhat, bound)
    assert err <= TOL, f"error {err:.3e} at row {row}"


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_alignment(shift):
    """A^T ybar with ybar and xbar `shift` and `3 - shift` floats past a 16-byte boundary."""
    case = _banded(5001, 5001, BANDS["nine"], 198)
    h, w, r, c, v = case
    ybar, xbar0 = vector(h, seed=99), vector(w, seed=100)
    hd = Handle(Cocktail.single("dia", coo_of(case), 1), vector(w, seed=101), None, CSP_FLAG_ADJOINT)
    yb, xb = torch.zeros(h + 3, device="cuda"), torch.zeros(w + 3, device="cuda")
    yb[shift:shift + h] = torch.from_numpy(ybar).cuda()
    xb[3 - shift:3 - shift + w] = torch.from_numpy(xbar0).cuda()
    torch.cuda.synchronize()
    hd.spmv_adjoint(yb[shift:].data_ptr(), xb[3 - shift:].data_ptr(), None)
    hd.synchronize()
    got = xb[3 - shift:3 - shift + w].cpu().numpy()
    hd.free()
    want, bound = _oracle.fp64_spmv(h, w, csr_from_coo(h, r), c, v, ybar, xbar0, transpose=True)
    err, row = _oracle.max_rel_err(got, want, bound)
    assert err <= TOL, f"error {err:.3e} at column {row}"


@pytest.mark.parametrize("k", [1, 2, 33])
@pytest.mark.parametrize("flags", [0, CSP_FLAG_GRAPH, CSP_FLAG_BF16 | CSP_FLAG_GRAPH])
def test_steps(k, flags):
    case = _scaled(_banded(2_025, 2_025, BANDS["nine"], 199), 0.05)
    mat = Cocktail.single("dia", coo_of(case), 1)
    x, y0 = vector(2_025, seed=6), vector(2_025, seed=7)
    assert _iterated(mat, x, y0, k, flags).tobytes() == _manual(mat, x, y0, k, flags & CSP_FLAG_BF16).tobytes()


@pytest.mark.parametrize("bf16,gbs", [(False, 3700), (True, 2000)])
def test_bytes_in_flight(bf16, gbs):
    """27 diagonals 37 apart on 2 M rows (one B200: 4,900 GB/s of values FP32, 2,800 BF16; in groups of
    one diagonal with two groups in flight 2,900 and 1,700)."""
    n, nd = 2_000_000, 27
    off = np.array([37 * (i - 13) for i in range(nd)], np.int32)
    data = np.ones(nd * n, np.float32)
    mat = Cocktail(n, n, nd * n)
    d = mat.s.dia
    d.matinfo.width = d.matinfo.height = n
    d.matinfo.nnz = nd * n
    d.dia_num, d.dia_length_aligned = nd, n
    d.dia_offsets, d.dia_data = capi.as_ptr(off, C.c_int), capi.as_ptr(data, C.c_float)
    mat.s.ifusedia, mat.s.dia_meth_num, mat._owned = True, 1, False
    hd = Handle(mat, None, None, CSP_FLAG_BF16 if bf16 else 0)
    us = spmv_us(hd)
    hd.free()
    assert nd * n * (2 if bf16 else 4) / us / 1e3 >= gbs, f"{us} us"
