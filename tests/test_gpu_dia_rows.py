"""The four-row DIA / BDIA kernel at its edges: bands of 1 to 7 adjacent diagonals (groups of
at most 3), offsets of every residue, unsorted diagonals, no interior CTA at all, rows that
are no multiple of 4 or of a CTA, rectangular shapes, and x / y at 4-byte alignment (the
adjoint's vectors), against the FP64 oracle."""
import numpy as np
import pytest
import torch

from clspmv_b200 import CSP_FLAG_ADJOINT, CSP_FLAG_BF16, Cocktail, Handle
from clspmv_b200.matrices import csr_from_coo, vector
from tests import _oracle
from tests.gpu_util import TOL, coo_of
from tests.test_gpu_bf16 import bf16_round

pytestmark = pytest.mark.gpu


def _banded(h, w, offsets, seed):
    rng = np.random.default_rng(seed)
    r = np.concatenate([np.arange(max(0, -o), min(h, w - o), dtype=np.int64) for o in offsets if max(0, -o) < min(h, w - o)])
    c = np.concatenate([np.arange(max(0, -o), min(h, w - o), dtype=np.int64) + o for o in offsets if max(0, -o) < min(h, w - o)])
    order = np.lexsort((c, r))
    return h, w, r[order].astype(np.int32), c[order].astype(np.int32), rng.uniform(0.5, 1.5, r.size).astype(np.float32)


BANDS = {
    "one": [0],
    "tri": [-1, 0, 1],
    "seven": list(range(-3, 4)),
    "laplacian": [-100, -1, 0, 1, 100],
    "residues": [-1029, -514, -3, -2, 5, 6, 7, 8, 1030, 2051],
    "many": [o for b in range(-40, 41, 4) for o in (b * 9, b * 9 + 1, b * 9 + 2)],
}
SIZES = [(1, 1), (37, 37), (1023, 1023), (5001, 5001), (4010, 4003), (3002, 6001)]
CASES = [(b, s) for b in sorted(BANDS) for s in SIZES if not (b == "many" and s == (37, 37))]   # refused: too much padding


@pytest.mark.parametrize("band,size", CASES)
@pytest.mark.parametrize("fmt", ["dia", "bdia"])
@pytest.mark.parametrize("bf16", [False, True])
def test_dia_rows(band, size, fmt, bf16):
    offs = [o for o in BANDS[band] if -size[0] < o < size[1]] or [0]   # no offset inside a 1 x 1 matrix
    case = _banded(*size, offs, 95)
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
def test_dia_rows_alignment(shift):
    """A^T ybar with ybar and xbar `shift` floats past a 16-byte boundary."""
    case = _banded(5001, 5001, BANDS["residues"], 98)
    h, w, r, c, v = case
    ybar, xbar0 = vector(h, seed=99), vector(w, seed=100)
    hd = Handle(Cocktail.single("dia", coo_of(case), 1), vector(w, seed=101), None, CSP_FLAG_ADJOINT)
    yb, xb = torch.zeros(h + shift, device="cuda"), torch.zeros(w + shift, device="cuda")
    yb[shift:] = torch.from_numpy(ybar).cuda()
    xb[shift:] = torch.from_numpy(xbar0).cuda()
    torch.cuda.synchronize()
    hd.spmv_adjoint(yb[shift:].data_ptr(), xb[shift:].data_ptr(), None)
    hd.synchronize()
    got = xb[shift:].cpu().numpy()
    hd.free()
    want, bound = _oracle.fp64_spmv(h, w, csr_from_coo(h, r), c, v, ybar, xbar0, transpose=True)
    err, row = _oracle.max_rel_err(got, want, bound)
    assert err <= TOL, f"error {err:.3e} at column {row}"
