"""The four-row DIA / BDIA kernel's vector windows of x with x at every 4-byte alignment: bands of all four
residues and of groups of one to three diagonals, on matrices where some CTAs are interior (the kernel's
condition, restated here) and some are not, against the FP64 oracle.  The adjoint takes the
caller's vectors as they are, at independent alignments."""
import numpy as np
import pytest
import torch

from clspmv_b200 import CSP_FLAG_ADJOINT, CSP_FLAG_BF16, Cocktail, Handle
from clspmv_b200.matrices import csr_from_coo, vector
from tests import _oracle
from tests.gpu_util import TOL, coo_of
from tests.test_gpu_bf16 import bf16_round
from tests.test_gpu_dia_rows import _banded

pytestmark = pytest.mark.gpu

BANDS = {
    "residues": [-101, -100, -50, -49, -48, -3, -2, 5, 6, 7, 8, 103, 104],
    "tri": [-1, 0, 1],
    "seven": list(range(-3, 4)),
    "laplacian": [-700, -1, 0, 1, 700],
}
N = 12_001


def _interior_ctas(n, offsets):
    """CTAs of 1,024 rows that take the vector path (dia_rows_kernel) for an n x n matrix."""
    return [rb for rb in range(0, n, 1024) if rb + min(offsets) - 3 >= 0 and rb + 1020 + max(offsets) + 12 <= n]


@pytest.mark.parametrize("band", sorted(BANDS))
@pytest.mark.parametrize("fmt", ["dia", "bdia"])
@pytest.mark.parametrize("shift_y", [0, 1, 2, 3])
@pytest.mark.parametrize("shift_x", [0, 1, 2, 3])
@pytest.mark.parametrize("bf16", [False, True])
def test_windows_at_every_alignment(band, fmt, shift_y, shift_x, bf16):
    offs = BANDS[band]
    assert len(offs) * 3 >= 5 * sum(1 for i, o in enumerate(offs) if i == 0 or offs[i - 1] != o - 1)   # grouped, not one by one
    interior = _interior_ctas(N, [-o for o in offs])
    assert 0 < len(interior) < (N + 1023) // 1024
    case = _banded(N, N, offs, 398)
    h, w, r, c, v = case
    ybar, xbar0 = vector(h, seed=99), vector(w, seed=100)
    hd = Handle(Cocktail.single(fmt, coo_of(case), 1), vector(w, seed=101), None, CSP_FLAG_ADJOINT | (CSP_FLAG_BF16 if bf16 else 0))
    yb, xb = torch.zeros(h + 4, device="cuda"), torch.zeros(w + 4, device="cuda")
    yb[shift_y:shift_y + h] = torch.from_numpy(ybar).cuda()
    xb[shift_x:shift_x + w] = torch.from_numpy(xbar0).cuda()
    torch.cuda.synchronize()
    hd.spmv_adjoint(yb[shift_y:].data_ptr(), xb[shift_x:].data_ptr(), None)
    hd.synchronize()
    got = xb[shift_x:shift_x + w].cpu().numpy()
    assert float(xb[:shift_x].abs().sum() + xb[shift_x + w:].abs().sum()) == 0.0   # nothing beside the vector
    hd.free()
    want, bound = _oracle.fp64_spmv(h, w, csr_from_coo(h, r), c, bf16_round(v) if bf16 else v, ybar, xbar0, transpose=True)
    err, row = _oracle.max_rel_err(got, want, bound)
    assert err <= TOL, f"error {err:.3e} at column {row}"
