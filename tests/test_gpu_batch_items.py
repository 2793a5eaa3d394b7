"""The batch kernel's work list where it can go wrong: items with rows far longer than their
lane groups take (summed by the whole warp), fewer items than warps, more items than the one
a time tail, and counters that the kernel itself resets -- several runs in a row, in both
directions and in turn, give the oracle's result and the same bits."""
import numpy as np
import pytest

from clspmv_b200 import CSP_FLAG_ADJOINT, CSP_FLAG_BF16, CSP_FLAG_GRAPH, matrices as M
from clspmv_b200.batch import (CSP_BATCH_ADJ, CSP_BATCH_FWD, CSP_BV_ABAR, CSP_BV_X, CSP_BV_XBAR, CSP_BV_Y, CSP_BV_YBAR, Batch)
from clspmv_b200.capi import CSP_BFMT_CSR
from tests import _oracle
from tests.gpu_util import TOL, coo_of
from tests.test_gpu_bf16 import bf16_round
from tests.test_gpu_csr_skewed import _rows

pytestmark = pytest.mark.gpu

SKEWED = [
    _rows([1] * 30 + [200] + [0] * 20 + [17, 16, 18], 900, 1),
    _rows([2] * 15 + [100, 33, 32], 900, 2),
    _rows([60, 190, 1, 0, 65, 64, 129], 900, 3),
    _rows([252, 253, 1, 600, 251, 1], 900, 4),
    _rows([1] * 63 + [180] + [1] * 64, 900, 5),
]
BATCHES = {
    "skewed": (SKEWED, CSP_BFMT_CSR),
    "few_items": ([M.zipf_rows(50, seed=3, max_len=12), M.laplacian_2d(9), M.block_3x3(20, deg=(2, 5), band=9, seed=4)], -1),
    "many_items": ([M.zipf_rows(150_000, s=1.85, max_len=3000, seed=i) for i in range(4)], CSP_BFMT_CSR),
    "mixed": (SKEWED + [M.laplacian_2d(60), M.block_3x3(900, seed=6), M.zipf_rows(4000, s=1.85, max_len=900, seed=7)], -1),
}


@pytest.mark.parametrize("name", sorted(BATCHES))
@pytest.mark.parametrize("flags", [0, CSP_FLAG_GRAPH, CSP_FLAG_BF16])
def test_batch_items(name, flags):
    mats, fmt = BATCHES[name]
    b = Batch([coo_of(m) for m in mats], flags=flags | CSP_FLAG_ADJOINT, fmt=fmt)
    x = M.vector(int(b.x_off[-1]), seed=31)
    ybar = M.vector(int(b.y_off[-1]), seed=32)
    y0, xbar0 = M.vector(ybar.size, seed=33), M.vector(x.size, seed=34)
    b.copy_in(CSP_BV_X, x)
    b.copy_in(CSP_BV_YBAR, ybar)
    first = None
    for what in (3, CSP_BATCH_FWD, CSP_BATCH_ADJ, 3, 3):
        b.copy_in(CSP_BV_Y, y0)
        b.copy_in(CSP_BV_XBAR, xbar0)
        b.run(what)
        y, xbar, abar = b.copy_out(CSP_BV_Y), b.copy_out(CSP_BV_XBAR), b.copy_out(CSP_BV_ABAR)
        if first is None:
            first = (y, xbar, abar)
        if what & CSP_BATCH_FWD:
            assert y.tobytes() == first[0].tobytes()
        if what & CSP_BATCH_ADJ:
            assert xbar.tobytes() == first[1].tobytes() and abar.tobytes() == first[2].tobytes()
    b.synchronize()
    for i, m in enumerate(mats):
        h, w, r, c, v = m
        order = np.lexsort((c, r))
        r, c, v = r[order], c[order], (bf16_round(v) if flags & CSP_FLAG_BF16 else v)[order]
        rp = M.csr_from_coo(h, r)
        xs, ys = slice(int(b.x_off[i]), int(b.x_off[i + 1])), slice(int(b.y_off[i]), int(b.y_off[i + 1]))
        for out, vec, start, tr in ((first[0][ys], x[xs], y0[ys], False), (first[1][xs], ybar[ys], xbar0[xs], True)):
            want, bound = _oracle.fp64_spmv(h, w, rp, c, v, vec, start, transpose=tr)
            err, row = _oracle.max_rel_err(out, want, bound)
            assert err <= TOL, f"matrix {i} transpose {tr}: {err:.3e} at {row}"
    b.free()
