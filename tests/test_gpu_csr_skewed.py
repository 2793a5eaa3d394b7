"""CSR adaptive blocks whose rows are much longer than the block's lane groups take (summed
by a warp each): one long row among many short ones at every group width, thresholds hit
exactly, several long rows in one block, rows of a whole block and longer, against the FP64
oracle, and the same bits on a second run."""
import numpy as np
import pytest

from clspmv_b200 import CSP_FLAG_BF16, Cocktail, matrices as M
from tests.gpu_util import TOL, coo_of, run, vecs
from tests import _oracle
from tests.test_gpu_bf16 import bf16_round

pytestmark = pytest.mark.gpu


def _rows(lens, w, seed):
    rng = np.random.default_rng(seed)
    r = np.repeat(np.arange(len(lens), dtype=np.int32), lens)
    c = np.concatenate([np.sort(rng.choice(w, n, replace=False)) for n in lens] or [np.zeros(0)]).astype(np.int32)
    return len(lens), w, r, c, rng.standard_normal(r.size).astype(np.float32)


CASES = {
    # 256 rows a block: one lane a row, threshold 32
    "at_16": _rows([16] * 100 + [17] + [1] * 300, 4000, 1),
    "at_32": _rows([32] * 40 + [33] + [1] * 300 + [32, 33, 34] + [2] * 200, 4000, 8),
    "one_long": _rows([1] * 128 + [1700] + [1] * 127 + [0] * 300, 4000, 2),
    "many_long": _rows(([2] * 20 + [130, 0, 17]) * 30, 4000, 3),
    # 2, 4, 8, 16, 32 lanes a row: thresholds 64 .. 1024
    "two_lanes": _rows(([14] * 100 + [33, 65, 64, 500]) * 6, 4000, 4),
    "eight_lanes": _rows(([60] * 20 + [129, 257, 256, 400]) * 8, 4000, 5),
    "wide_rows": _rows([500, 600, 900] * 5 + [2040, 2041, 1, 3900, 0, 513, 512, 1015], 4000, 6),
    "zipf": M.zipf_rows(20_000, seed=7, max_len=3000),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("bf16", [False, True])
def test_skewed_blocks(name, bf16):
    case = CASES[name]
    h, w, r, c, v = case
    x, y0 = vecs(h, w, seed=13)
    mat = Cocktail.single("csr", coo_of(case), 2)
    flags = CSP_FLAG_BF16 if bf16 else 0
    y = run(mat, x, y0, flags=flags)
    rp = M.csr_from_coo(h, r)
    yhat, bound = _oracle.fp64_spmv(h, w, rp, c, bf16_round(v) if bf16 else v, x, y0)
    err, row = _oracle.max_rel_err(y, yhat, bound)
    assert err <= TOL, f"error {err:.3e} at row {row}"
    assert run(mat, x, y0, flags=flags).tobytes() == y.tobytes()
