"""The four-row ELL kernel around the slots that it requests ahead (5): 1 to 23 slots, rows that
are no multiple of 4, against the FP64 oracle; and rows of many slots, whose gathers have to
stay in flight together."""
import numpy as np
import pytest

from clspmv_b200 import CSP_FLAG_BF16, Cocktail, Handle
from clspmv_b200.matrices import csr_from_coo, vector
from tests import _oracle
from tests.gpu_timing import spmv_us
from tests.gpu_util import TOL, coo_of
from tests.test_gpu_bf16 import bf16_round

pytestmark = pytest.mark.gpu


def _uniform(n, w, slots, seed):
    rng = np.random.default_rng(seed)
    c = np.sort(rng.integers(0, w, (n, slots)), axis=1).astype(np.int32)
    return n, w, np.repeat(np.arange(n, dtype=np.int32), slots), c.reshape(-1), rng.standard_normal(n * slots).astype(np.float32)


@pytest.mark.parametrize("slots", [1, 2, 4, 5, 6, 8, 9, 10, 13, 23])
@pytest.mark.parametrize("n,w", [(1, 40), (1027, 513)])
@pytest.mark.parametrize("bf16", [False, True])
def test_slots(slots, n, w, bf16):
    case = _uniform(n, w, slots, 7 * slots + n)
    h, w, r, c, v = case
    x, y0 = vector(w, seed=1), vector(h, seed=2)
    hd = Handle(Cocktail.single("ell", coo_of(case), 1), x, y0, CSP_FLAG_BF16 if bf16 else 0)
    hd.do_spmv(1)
    y = hd.cpy_result_to_cpu()
    hd.free()
    yhat, bound = _oracle.fp64_spmv(h, w, csr_from_coo(h, r), c, bf16_round(v) if bf16 else v, x, y0)
    err, row = _oracle.max_rel_err(y, yhat, bound)
    assert err <= TOL, f"error {err:.3e} at row {row}"


def test_many_slots_keep_their_gathers_in_flight():
    """50,000 rows of 40 entries at random columns: ELL takes about as long as CSR (10.5 us each on one
    B200; 23.3 with a test between the gathers)."""
    case = _uniform(50_000, 50_000, 40, 3)
    us = {}
    for fmt, method in (("ell", 1), ("csr", 2)):
        hd = Handle(Cocktail.single(fmt, coo_of(case), method), vector(50_000, seed=1))
        us[fmt] = spmv_us(hd)
        hd.free()
    assert us["ell"] <= 1.5 * us["csr"], us
