"""The streaming SpMM kernel (k a multiple of 4) where its chunks, rings and row groups
end: block rows of 0 blocks to several rings, a single block row, partial last blocks,
every block shape and every split of the right-hand sides, against the FP64 oracle."""
import ctypes as C

import numpy as np
import pytest

from clspmv_b200 import CSP_FLAG_BF16, Handle, capi
from tests.gpu_util import coo_of
from tests.test_gpu_bf16 import bf16_round
from tests.test_gpu_spmm import _check_cols, _ragged, _xy

pytestmark = pytest.mark.gpu

CASES = {
    "ragged": _ragged(4_001, 3_007, 700, 91),
    "one_row": _ragged(1, 500, 37, 92),
    "few_rows": _ragged(70, 65, 64, 93),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("bs", [1, 2, 3, 4, 6])
@pytest.mark.parametrize("k", [4, 8, 12, 16, 20, 32, 36])
@pytest.mark.parametrize("bf16", [False, True])
def test_generic_bcsr_stream(name, bs, k, bf16):
    case = CASES[name]
    h, w, r, c, v = case
    b = capi.bcsr_matrix()
    assert capi.lib().csp_coo2bcsr(coo_of(case).ref(), C.byref(b), bs, bs, 32) == 0
    X, Y0 = _xy(h, w, k, seed=12)
    hd = Handle(None, X, Y0, flags=CSP_FLAG_BF16 if bf16 else 0, nrhs=k, bcsr=b)
    hd.do_spmv(1)
    Y = hd.cpy_result_to_cpu()
    hd.free()
    capi.lib().csp_free_bcsr_matrix(C.byref(b))
    _check_cols(case, Y, X, Y0, k, values=bf16_round(v) if bf16 else None)
