"""Set-up of SpMM handles: blocks become records on the host or on the device, with the
temporary inside or outside their allocation, at the sizes where that changes; and its time."""
import time

import numpy as np
import pytest
import torch

from clspmv_b200 import CSP_FLAG_BF16, Handle
from clspmv_b200.matrices import csr_from_coo
from tests import _oracle
from tests.gpu_util import TOL
from tests.test_gpu_bf16 import bf16_round
from tests.test_gpu_spmm_groups import _bcsr

pytestmark = pytest.mark.gpu


# blocks a row: 131,072 words of records are made on the host (10,890 3x3 blocks FP32, 21,813 BF16 with the
# zero records behind them), 16 MiB of columns and planes fit the temporary inside (419,430 blocks, 762,600)
@pytest.mark.parametrize("bf16,blocks", [(False, 10_800), (False, 11_000), (False, 419_000), (False, 420_000), (True, 21_800),
                                         (True, 21_900), (True, 762_000), (True, 763_000)])
def test_records(bf16, blocks):
    k = 4
    b, (h, w, r, c, v) = _bcsr(np.full(blocks // 20, 20), 3, 11)
    rng = np.random.default_rng(12)
    X, Y0 = rng.uniform(-1, 1, (w, k)).astype(np.float32), rng.uniform(-1, 1, (h, k)).astype(np.float32)
    hd = Handle(None, X, Y0, CSP_FLAG_BF16 if bf16 else 0, nrhs=k, bcsr=b)
    hd.do_spmv(1)
    Y = hd.cpy_result_to_cpu().reshape(h, k)
    hd.free()
    rp, v = csr_from_coo(h, r), bf16_round(v) if bf16 else v
    for j in range(k):
        yhat, bound = _oracle.fp64_spmv(h, w, rp, c, v, np.ascontiguousarray(X[:, j]), np.ascontiguousarray(Y0[:, j]))
        err, row = _oracle.max_rel_err(np.ascontiguousarray(Y[:, j]), yhat, bound)
        assert err <= TOL, f"column {j}: error {err:.3e} at row {row}"


def test_time():
    """1,000 block rows of 20 6x6 blocks: the set-up takes at most 1.6 times that of the same handle for five
    right-hand sides, whose kernel reads the caller's element planes (one B200: 1.0 and 0.95 ms; 2.0 with
    a copy for each plane into a temporary of its own)."""
    b, (h, w, *_) = _bcsr(np.full(1_000, 20), 6, 13)
    ms = {}
    for k in (4, 5):
        X, times = np.ones((w, k), np.float32), []
        for _ in range(30):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            hd = Handle(None, X, None, nrhs=k, bcsr=b)
            times.append(1e3 * (time.perf_counter() - t0))
            hd.free()
        ms[k] = min(times)
    assert ms[4] <= 1.6 * ms[5], ms


def test_device_nearly_full():
    """1 M 3x3 blocks (40 MB of columns and planes) with 56 to 72 MB left on the device: no room for records
    and their temporary, so the handle keeps the element planes, and the result is the same."""
    k = 4
    b, (h, w, r, c, v) = _bcsr(np.full(50_000, 20), 3, 14)
    rng = np.random.default_rng(15)
    X, Y0 = rng.uniform(-1, 1, (w, k)).astype(np.float32), rng.uniform(-1, 1, (h, k)).astype(np.float32)
    small, _ = _bcsr(np.full(50, 20), 3, 16)
    for n in (4, 5):   # loads the kernels of both layouts
        hd = Handle(None, np.ones((9_003, n), np.float32), None, nrhs=n, bcsr=small)
        hd.do_spmv(1)
        hd.free()
    torch.cuda.empty_cache()
    fill, mib = [], 1 << 20
    try:
        fill.append(torch.empty(torch.cuda.mem_get_info()[0] - 66 * mib, dtype=torch.uint8, device="cuda"))
        left = torch.cuda.mem_get_info()[0] // mib
        assert 54 <= left <= 70, left
        hd = Handle(None, X, Y0, nrhs=k, bcsr=b)
        hd.do_spmv(1)
        Y = hd.cpy_result_to_cpu().reshape(h, k)
        hd.free()
    finally:
        fill.clear()
        torch.cuda.empty_cache()
    rp = csr_from_coo(h, r)
    for j in range(k):
        yhat, bound = _oracle.fp64_spmv(h, w, rp, c, v, np.ascontiguousarray(X[:, j]), np.ascontiguousarray(Y0[:, j]))
        err, row = _oracle.max_rel_err(np.ascontiguousarray(Y[:, j]), yhat, bound)
        assert err <= TOL, f"column {j}: error {err:.3e} at row {row}"
