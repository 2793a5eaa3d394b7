"""The streaming SpMM kernel with several block rows a lane group: enough block rows that every
lane split takes 2 to 8 of them, with empty rows, rows of several rings among short ones and a
last group that is not full, against the FP64 oracle; and neighbouring long rows, which must
not be summed one after the other."""
import ctypes as C

import numpy as np
import pytest
import torch

from clspmv_b200 import CSP_FLAG_BF16, Handle, capi
from clspmv_b200.matrices import csr_from_coo
from tests import _oracle
from tests.gpu_util import TOL
from tests.test_gpu_bf16 import bf16_round

pytestmark = pytest.mark.gpu


def _bcsr(degs, bs, seed, nbc=3001):
    """(struct, COO arrays): block rows of degs blocks at distinct random block columns."""
    rng = np.random.default_rng(seed)
    nbr, nb = len(degs), int(degs.sum())
    rp = np.zeros(nbr + 1, np.int32)
    rp[1:] = np.cumsum(degs)
    brow = np.repeat(np.arange(nbr), degs)
    first = rng.integers(0, nbc, nbr)
    bcol = (first[brow] + (np.arange(nb) - rp[brow])) % nbc     # distinct inside a row
    col = (bs * bcol).astype(np.int32)
    al = (nb + 31) // 32 * 32
    data = np.zeros((bs * bs, al), np.float32)
    data[:, :nb] = rng.standard_normal((bs * bs, nb))
    b = capi.bcsr_matrix()
    b.matinfo.width, b.matinfo.height, b.matinfo.nnz = bs * nbc, bs * nbr, bs * bs * nb
    b.bcsr_bwidth = b.bcsr_bheight = bs
    b.bcsr_row_num, b.bcsr_aligned_size, b.bcsr_block_num = nbr, al, nb
    flat = data.reshape(-1)
    b.bcsr_row_ptr, b.bcsr_col_id = capi.as_ptr(rp, C.c_int), capi.as_ptr(col, C.c_int)
    b.bcsr_data = capi.as_ptr(flat, C.c_float)
    b._arrays = (rp, col, flat)
    q = np.arange(bs * bs)
    r = (bs * brow[:, None] + q // bs).reshape(-1)
    c = (bs * bcol[:, None] + q % bs).reshape(-1)
    v = data[:, :nb].T.reshape(-1)
    order = np.lexsort((c, r))
    return b, (bs * nbr, bs * nbc, r[order].astype(np.int32), c[order].astype(np.int32), np.ascontiguousarray(v[order]))


def _degrees(nbr, seed):
    """0 to 3 blocks a row, and every 1,000th row 41: a third of a ring to several rings."""
    d = np.random.default_rng(seed).integers(0, 4, nbr)
    d[::1000] = 41
    d[nbr // 2:nbr // 2 + 9] = [0, 200, 0, 0, 1, 300, 301, 0, 2]
    return d


# k: block rows for 2 and for the most rows a group (a wave holds 37,888 / 18,944 / 9,472 / 4,736
# groups of 4 / 8 / 16 / 32 lanes, fewer for larger blocks)
ROWS = {4: (45_001, 155_003), 8: (22_001, 78_003), 12: (11_001, 40_003), 20: (6_001, 20_003), 32: (9_001, 39_003), 36: (9_001, 39_003)}


@pytest.mark.parametrize("bs", [1, 2, 3, 4, 6])
@pytest.mark.parametrize("k,most", [(k, i) for k in sorted(ROWS) for i in (0, 1)])
@pytest.mark.parametrize("bf16", [False, True])
def test_row_groups(bs, k, most, bf16):
    b, (h, w, r, c, v) = _bcsr(_degrees(ROWS[k][most], k + bs), bs, 5 * k + bs)
    rng = np.random.default_rng(1)
    X, Y0 = rng.uniform(-1, 1, (w, k)).astype(np.float32), rng.uniform(-1, 1, (h, k)).astype(np.float32)
    hd = Handle(None, X, Y0, CSP_FLAG_BF16 if bf16 else 0, nrhs=k, bcsr=b)
    hd.do_spmv(1)
    Y = hd.cpy_result_to_cpu().reshape(h, k)
    hd.free()
    rp, v = csr_from_coo(h, r), bf16_round(v) if bf16 else v
    for j in {0, 1, k // 2 + 1, k - 1}:   # one column of each lane position that ends a row differently
        yhat, bound = _oracle.fp64_spmv(h, w, rp, c, v, np.ascontiguousarray(X[:, j]), np.ascontiguousarray(Y0[:, j]))
        err, row = _oracle.max_rel_err(np.ascontiguousarray(Y[:, j]), yhat, bound)
        assert err <= TOL, f"column {j}: error {err:.3e} at row {row}"


def _time_us(degs, k, bs=3):
    b, (h, w, *_) = _bcsr(degs, bs, 3, nbc=20_000)
    hd = Handle(None, np.ones((w, k), np.float32), None, nrhs=k, bcsr=b)
    st = torch.cuda.Stream()
    hd.set_stream(st.cuda_stream)
    hd.do_spmv(2)
    st.synchronize()
    best = []
    for _ in range(5):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(st)
        hd.do_spmv(1)
        e1.record(st)
        st.synchronize()
        best.append(1e3 * e0.elapsed_time(e1))
    hd.free()
    return min(best)


@pytest.mark.parametrize("k", [16, 32])
def test_neighbouring_long_rows(k):
    """Eight block rows of 10,000 blocks among 50,000 short ones: next to one another they take
    about the time that they take far apart (in one lane group they would take 4 or 8 times as
    long; the bound leaves room for X rows shared or not)."""
    d = np.full(50_000, 3)
    near, far = d.copy(), d.copy()
    near[20_000:20_008] = 10_000
    far[3_000::6_000][:8] = 10_000
    assert near.sum() == far.sum()
    assert _time_us(near, k) <= 2 * _time_us(far, k)


def test_long_row_of_single_entries():
    """A row of 20,000 1x1 blocks at 4 right-hand sides has as many loads in flight as at 32, so it
    takes no longer (with one load a lane in flight it took 2.4 times as long)."""
    d = np.full(50_000, 3)
    d[::10_000] = 20_000
    assert _time_us(d, 4, bs=1) <= 1.6 * _time_us(d, 32, bs=1)


def test_two_passes_cost_twice_one():
    """4x4 blocks at k = 64 are two passes of the kernel at k = 32 (with 24 warps an SM they took
    2.4 times as long, the kernel that takes any k being short of registers)."""
    d = np.random.default_rng(5).integers(10, 31, 30_000)
    assert _time_us(d, 64, bs=4) <= 2.25 * _time_us(d, 32, bs=4)
