"""csp_coo_spmv_noalloc where its scratch pairs and chunks matter: rows over one to many
chunks (the fix-up follows a run through several warps of pairs), rows ending on chunk and
tile boundaries, entry counts around tiles, chunks and the change of the chunk size, empty rows
between, and indices outside the matrix, against the FP64 oracle, twice with the same bits."""
import numpy as np
import pytest
import torch

from clspmv_b200 import capi
from clspmv_b200.matrices import csr_from_coo, vector
from tests import _oracle
from tests.gpu_util import TOL

pytestmark = pytest.mark.gpu

LENS = {
    "one_row": [5000],
    "row_of_all_pairs": [3, 40_000, 2],
    "chunk_rows": [256] * 40,
    "chunk_rows_512": [512] * 33 + [1],
    "tile_rows": [128] * 70,
    "off_by_one": [127, 129, 255, 257, 511, 513, 1, 1023, 1025] * 5,
    "long_and_short": ([1] * 300 + [0, 0, 9000, 0] + [3] * 50 + [4200]) * 3,
    "pairs_of_runs": [700] * 64 + [16_384] + [700] * 64,
    "tail_1": [1] * 1281,
}


def _call(h, w, dev, y):
    capi.check(capi.lib().csp_coo_spmv_noalloc(h, w, dev[0].numel(), dev[0].data_ptr(), dev[1].data_ptr(), dev[2].data_ptr(),
                                               dev[3].data_ptr(), y.data_ptr(), None), "noalloc")


@pytest.mark.parametrize("name", sorted(LENS))
@pytest.mark.parametrize("extra", [0, 1_300_000])   # past the change of the chunk size
def test_noalloc_pairs(name, extra):
    lens = np.array(LENS[name] + [1000] * (extra // 1000), np.int64)
    rng = np.random.default_rng(41)
    h, w = lens.size, 50_000
    r = np.repeat(np.arange(h, dtype=np.int32), lens)
    c = rng.integers(0, w, r.size).astype(np.int32)
    v = rng.standard_normal(r.size).astype(np.float32)
    x, y0 = vector(w, seed=42), vector(h, seed=43)
    dev = [torch.from_numpy(a).cuda() for a in (r, c, v, x)]
    out = []
    for _ in range(2):
        y = torch.from_numpy(y0).cuda()
        torch.cuda.synchronize()
        _call(h, w, dev, y)
        torch.cuda.synchronize()
        out.append(y.cpu().numpy())
    assert out[0].tobytes() == out[1].tobytes()
    want, bound = _oracle.fp64_spmv(h, w, csr_from_coo(h, r), c, v, x, y0)
    err, row = _oracle.max_rel_err(out[0], want, bound)
    assert err <= TOL, f"{err:.3e} at {row}"


def test_noalloc_outside_indices():
    """Entries with a row or column outside the matrix add nothing."""
    rng = np.random.default_rng(44)
    h, w, n = 900, 700, 20_000
    r = np.sort(rng.integers(-3, h + 3, n)).astype(np.int32)
    c = rng.integers(-2, w + 2, n).astype(np.int32)
    v = rng.standard_normal(n).astype(np.float32)
    ok = (r >= 0) & (r < h) & (c >= 0) & (c < w)
    x, y0 = vector(w, seed=45), vector(h, seed=46)
    dev = [torch.from_numpy(a).cuda() for a in (r, c, v, x)]
    y = torch.from_numpy(y0).cuda()
    torch.cuda.synchronize()
    _call(h, w, dev, y)
    torch.cuda.synchronize()
    want, bound = _oracle.fp64_spmv(h, w, csr_from_coo(h, r[ok]), c[ok], v[ok], x, y0)
    err, row = _oracle.max_rel_err(y.cpu().numpy(), want, bound)
    assert err <= TOL, f"{err:.3e} at {row}"
