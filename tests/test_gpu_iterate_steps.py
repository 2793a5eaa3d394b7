"""csp_iterate where its steps alternate between two vectors (one DIA, BDIA, ELL or CSR
adaptive part that covers every row): identical bits to the loop driven call by call, for
step counts around the alternation and the graph chunk, and with calls in between; and the
cases that must not alternate (a part shorter than the matrix, two parts)."""
import numpy as np
import pytest

from clspmv_b200 import CSP_FLAG_BF16, CSP_FLAG_GRAPH, Cocktail, Handle, matrices as M
from tests.gpu_util import coo_of, vecs
from tests.test_gpu_iterate import _iterated, _manual, _scaled

pytestmark = pytest.mark.gpu

CASES = {
    "grid": _scaled(M.laplacian_2d(45), 0.1),      # 2,025 rows: no multiple of 4
    "zipf": _scaled(M.zipf_rows(9_001, seed=42, max_len=3000), 0.05),   # rows longer than a work block
}
FORMATS = [("grid", "dia", 1), ("grid", "bdia", 1), ("grid", "ell", 1), ("grid", "csr", 2), ("zipf", "csr", 2)]


@pytest.mark.parametrize("name,fmt,method", FORMATS)
@pytest.mark.parametrize("k", [1, 2, 3, 32, 33, 34, 65])
@pytest.mark.parametrize("flags", [0, CSP_FLAG_GRAPH, CSP_FLAG_BF16 | CSP_FLAG_GRAPH])
def test_steps_match_call_by_call(name, fmt, method, k, flags):
    case = CASES[name]
    mat = Cocktail.single(fmt, coo_of(case), method)
    x, y0 = vecs(case[0], case[1], seed=6)
    assert _iterated(mat, x, y0, k, flags).tobytes() == _manual(mat, x, y0, k, flags & CSP_FLAG_BF16).tobytes()


@pytest.mark.parametrize("graph", [False, True])
def test_iterate_between_other_calls(graph):
    """iterate, do_spmv and a new vector in turn: x and res hold what the loop leaves."""
    case = CASES["grid"]
    h, w = case[0], case[1]
    x, y0 = vecs(h, w, seed=7)
    out = []
    for manual in (False, True):
        hd = Handle(Cocktail.single("dia", coo_of(case), 1), x, y0, CSP_FLAG_GRAPH if graph else 0)
        for part in range(2):
            if manual:
                for _ in range(5):
                    hd.do_spmv(1)
                    hd.cpy_vector_from_gpu(hd.res_ptr, h)
            else:
                hd.iterate(5)
            hd.do_spmv(1)                    # reads the vector the loop left
            hd.cpy_vector_from_cpu(x)
        hd.do_spmv(1)
        out.append(hd.cpy_result_to_cpu())
        hd.free()
    assert out[0].tobytes() == out[1].tobytes()


def test_short_part_and_two_parts():
    """Rows past a part's height keep their value; two parts accumulate in turn."""
    h, w, r, c, v = CASES["grid"]
    top = r < 2000
    short = Cocktail.single("csr", coo_of((2000, w, r[top], c[top], v[top])), 2)
    short.s.mat_height, short.s.mat_width = h, w
    both = Cocktail.single("csr", coo_of((h, w, r[top], c[top], v[top])), 2)
    rest = Cocktail.single("ell", coo_of((h, w, r[~top], c[~top], v[~top])), 1)
    both.s.ell, both.s.ifuseell, both.s.ell_meth_num = rest.s.ell, True, 1
    rest._owned = False   # both frees the ELL arrays
    x, y0 = vecs(h, w, seed=8)
    for mat in (short, both):
        a = _iterated(mat, x, y0, 6, CSP_FLAG_GRAPH)
        b = _manual(mat, x, y0, 6)
        assert a.tobytes() == b.tobytes()
    assert np.isfinite(a).all()
