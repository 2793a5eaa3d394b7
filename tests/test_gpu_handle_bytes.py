"""Device memory of a handle: csp_iterate's second vector is part of it only where the steps of
csp_iterate alternate between two vectors."""
import numpy as np
import pytest

from clspmv_b200 import CSP_METH_XPANEL, Cocktail, Handle, matrices as M
from tests.gpu_util import coo_of

pytestmark = pytest.mark.gpu

N = 60 * 60   # the padded lengths of x are those of N + 1 columns


def _bytes(fmt, method, width):
    h, _, r, c, v = M.laplacian_2d(60)
    hd = Handle(Cocktail.single(fmt, coo_of((h, width, r, c, v)), method), np.ones(width, np.float32))
    n = hd.device_bytes
    hd.free()
    return n


@pytest.mark.parametrize("fmt,method,steps", [("dia", 1, True), ("bdia", 1, True), ("ell", 1, True), ("csr", 2, True),
                                              ("csr", 0, False), ("csr", 3, False), ("csr", CSP_METH_XPANEL, False),
                                              ("coo", 0, False), ("ell", 0, False), ("sell", 1, False), ("bell", 0, False),
                                              ("bcsr", 0, False), ("sbell", 0, False)])
def test_second_vector_only_for_steps(fmt, method, steps):
    extra = _bytes(fmt, method, N) - _bytes(fmt, method, N + 1)
    x = 4 * ((N + 63) // 64 * 64 + 64)
    assert extra == (x if steps else 0)


def test_two_parts_have_no_second_vector():
    h, _, r, c, v = M.laplacian_2d(60)
    total = []
    for width in (N, N + 1):
        top = r < 1800
        both = Cocktail.single("csr", coo_of((h, width, r[top], c[top], v[top])), 2)
        rest = Cocktail.single("ell", coo_of((h, width, r[~top], c[~top], v[~top])), 1)
        both.s.ell, both.s.ifuseell, both.s.ell_meth_num = rest.s.ell, True, 1
        rest._owned = False
        hd = Handle(both, np.ones(width, np.float32))
        total.append(hd.device_bytes)
        hd.free()
    assert total[0] == total[1]
