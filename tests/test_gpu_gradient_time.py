"""Value gradients of many slots as a kernel of many short CTAs."""
import numpy as np
import pytest
import torch

from clspmv_b200 import CSP_FLAG_ADJOINT, Cocktail, Handle, matrices as M
from tests.gpu_util import coo_of

pytestmark = pytest.mark.gpu


def test_gradients_of_a_stencil():
    """3.2 M CSR slots: the gradients take at most 1.8 times the transposed product's time (one B200: 8.4
    and 6.2 us; 13.9 where each of 12,500 CTAs lets the next kernel in)."""
    case = M.stencil_27(50)
    h, w = case[0], case[1]
    hd = Handle(Cocktail.single("csr", coo_of(case), 2), np.ones(w, np.float32), None, CSP_FLAG_ADJOINT)
    st = torch.cuda.Stream()
    hd.set_stream(st.cuda_stream)
    ybar, xbar = torch.rand(h, device="cuda"), torch.zeros(w, device="cuda")
    abar = torch.zeros(hd.adjoint_slots, device="cuda")
    torch.cuda.synchronize()

    def best(xp, ap):
        times = []
        for _ in range(8):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(st)
            for _ in range(20):
                hd.spmv_adjoint(ybar.data_ptr(), xp, ap)
            e1.record(st)
            st.synchronize()
            times.append(e0.elapsed_time(e1))
        return min(times[1:])

    assert best(None, abar.data_ptr()) <= 1.8 * best(xbar.data_ptr(), None)
