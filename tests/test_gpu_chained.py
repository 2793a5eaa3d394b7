"""Launches with programmatic stream serialization (csrc/launch.h): results must not depend
on what runs before and after them in the stream.  Torch kernels write x, y and ybar right
before a call and read and overwrite the results right after it, many times without a
synchronization, with matrices large enough that neighbouring kernels overlap; the same
inside a captured graph."""
import numpy as np
import pytest
import torch

from clspmv_b200 import CSP_FLAG_ADJOINT, Cocktail, Handle, matrices as M
from clspmv_b200.batch import CSP_BATCH_ADJ, CSP_BATCH_FWD, Batch
from tests.gpu_util import coo_of

pytestmark = pytest.mark.gpu

CASES = {
    "zipf": M.zipf_rows(60_000, seed=21, max_len=5000),
    "grid": M.laplacian_2d(250),
}
FORMATS = [("grid", "dia", 1), ("grid", "ell", 1), ("grid", "csr", 3), ("zipf", "csr", 2), ("zipf", "csr", 16),
           ("zipf", "coo", 0)]


class _View:
    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "data": (ptr, False), "version": 3}


def _view(owner, ptr, n):
    return torch.as_tensor(_View(owner, ptr, n), device="cuda")


def _round(hd, x, y, ybar, xbar, abar, src, k):
    """One round: inputs written by torch kernels, the calls, the results folded into one vector."""
    x.copy_(src * (1.0 + 0.25 * (k % 4)))
    y.mul_(0.0)
    hd.do_spmv(1)
    ybar.copy_(y + src)
    xbar.zero_()
    hd.spmv_adjoint(ybar.data_ptr(), xbar.data_ptr(), abar.data_ptr())
    out = y + xbar + abar.sum()
    ybar.fill_(float("nan"))    # overwritten while the next launches are in the stream
    abar.fill_(float("nan"))
    y.fill_(0.0)
    return out


@pytest.mark.parametrize("name,fmt,method", FORMATS)
def test_neighbours_in_the_stream(name, fmt, method):
    case = CASES[name]
    n = case[0]
    st = torch.cuda.Stream()
    src = torch.rand(n, device="cuda") - 0.5
    hd = Handle(Cocktail.single(fmt, coo_of(case), method), None, None, CSP_FLAG_ADJOINT)
    hd.set_stream(st.cuda_stream)
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        x, y = _view(hd, hd.vec_ptr, n), _view(hd, hd.res_ptr, n)
        ybar, xbar = torch.empty(n, device="cuda"), torch.empty(n, device="cuda")
        abar = torch.empty(hd.adjoint_slots, device="cuda")
        want = []
        for k in range(4):
            want.append(_round(hd, x, y, ybar, xbar, abar, src, k))
            torch.cuda.synchronize()
        got = [_round(hd, x, y, ybar, xbar, abar, src, k) for k in range(24)]
        torch.cuda.synchronize()
        for k, g in enumerate(got):
            assert torch.equal(g, want[k % 4]), f"round {k}"
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            outs = [_round(hd, x, y, ybar, xbar, abar, src, k) for k in range(8)]
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
        for k, g in enumerate(outs):
            assert torch.equal(g, want[k % 4]), f"captured round {k}"
    del graph
    hd.synchronize()


@pytest.mark.parametrize("flags", [CSP_FLAG_ADJOINT, CSP_FLAG_ADJOINT | 0x4])
def test_batch_neighbours_in_the_stream(flags):
    mats = [M.zipf_rows(3000, seed=i, max_len=900) for i in range(4)] + [M.laplacian_2d(40), M.block_3x3(700, seed=8)]
    st = torch.cuda.Stream()
    b = Batch([coo_of(m) for m in mats], flags=flags)
    b.set_stream(st.cuda_stream)
    nx, ny, na = int(b.x_off[-1]), int(b.y_off[-1]), int(b.abar_off[-1])
    p = b.device_ptrs()
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        x, y, ybar, xbar, abar = (_view(b, p[k], n) for k, n in (("x", nx), ("y", ny), ("ybar", ny), ("xbar", nx), ("abar", na)))
        src, srcy = torch.rand(nx, device="cuda") - 0.5, torch.rand(ny, device="cuda") - 0.5

        def once(k):
            x.copy_(src * (1 + k % 3))
            y.zero_()
            xbar.zero_()
            ybar.copy_(srcy)
            b.run(CSP_BATCH_FWD if k % 2 else CSP_BATCH_FWD | CSP_BATCH_ADJ)
            out = torch.cat([y, xbar, abar])
            x.fill_(0.0)
            y.fill_(5.0)
            return out

        want = []
        for k in range(6):
            want.append(once(k))
            torch.cuda.synchronize()
        got = [once(k) for k in range(36)]
        torch.cuda.synchronize()
        for k, g in enumerate(got):
            assert torch.equal(g, want[k % 6]), f"run {k}"
    b.synchronize()


@pytest.mark.parametrize("name,fmt,method", FORMATS)
def test_event_between_streams(name, fmt, method):
    """x is written late on another stream and handed over by an event; that stream overwrites
    it as soon as an event says the product is done."""
    case = CASES[name]
    n = case[0]
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    hd = Handle(Cocktail.single(fmt, coo_of(case), method))
    hd.set_stream(b.cuda_stream)
    x, y = _view(hd, hd.vec_ptr, n), _view(hd, hd.res_ptr, n)
    src = torch.rand(n, device="cuda") - 0.5
    torch.cuda.synchronize()
    outs = []
    for late in (False, True):
        got = []
        for k in range(6):
            with torch.cuda.stream(a):
                if late:
                    torch.cuda._sleep(200_000)
                x.copy_(src * (k + 1))
                written = torch.cuda.Event()
                written.record(a)
            with torch.cuda.stream(b):
                y.zero_()
                b.wait_event(written)
                hd.do_spmv(1)
                read = torch.cuda.Event()
                read.record(b)
                got.append(y.clone())
            with torch.cuda.stream(a):
                a.wait_event(read)
                x.fill_(float("nan"))
            if not late:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        outs.append(got)
    for k, (p, q) in enumerate(zip(*outs)):
        assert torch.isfinite(q).all() and torch.equal(p, q), f"round {k}"
