"""Times of handles on the device, for tests that compare one path with another."""
import numpy as np
import torch


def spmv_us(hd, calls=8, reps=7):
    """Microseconds of one do_spmv among `calls` in a row, the best of `reps`."""
    st = torch.cuda.Stream()
    hd.set_stream(st.cuda_stream)
    hd.do_spmv(calls)
    st.synchronize()
    best = np.inf
    for _ in range(reps):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(st)
        hd.do_spmv(calls)
        e1.record(st)
        st.synchronize()
        best = min(best, 1e3 * e0.elapsed_time(e1) / calls)
    hd.synchronize()
    return best
