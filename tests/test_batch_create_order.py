"""csp_batch_create clears and fills its memory on the legacy stream, and the batch runs on a
non-blocking one: what is still in flight there when the call returns would land in the
middle of the first run (the item counters back at zero hand items out twice)."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "clspmv_b200", "csrc", "batch.cu")


def test_nothing_in_flight_when_create_returns():
    with open(SRC) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    body = text[text.index("int csp_batch_create("):text.index("int csp_batch_free(")]
    device_work = [m.start() for m in re.finditer(r"\bcudaMem(?:cpy|set)\w*\(|<<<|launch_\w+\(|\.commit\(", body)]
    waits = [m.start() for m in re.finditer(r"\bcuda(?:DeviceSynchronize|StreamSynchronize)\(", body)]
    assert device_work and waits and max(waits) > max(device_work)
    assert "cudaMemset(" not in body   # Arena::commit has cleared the counters with everything else
