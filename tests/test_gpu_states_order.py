"""State counts in device memory, written by work on a blocking stream that is
still running when the graph is created: a copy of the array to the host waited
for it, and so does the scan on the device."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_counts_written_on_a_blocking_stream(bp):
    import torch
    from belief_propagation_b200.engine import BPGraph
    torch.cuda.init()
    rt = C.CDLL("libcudart.so.12")
    handle = C.c_void_p()
    assert rt.cudaStreamCreate(C.byref(handle)) == 0   # blocking, unlike torch's own streams
    try:
        rng = np.random.default_rng(2)
        V, E, S = 3000, 9000, 4
        counts = rng.choice(np.array([2, 3, 4], np.int32), V)
        src = np.sort(rng.integers(0, V, E))
        dst = (src + rng.integers(1, V, E)) % V
        j = rng.random((E, S, S), dtype=np.float32)
        j *= np.arange(S)[None, :, None] < counts[src][:, None, None]
        j *= np.arange(S)[None, None, :] < counts[dst][:, None, None]
        want = torch.from_numpy(counts).cuda()
        s32, d32 = (torch.from_numpy(x.astype(np.int32)).cuda() for x in (src, dst))
        joint = torch.from_numpy(j).cuda()
        late = torch.full((V,), 99, dtype=torch.int32, device="cuda")   # no valid count
        torch.cuda.synchronize()
        stream = torch.cuda.ExternalStream(handle.value)
        for _ in range(2):   # first calls load code and grow pools, and wait for the device
            BPGraph(V, s32, d32, joint, num_states=want).close()
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(100_000_000)   # some 50 ms
            late.copy_(want)
        with BPGraph(V, s32, d32, joint, num_states=late) as g:
            assert g.uniform == 0 and g.ms == S
        stream.synchronize()
    finally:
        rt.cudaStreamDestroy(handle)
