"""The public scan on several streams and threads at once, and recorded into a
graph: each call has its own block sums. Integers, compared with numpy."""
import threading

import numpy as np
import pytest

from splattar_b200 import exclusive_scan_u32

pytestmark = pytest.mark.gpu


def _arrays(n, seed):
    import torch
    a = np.random.default_rng(seed).integers(0, 1 << 10, n)  # sums below 2^32
    a = a.astype(np.uint32)
    t = torch.from_numpy(a.view(np.int32).copy()).cuda()
    exp = (np.cumsum(a, dtype=np.uint64) - a).astype(np.uint32)
    return a, t, torch.zeros_like(t), torch.zeros(1, dtype=torch.int32, device="cuda"), exp


def test_scans_overlap_on_streams_and_threads():
    import torch
    sizes = (3_000_001, 1_000_000, 70_001, 2_500_000)
    data = [_arrays(n, n) for n in sizes]
    streams = [torch.cuda.Stream() for _ in sizes]
    torch.cuda.synchronize()

    def call(k):
        _, t, out, total, _ = data[k]
        for _ in range(50):
            exclusive_scan_u32(t.data_ptr(), out.data_ptr(), t.numel(), total.data_ptr(), streams[k].cuda_stream)

    threads = [threading.Thread(target=call, args=(k,)) for k in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for a, _, out, total, exp in data:
        assert np.array_equal(out.cpu().numpy().view(np.uint32), exp)
        assert int(total.cpu().numpy().view(np.uint32)[0]) == int(a.sum(dtype=np.uint64))


def test_captured_scan_replays():
    import torch
    a, t, out, total, exp = _arrays(200_003, 5)
    exclusive_scan_u32(t.data_ptr(), out.data_ptr(), t.numel(), total.data_ptr())  # first use on the device
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        exclusive_scan_u32(t.data_ptr(), out.data_ptr(), t.numel(), total.data_ptr(),
                           torch.cuda.current_stream().cuda_stream)
    for _ in range(3):
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy().view(np.uint32), exp)
