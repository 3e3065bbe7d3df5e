"""The bench's count of kernel launches per step against the kernels that a
step's trace shows, in both forms."""
import json

import numpy as np
import pytest

from splattar_b200 import AdamSettings, Rasterizer, StepSettings
from splattar_b200.synthetic import make_surfels, ring_cameras

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["chosen", "plain"])
@pytest.mark.parametrize("sizes", [[(320, 240), (256, 256)], [(200, 100), (96, 64)]])
def test_launches_of_a_step(form, sizes, tmp_path):
    import torch
    from torch.profiler import ProfilerActivity, profile

    import bench
    n = 9000
    cams = ring_cameras(sizes)
    pixels = sum(w * h for w, h in sizes)
    r = Rasterizer(n, 0, 0, 64 * n * len(sizes), max_views=len(sizes), max_pixels=pixels, color_only=True)
    r.upload_scene(make_surfels(n, 7, True, 0, 0.1).scene_input())
    r.optimizer_init(n)
    r.write("target", np.full(4 * pixels, 0.3, np.float32))
    step = StepSettings(0.8, 0.2, AdamSettings(), form)
    for _ in range(3):
        r.train_step(cams, n, step)
    r.check()
    steps = 2
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        for _ in range(steps):
            r.train_step(cams, n, step)
        torch.cuda.synchronize()
    r.check()
    p.export_chrome_trace(str(tmp_path / "trace.json"))
    events = json.load(open(tmp_path / "trace.json"))["traceEvents"]
    kernels = [e["name"] for e in events if e.get("cat") == "kernel" and "gs::" in e["name"]]  # (not memsets in a graph)
    tiles = [-(-w // 16) * -(-h // 16) for w, h in sizes]
    # the chosen form bins all views together, the plain form each by itself
    want = bench.launches_per_step(sum(tiles), len(sizes), form) if form == "chosen" else (
        sum(bench.launches_per_step(t, 1, form) - 6 for t in tiles) + 6)
    assert len(kernels) == steps * want, sorted(kernels)
