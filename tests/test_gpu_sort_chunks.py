"""Tile sorts of many entries (by chunks from 9 million on when two passes are
needed): around that number, with one pass, and with every wait expiring at
once. Integers: compared with a stable numpy sort by (tile, depth, item)."""
import numpy as np
import pytest

from splattar_b200 import Rasterizer, TileBinner
from splattar_b200.synthetic import make_surfels, ring_cameras
from test_gpu_project_binning import dev_to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("total,tiles_x,tiles_y", [(8_999_999, 120, 68), (9_000_000, 120, 68), (9_000_001, 160, 90),
                                                   (9_699_328, 32, 9), (10_000_003, 16, 16), (20_000_000, 257, 181)])
def test_binner_of_many_entries(total, tiles_x, tiles_y):
    """Items of `k` tiles in a row (the last one shorter), random places and depths with ties."""
    import torch
    k = 8
    n = -(-total // k)
    rng = np.random.default_rng(total)
    x0, y0 = rng.integers(0, tiles_x - k + 1, n), rng.integers(0, tiles_y, n)
    length = np.full(n, k)
    length[-1] = total - k * (n - 1)
    rects = np.stack([x0, y0, x0 + length - 1, y0], axis=1).astype(np.int32)
    depths = rng.integers(0, n // 3, n).astype(np.int32)
    b = TileBinner(n, total, tiles_x * tiles_y)
    tr, td = torch.from_numpy(rects).cuda(), torch.from_numpy(depths).cuda()
    b.encode(tr.data_ptr(), td.data_ptr(), n, tiles_x)
    entry = lambda name, m: dev_to_host(b.buffer(name)[0], m, np.uint32)  # noqa: E731
    # entries in item order; a tile's entries by depth, then item
    item = np.repeat(np.arange(n), length)
    tile = (y0 * tiles_x + x0)[item] + np.arange(total) - k * item
    order = np.argsort(tile.astype(np.int64) * n + depths[item], kind="stable")
    assert np.array_equal(entry("sorted_entries", total), order)
    counts = np.bincount(tile, minlength=tiles_x * tiles_y)
    end = np.cumsum(counts)
    want = np.stack([end - counts, end], axis=1)
    want[counts == 0] = 0
    assert np.array_equal(entry("ranges", 2 * tiles_x * tiles_y).reshape(-1, 2), want)


def test_expired_waits_change_nothing_by_chunks():
    n, sizes = 400000, [(1600, 900)] * 3
    cams = ring_cameras(sizes)
    r = Rasterizer(n, 0, 0, 128 * n, max_views=3, max_pixels=sum(w * h for w, h in sizes))
    r.upload_scene(make_surfels(n, 7, True, 0, 0.1).scene_input())
    got = []
    for limit in (2_000_000_000, 0, 0):
        r.set_wait_limits(limit)
        r.forward(cams, n)
        r.check()
        total = int(r.read("entry_count", 1)[0])
        assert total > 9_000_000
        got.append((r.read("ranges", 2 * 3 * 100 * 57), r.read("sorted_items", 2 * total)))
    for a in got[1:]:
        assert np.array_equal(a[0], got[0][0]) and np.array_equal(a[1], got[0][1])
