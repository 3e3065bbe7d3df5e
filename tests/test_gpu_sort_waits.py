"""A sort's or entry scan's block that runs out of its wait for an earlier tile
counts that tile itself: with a wait limit of 0 (every look-back that meets an
unpublished tile does so) the binning and the image are word for word those of
the default limit. Sizes: a few look-back tiles up to more than the resident
blocks (296 of a sort pass, 592 of a scan), item and expansion indices in the
pairs, one view and several."""
import numpy as np
import pytest

from splattar_b200 import Rasterizer
from splattar_b200.synthetic import make_surfels, ring_cameras

pytestmark = pytest.mark.gpu


def _binning(r, cams, n, limit):
    r.set_wait_limits(limit)
    r.forward(cams, n)
    r.check()
    total = int(r.read("entry_count", 1)[0])
    tiles = sum(-(-c.width // 16) * -(-c.height // 16) for c in cams)
    pixels = sum(c.width * c.height for c in cams)
    return (r.read("depth_order", n * len(cams)), r.read("ranges", 2 * tiles), r.read("sorted_items", 2 * total),
            r.read("out_color", 4 * pixels), total)


@pytest.mark.parametrize("n,sizes", [(3000, [(200, 117)]), (9001, [(320, 240), (131, 90)]), (200000, [(1280, 720)] * 3),
                                     (900000, [(160, 120)] * 3)])
@pytest.mark.parametrize("deterministic", [False, True])
def test_expired_waits_change_nothing(n, sizes, deterministic):
    cams = ring_cameras(sizes)
    r = Rasterizer(n, 0, 0, 128 * n * len(cams), max_views=len(cams), max_pixels=sum(w * h for w, h in sizes),
                   deterministic=deterministic)
    r.upload_scene(make_surfels(n, 7, True, 0, 0.1).scene_input())
    want = _binning(r, cams, n, 2_000_000_000)
    assert want[-1] > 4096
    for _ in range(3):
        got = _binning(r, cams, n, 0)
        assert got[-1] == want[-1]
        for a, b in zip(got[:-1], want[:-1]):
            assert np.array_equal(a, b)
