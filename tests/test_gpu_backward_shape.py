"""The backward raster's shape as the number of tiles chooses it (below 4, or 6
in the persistent form, and from 32 tiles per SM on, and between) against a
fixed shape: the same gradients up to the order of float sums (bound: f32
tolerance of a step, 2e-4 in the 2-norm)."""
import numpy as np
import pytest

from gpu_util import raster_camera, scene_input
from scenes import make_scene
from splattar_b200 import Rasterizer

pytestmark = pytest.mark.gpu
WIDTHS = {"grad_pos": 4, "grad_scales": 2, "grad_quat": 4, "grad_opacity": 1, "grad_sh": 48}


@pytest.mark.parametrize("W,H", [(64, 48), (16 * 37, 16 * 15), (16 * 37, 16 * 16), (16 * 37, 16 * 17),
                                 (16 * 37, 16 * 23), (16 * 37, 16 * 24), (16 * 37, 16 * 31), (16 * 37, 16 * 32),
                                 (16 * 37, 16 * 33), (1184, 16 * 63), (1184, 16 * 64), (1183, 1039)])
@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("persistent", [False, True])
def test_chosen_by_tiles_equals_fixed(W, H, deterministic, persistent):
    scene, cam = make_scene(404, 2000, 1, 128)
    cam.focal *= W / cam.width
    cam.width, cam.height = W, H
    rng = np.random.default_rng(W + H)
    w = rng.normal(size=(W * H, 4)).astype(np.float32)
    w[:, 3] = 0
    got = []
    for fixed in (False, True):
        r = Rasterizer(scene.n, W, H, 4096 * scene.n, color_only=True, deterministic=deterministic,
                       persistent=persistent)
        if fixed:
            r.set_launch_shapes(128, 1, 128, 2)
        r.upload_scene(scene_input(scene))
        r.forward(raster_camera(cam, 1), scene.n)
        r.write("dl_dcolor", w.ravel())
        r.backward(scene.n)
        r.check()
        got.append({k: r.read(k, n * scene.n) for k, n in WIDTHS.items()} | {"grad_cam": r.read("grad_cam", 16)})
    for k, a in got[0].items():
        b = got[1][k].astype(np.float64)
        assert np.linalg.norm(a - b) <= 2e-4 * np.linalg.norm(b), k
