"""The losses' block and tile edges: L1+SSIM on images of many 32-pixel tiles
(whole, and a pixel more or less each way; narrow ones, which go by 16-pixel
tiles when too little of the large ones is image) and the normal loss summed over
several blocks of several views, against the oracle."""
import numpy as np
import pytest

import oracle
from gpu_util import forward, raster_camera, scene_input
from scenes import make_scene
from splattar_b200 import Rasterizer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(1024, 768), (1023, 801), (33, 12001), (12001, 33), (125, 8001), (8001, 125)])
@pytest.mark.parametrize("level", [(0.0, 1.0), (0.0, 0.05), (0.9, 1.6)])
def test_l1_ssim_large_tiles(W, H, level):
    """Bounds of test_l1_ssim_matches_oracle."""
    scene, cam = make_scene(5, 10, 0, 32)
    cam.width, cam.height = W, H
    rast, _ = forward(scene, cam)
    P = W * H
    rng = np.random.default_rng(W * 7 + H)
    img = rng.uniform(level[0], level[1], (P, 4)).astype(np.float32)
    ref = np.clip(img + rng.normal(0, 0.15 * (level[1] - level[0]), (P, 4)), level[0], level[1]).astype(np.float32)
    rast.write("out_color", img.ravel())
    rast.write("target", ref.ravel())
    rast.loss_l1_ssim(0.8, 0.2)
    rast.check()
    dl = rast.read("dl_dcolor", 4 * P).reshape(P, 4)
    sums = rast.read("loss", 2)
    _, dl_o, l1_o, ss_o = oracle.l1_ssim(img, ref, W, H, 0.8, 0.2)
    assert abs(sums[0] - l1_o) <= 1e-4 * abs(l1_o) + 1e-3
    assert abs(sums[1] - ss_o) <= 1e-4 * abs(ss_o) + 1e-3
    assert np.abs(dl[:, :3] - dl_o[:, :3]).max() <= 2e-4 * np.abs(dl_o[:, :3]).max()
    assert np.all(dl[:, 3] == 0)


def _pair(kind, W, H):
    """Image and target of one kind (rgba, float32)."""
    rng = np.random.default_rng(3)
    yy, xx = np.mgrid[0:H, 0:W]
    if kind == "object on black":
        a = np.zeros((H, W, 3))
        on = (xx // 97 + yy // 83) % 5 == 0
        a[on] = rng.uniform(0.3, 0.9, (on.sum(), 3))
        b = a + 0.004 * ~on[..., None]
    elif kind == "bright points on dark":
        a = rng.uniform(0, 0.01, (H, W, 3))
        a[rng.random((H, W)) < 0.01] = 1.0
        b = a + 0.002 * rng.normal(size=a.shape)
    elif kind == "smooth":
        s = (0.5 + 0.25 * np.sin(xx * 0.05) + 0.25 * np.cos(yy * 0.037))[..., None] * np.ones(3)
        a, b = s + 0.03 * rng.normal(size=s.shape), 0.9 * s + 0.05
    else:
        a = rng.uniform(*kind, (H, W, 3))
        b = np.clip(a + rng.normal(0, 0.15 * (kind[1] - kind[0]), a.shape), *kind)
    return [np.concatenate([np.clip(t, 0, None).reshape(-1, 3), np.ones((W * H, 1))], 1).astype(np.float32)
            for t in (a, b)]


@pytest.mark.parametrize("kind", [(0.0, 1.0), (0.0, 0.25), (0.0, 0.05), (0.0, 0.001), (0.4, 0.6), (0.9, 1.6),
                                  "object on black", "bright points on dark", "smooth"])
def test_large_tiles_are_as_exact_as_small_ones(kind):
    """Against 64 bits, in the 2-norm: an image of 800 32-pixel tiles and one of 208, which 16-pixel tiles
    take, of the same kind. 1.3: the two images' own difference (up to 1.05 with one kernel) and the
    other rounding of four maps instead of five."""
    err, l1 = [], []
    for W, H in ((1024, 800), (512, 400)):
        x, y = _pair(kind, W, H)
        scene, cam = make_scene(5, 10, 0, 32)
        cam.width, cam.height = W, H
        rast, _ = forward(scene, cam)
        rast.write("out_color", x.ravel())
        rast.write("target", y.ravel())
        rast.loss_l1_ssim(0.8, 0.2)
        rast.check()
        dl = rast.read("dl_dcolor", 4 * W * H).reshape(-1, 4)[:, :3]
        _, want, l1_o, _ = oracle.l1_ssim(x, y, W, H, 0.8, 0.2)
        err.append(np.linalg.norm(dl - want[:, :3]) / np.linalg.norm(want[:, :3]))
        l1.append(abs(rast.read("loss", 2)[0] - l1_o) / l1_o)
    assert err[0] <= 1.3 * err[1]
    assert max(l1) <= 2e-7  # differences of float32 values, summed: half an ulp per term at most


def _surface(W, H, seed):
    rng = np.random.default_rng(seed)
    ys, xs = np.mgrid[0:H, 0:W]
    alpha = np.clip(0.6 + 0.3 * np.sin(xs * 0.3) * np.cos(ys * 0.2) + 0.05 * rng.normal(size=(H, W)), 0, 1)
    depth = 2.0 + 0.2 * np.sin(xs * 0.25 + ys * 0.15) + 0.02 * rng.normal(size=(H, W))
    normal = rng.normal(size=(H, W, 3)) * 0.3 + np.array([0.0, 0.0, 1.0])
    return alpha.ravel(), (depth * alpha).ravel(), normal.reshape(-1, 3)


def test_normal_loss_sums_each_view_by_itself():
    """Bounds of test_cuda_normal_loss_matches_restatement."""
    sizes = ((67, 45), (21, 190), (5, 3))
    scene, cam = make_scene(5, 10, 0, 32)
    cams = []
    for w, h in sizes:
        cam.width, cam.height = w, h
        cams.append(raster_camera(cam, 0))
    P = sum(w * h for w, h in sizes)
    r = Rasterizer(scene.n, 0, 0, 64 * scene.n, max_views=3, max_pixels=P)
    r.upload_scene(scene_input(scene))
    r.forward(cams, scene.n)
    r.check()
    surf = [_surface(w, h, 7 + w) for w, h in sizes]
    col, aux, nr4, z = (np.zeros((P, 4), np.float32) for _ in range(4))
    col[:, 3] = np.concatenate([s[0] for s in surf])
    aux[:, 1] = np.concatenate([s[1] for s in surf])
    nr4[:, :3] = np.concatenate([s[2] for s in surf])
    for name, a in (("out_color", col), ("out_aux", aux), ("out_normal", nr4), ("dl_dcolor", z)):
        r.write(name, a.ravel())
    r.loss_normal(2.5, 0.2)
    r.check()
    got, dn = r.read("normal_loss", 3), r.read("dl_dnormal", 4 * P).reshape(P, 4)
    f32 = lambda a: np.asarray(a, np.float32).astype(np.float64)  # noqa: E731
    at = 0
    for v, ((w, h), (alpha, dacc, nrm)) in enumerate(zip(sizes, surf)):
        total, dno, _ = oracle.normal_loss(f32(alpha), f32(dacc), f32(nrm), w, h, float(np.float32(cam.focal)), 2.5)
        assert abs(got[v] - total) <= 1e-4 * abs(total)
        assert np.abs(dn[at:at + w * h, :3] - dno).max() <= 1e-4 * np.abs(dno).max() + 1e-9
        at += w * h
