"""The list tracer with the camera inside the scene: proxies that cross the
camera plane are tested by the rays that may meet them only, and the images
are the oracle's, bit for bit."""
import numpy as np
import pytest

from conftest import small_scene, view
from oracle import oracle
from gtrace.tracer import Scene
from gtrace.uniforms import look_at, pack_uniforms

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).reshape(-1, 4).view(np.uint32)


@pytest.mark.parametrize("w,h", [(200, 150), (400, 280)])
def test_face_tests_stay_near_the_hierarchys(ctx, w, h):
    """16,384 Gaussians seen from their centre, about 1,500 of them across the
    camera plane: at most as many face tests as the warp-per-ray kernel makes
    sphere tests (with every ray testing all of those, eleven times as many)."""
    pg = small_scene(n=16384, seed=7)
    s = Scene(ctx, pg.gaussiansBuffer, 0.01)
    u = view(w, h, pos=(0.0, 0.0, 0.0), target=(1.0, 0.2, -1.0), k=6).uniforms
    lists = ctx.render(s, u, w, h, stats=True)
    ctx.set_tune(s, u, w, h, block_threads=128, kbuf=64, blocks_per_sm=8)
    try:
        ref = ctx.render(s, u, w, h, stats=True)
    finally:
        ctx._lib.gt_autotune_reset(ctx._h)
        s.close()
    assert np.array_equal(_bits(lists[0]), _bits(ref[0]))
    assert lists[1]["node_visits"] < ref[1]["node_visits"]  # (lists did serve)
    assert lists[1]["proxy_tests"] <= ref[1]["proxy_tests"]


@pytest.mark.parametrize("hfov", [20.0, 75.0, 150.0, 172.0])
@pytest.mark.parametrize("seed", [0, 1, 2])
def test_proxies_across_and_beside_the_camera_plane(ctx, seed, hfov):
    """Needles, discs and balls of 0.01 to 2 about the camera, some of which it
    is inside of, some tangent to its plane, under random turns of the camera."""
    rng = np.random.default_rng(700 + seed)
    n, w, h = 1500, 190, 131
    rec = np.zeros((n, 80), np.float32)
    eye = np.array([0.3, -0.2, 0.1])
    d = rng.normal(size=(n, 3))
    rec[:, 0:3] = eye + d / np.linalg.norm(d, axis=1, keepdims=True) * 10.0 ** rng.uniform(-1.3, 0.8, size=(n, 1))
    rec[:, 4:7] = 10.0 ** rng.uniform(-2.0, -0.3, size=(n, 3))
    q = rng.normal(size=(n, 4))
    rec[:, 8:12] = q / np.linalg.norm(q, axis=1, keepdims=True)
    rec[:, 12] = rng.uniform(0.02, 0.5, size=n)
    rec[:, 16:19] = rng.normal(size=(n, 3))
    m = look_at(eye, eye + rng.normal(size=3))
    # balls whose tops touch the camera plane: radius 1.2584 sqrt(2 ln(o / alpha_min)) scale
    back = m.reshape(4, 4)[2, :3].astype(np.float64)
    reach = 1.2584 * np.sqrt(2.0 * np.log(rec[:200, 12] / 0.01)) * rec[:200, 4]
    rec[:200, 5] = rec[:200, 6] = rec[:200, 4]
    side = rng.normal(size=(200, 3))
    side -= np.outer(side @ back, back)
    rec[:200, 0:3] = eye + side * 0.7 - np.outer(reach * (1.0 + rng.choice([-1e-3, 0.0, 1e-3], size=200)), back)
    u = pack_uniforms(m, w, h, hfov=hfov, k=8, alpha_min=0.01, T_min=0.001)
    s = Scene(ctx, rec, 0.01)
    img = ctx.render(s, u, w, h)
    s.close()
    assert np.array_equal(_bits(img), oracle.Scene(rec, 0.01, "f32").render(u, w, h)[0].view(np.uint32))


@pytest.mark.parametrize("w,h", [(200, 150), (330, 300)])
def test_dense_scenes_stay_with_the_lists(ctx, w, h):
    """Large proxies all around the camera, many of them about it: between 128 and
    256 hits of every ray wait for the last of these, and its column holds them."""
    rng = np.random.default_rng(710)
    n = 20000
    rec = np.zeros((n, 80), np.float32)
    rec[:, 0:3] = np.clip(rng.normal(size=(n, 3)), -3, 3)
    rec[:, 4:7] = np.exp(rng.uniform(-4.5, -2.5, size=(n, 3))) * 4.0
    q = rng.normal(size=(n, 4))
    rec[:, 8:12] = q / np.linalg.norm(q, axis=1, keepdims=True)
    rec[:, 12] = rng.uniform(0.05, 0.99, size=n)
    rec[:, 16:19] = rng.normal(size=(n, 3))
    s = Scene(ctx, rec, 0.01)
    u = view(w, h, pos=(0.0, 0.0, 0.0), target=(1.0, 0.2, -1.0), k=6).uniforms
    img, st = ctx.render(s, u, w, h, stats=True)
    ctx.set_tune(s, u, w, h, block_threads=128, kbuf=64, blocks_per_sm=8)
    try:
        ref = ctx.render(s, u, w, h)
    finally:
        ctx._lib.gt_autotune_reset(ctx._h)
        s.close()
    assert np.array_equal(_bits(img), _bits(ref))
    assert st["handed"] < 0.5 * w * h
