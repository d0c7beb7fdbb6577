"""Views of a far scene: few rays can meet it, and the launch is chosen by
these, not by the image size.  Images are the oracle's, bit for bit."""
import numpy as np
import pytest

from conftest import small_scene, view
from oracle import oracle
from gtrace.tracer import Scene

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).reshape(-1, 4).view(np.uint32)


# 148 SMs: the scene covers all of the image, about 2 % and about 0.2 % of it
@pytest.mark.parametrize("distance,lists", [(5.0, True), (60.0, False), (200.0, False)])
@pytest.mark.parametrize("w,h,target", [(220, 170, (0.0, 0.0, 0.0)), (400, 300, (9.0, -7.0, 0.0))])
def test_far_scenes(ctx, distance, lists, w, h, target):
    pg = small_scene(n=16384, seed=7)
    s = Scene(ctx, pg.gaussiansBuffer, 0.01)
    u = view(w, h, pos=(0.0, 0.0, distance), target=(target if distance > 10.0 else (0.0, 0.0, 0.0)), k=6).uniforms
    img, st = ctx.render(s, u, w, h, stats=True)
    ctx.set_tune(s, u, w, h, block_threads=128, kbuf=64, blocks_per_sm=8)
    try:
        warp = ctx.render(s, u, w, h, stats=True)[1]
    finally:
        ctx._lib.gt_autotune_reset(ctx._h)
        s.close()
    assert np.array_equal(_bits(img), oracle.Scene(pg.gaussiansBuffer, 0.01, "f32").render(u, w, h)[0].view(np.uint32))
    same = (st["node_visits"], st["proxy_tests"]) == (warp["node_visits"], warp["proxy_tests"])
    assert same != lists  # (the warp-per-ray kernel's own counts)


# (16 quarter tiles of 8 rays, 16 tiles of 32: those of the four bins in the middle)
@pytest.mark.parametrize("w,h,rays", [(230, 170, 128), (400, 300, 512)])
def test_far_scene_with_outliers(ctx, w, h, rays):
    """Eight proxies far out stretch the scene's box over the image, so lists
    serve; the few tiles that show the rest, or lie beside it, hand their rays
    over instead of going through lists of 30,000 proxies while all others are
    idle."""
    rec = small_scene(n=30000, seed=8).gaussiansBuffer.copy().reshape(-1, 80)
    for i in range(8):
        rec[i, 0:3] = [1e3 * (1 if i >> a & 1 else -1) for a in range(3)]
        rec[i, 12] = 0.9
    s = Scene(ctx, rec, 0.01)
    u = view(w, h, pos=(0.0, 0.0, 150.0), k=6).uniforms
    img, st = ctx.render(s, u, w, h, stats=True)
    s.close()
    assert np.array_equal(_bits(img), oracle.Scene(rec, 0.01, "f32").render(u, w, h)[0].view(np.uint32))
    assert 0.75 * rays <= st["handed"] <= 2 * rays
