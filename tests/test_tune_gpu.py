"""The launch tuners (gt_autotune, gt_autotune_batch): the default launch is one
of their candidates."""
import pytest

from conftest import small_scene, view
from gtrace.tracer import Context, Scene

pytestmark = pytest.mark.gpu


# 148 SMs: below 56 rays an SM the default has a build of its own, lists begin
# at 160
@pytest.mark.parametrize("w,h,k,alpha_min", [(64, 64, 6, 0.2), (90, 60, 16, 0.2), (200, 150, 6, 0.01)])
def test_a_tuned_view_is_no_slower_than_the_default_launch(w, h, k, alpha_min):
    pg = small_scene(n=16384, seed=7)
    with Context(0) as c:
        s = Scene(c, pg.gaussiansBuffer, alpha_min)
        u = view(w, h, k=k, alpha_min=alpha_min, T_min=0.03).uniforms
        r = c.autotune(s, u, w, h)
        assert r["best_ms"] <= r["default_ms"]
        assert r["block_threads"] == 32 or r["kbuf"] >= k
        s.close()


def test_a_batch_result_names_the_shape_that_won(ctx):
    """A small far view, which lists serve: a warp per ray takes half their time
    and a tenth of the tile packets', and the result says so."""
    pg = small_scene(n=16384, seed=7)
    s = Scene(ctx, pg.gaussiansBuffer, 0.01)
    u = view(160, 150, pos=(0.0, 0.0, 60.0), k=32).uniforms
    try:
        r = ctx.autotune_batch([(s, u, 160, 150)])
        assert r["block_threads"] == 128
    finally:
        ctx._lib.gt_autotune_reset(ctx._h)
        s.close()


def test_a_batch_tries_the_default_launch_beside_a_cached_shape(ctx):
    """With tile packets cached for the view, the lists (twice as fast as any
    other launch here) are still tried, and win."""
    pg = small_scene(n=16384, seed=7)
    s = Scene(ctx, pg.gaussiansBuffer, 0.01)
    w, h = 640, 400
    u = view(w, h, k=6).uniforms
    try:
        ctx.set_tune(s, u, w, h, block_threads=32, kbuf=32)
        assert ctx.autotune_batch([(s, u, w, h)])["default"]
    finally:
        ctx._lib.gt_autotune_reset(ctx._h)
        s.close()
