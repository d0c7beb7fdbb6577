"""The hierarchy of a scene with a few proxies far out: the others are divided as
finely as without them."""
import numpy as np
import pytest

from conftest import small_scene, view
from gtrace.tracer import Scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("outliers", [1, 8, 300])
def test_outliers_do_not_coarsen_the_hierarchy(ctx, fast, outliers):
    """Node visits of a view that shows the rest, by the warp-per-ray kernel:
    at most a quarter more with the outliers (1.5 % of the proxies at most)."""
    n, w, h = 20000, 160, 120
    rec = small_scene(n=n, seed=97).gaussiansBuffer.reshape(-1, 80)
    far = rec.copy()
    pick = np.random.default_rng(97).choice(n, outliers, replace=False)
    d = np.random.default_rng(98).normal(size=(outliers, 3))
    far[pick, 0:3] = 2000.0 * d / np.linalg.norm(d, axis=1, keepdims=True)
    u = view(w, h, k=6).uniforms
    visits = []
    for r in (np.delete(rec, pick, axis=0), far):
        s = Scene(ctx, np.ascontiguousarray(r), 0.01, fast_build=fast)
        ctx.set_tune(s, u, w, h, block_threads=128, kbuf=64, blocks_per_sm=8)
        try:
            visits.append(ctx.render(s, u, w, h, stats=True)[1]["node_visits"])
        finally:
            ctx._lib.gt_autotune_reset(ctx._h)
            s.close()
    assert visits[1] <= 1.25 * visits[0]
