"""The warp-per-ray kernel's build and k-buffer sizes for launches of few rays
(below 56 rays an SM) against the oracle's float render, bit for bit,
on either side of the lines that choose them, and batches of one shape that
replay one graph although their views ask for other k-buffers."""
import numpy as np
import pytest

from conftest import small_scene, view
from oracle import oracle
from gtrace.tracer import Scene
from gtrace.uniforms import with_fields
from test_stream_gpu import _bits, _same

pytestmark = pytest.mark.gpu


# 148 SMs: 8,288 rays (56 an SM), 9,472 (64, the colour table's line) and 23,680 (160, where lists begin)
@pytest.mark.parametrize("w,h", [(1, 1), (37, 256), (74, 128), (111, 86), (185, 127), (185, 129)])
@pytest.mark.parametrize("k", [7, 8, 16, 17, 32])
def test_lines_between_builds_and_buffers(ctx, w, h, k):
    pg = small_scene(n=2500, seed=83)
    _same(ctx, pg.gaussiansBuffer, 0.01, view(w, h, k=k, T_min=0.002).uniforms, w, h)


def test_one_graph_for_several_buffers(ctx):
    pg = small_scene(n=2500, seed=84)
    s, o = Scene(ctx, pg.gaussiansBuffer, 0.01), oracle.Scene(pg.gaussiansBuffer, 0.01, "f32")
    for w, h in [(60, 50), (100, 90)]:
        for ks in [(4, 7), (8, 3), (5, 5), (16, 2), (9, 12), (32, 1), (17, 30)]:
            views = [(s, view(w, h, k=k, pos=(0.1 * k, 0.3, 4.0)).uniforms, w, h) for k in ks]
            outs, _ = ctx.render_batch(views)
            for (_, u, ww, hh), out in zip(views, outs):
                assert np.array_equal(_bits(out), o.render(u, ww, hh)[0].view(np.uint32)), ks
    s.close()


@pytest.mark.parametrize("w,h", [(5, 5), (25, 25), (26, 25), (25, 26)])
def test_line_of_the_colour_table(ctx, w, h):
    """625 rays of 2,500 particles, and a few more; as one view, and as a batch
    whose views count together."""
    pg = small_scene(n=2500, seed=85)
    u = view(w, h, k=6).uniforms
    _same(ctx, pg.gaussiansBuffer, 0.01, u, w, h)
    s, o = Scene(ctx, pg.gaussiansBuffer, 0.01), oracle.Scene(pg.gaussiansBuffer, 0.01, "f32")
    ref = o.render(u, w, h)[0].view(np.uint32)
    for _ in range(2):
        for out in ctx.render_batch([(s, u, w, h)] * 2)[0]:
            assert np.array_equal(_bits(out), ref)
    s.close()


@pytest.mark.parametrize("k,amin,w,h", [(6, 0.05, 25, 25), (6, 0.05, 26, 25), (5, 0.05, 25, 25), (6, 0.01, 13, 3),
                                        (6, 0.01, 20, 2), (16, 0.01, 25, 25), (8, 0.1, 25, 25), (8, 0.1, 130, 100),
                                        (8, 0.05, 112, 74), (8, 0.05, 111, 74)])
def test_lines_of_the_colour_table_and_the_deep_buffer(ctx, k, amin, w, h):
    """Either side of the other terms that choose the table (k, alpha_min, 64
    particles a ray), the 96-entry buffer (alpha_min) and the build (56 rays an
    SM), single and in a batch with another k."""
    pg = small_scene(n=2500, seed=86)
    u = with_fields(view(w, h, k=k).uniforms, alpha_min=amin)
    _same(ctx, pg.gaussiansBuffer, amin, u, w, h)
    s, o = Scene(ctx, pg.gaussiansBuffer, amin), oracle.Scene(pg.gaussiansBuffer, amin, "f32")
    u2 = with_fields(view(w, h, k=17).uniforms, alpha_min=amin)
    for out, uu in zip(ctx.render_batch([(s, u, w, h), (s, u2, w, h)])[0], (u, u2)):
        assert np.array_equal(_bits(out), o.render(uu, w, h)[0].view(np.uint32))
    s.close()


@pytest.mark.parametrize("k", [3, 4])
@pytest.mark.parametrize("w,h", [(163, 146), (163, 147)])
def test_lists_of_larger_scenes(ctx, k, w, h):
    """160 and 161 rays an SM of 14,100 proxies: with k 4 the lists begin one
    ray an SM later."""
    pg = small_scene(n=14_100, seed=89)
    _same(ctx, pg.gaussiansBuffer, 0.01, view(w, h, k=k, T_min=0.05).uniforms, w, h)
