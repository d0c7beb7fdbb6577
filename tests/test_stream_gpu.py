"""The per-view list tracer (gt_stream.cu), the default from 160 rays an SM,
against the oracle's float render, bit for bit: both ray counts per warp,
ragged image edges, cameras whose proxies straddle the camera plane, wide and
narrow fields of view, lists and heaps that do not fit (the warp-per-ray
kernel then finishes the rays), views the lists cannot serve, and the
checkpointing forward's gradients.  Images and counters must be equal (every
kernel runs the same float operations per ray); gradients have the tolerance
of test_backward_gpu.py."""
import numpy as np
import pytest

from conftest import small_scene, view
from oracle import oracle
from gtrace.tracer import Scene
from gtrace.uniforms import look_at, pack_uniforms, with_fields

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).reshape(-1, 4).view(np.uint32)


def _same(ctx, rec, amin, u, w, h):
    g = Scene(ctx, rec, amin)
    img, st = ctx.render(g, u, w, h, stats=True)
    ref, _ = oracle.Scene(rec, amin, "f32").render(u, w, h)
    assert np.array_equal(_bits(img), ref.view(np.uint32))
    assert st["rays"] == w * h
    # the warp-per-ray kernel's counters of the same view
    ctx.set_tune(g, u, w, h, kbuf=64, blocks_per_sm=8, block_threads=128)
    try:
        st2 = ctx.render(g, u, w, h, stats=True)[1]
    finally:
        ctx._lib.gt_autotune_reset(ctx._h)
        g.close()
    for name in ("rounds", "entries", "contributing"):
        assert st[name] == st2[name], name
    return st


def _records(n, pos, scale, opacity, seed):
    """Round Gaussians of one scale and opacity, random base colours."""
    rec = np.zeros((n, 80), np.float32)
    rec[:, 0:3] = pos
    rec[:, 4:7] = scale
    rec[:, 8] = 1.0
    rec[:, 12] = opacity
    rec[:, 16:19] = np.random.default_rng(seed).normal(size=(n, 3))
    return rec


# 148 SMs: lists from 23,680 rays, 32 rays a warp from 94,720; the sizes lie
# beside both and cut tiles, bins and blocks of tiles
@pytest.mark.parametrize("w,h", [(163, 146), (257, 129), (331, 287), (96000, 1), (3, 32000)])
@pytest.mark.parametrize("k", [1, 16])
def test_sizes_and_rounds(ctx, w, h, k):
    pg = small_scene(n=2500, seed=81)
    u = with_fields(view(w, h, k=k, T_min=0.003).uniforms, early_stop=3 if k == 1 else 0xFFFFFFFF)
    _same(ctx, pg.gaussiansBuffer, 0.01, u, w, h)


@pytest.mark.parametrize("kw", [dict(hfov=4.0), dict(hfov=150.0), dict(pos=(0.05, -0.02, 0.1), target=(1.0, 0.3, -2.0)),
                                dict(pos=(2.9, 0.1, 0.2), target=(3.5, 0.0, 0.0)), dict(pos=(0.0, 0.0, 400.0), hfov=1.0)])
@pytest.mark.parametrize("w,h", [(200, 130), (380, 270)])
def test_cameras(ctx, kw, w, h):
    """Inside the scene (proxies around and behind the camera plane), beside
    it, far away, and fields of view of 1 to 150 degrees."""
    pg = small_scene(n=3000, seed=82)
    _same(ctx, pg.gaussiansBuffer, 0.01, view(w, h, k=7, **kw).uniforms, w, h)


def test_anisotropic_scene_and_scaled_axes(ctx):
    """Needles and discs (ratio 1000), and a camera matrix whose axes have
    lengths other than 1 (rays are normalised)."""
    rng = np.random.default_rng(83)
    rec = _records(1500, rng.normal(size=(1500, 3)), 0.05, 0.8, 83)
    rec[:, 4:7] = 10.0 ** rng.uniform(-3.5, -0.5, size=(1500, 3))
    q = rng.normal(size=(1500, 4))
    rec[:, 8:12] = q / np.linalg.norm(q, axis=1, keepdims=True)
    m = look_at((0.5, 1.0, 4.0)).reshape(4, 4).copy()
    m[0, :3] *= 0.5
    m[1, :3] *= 2.0
    m[2, :3] *= 1.5
    w, h = 230, 160
    u = pack_uniforms(m.reshape(16), w, h, k=6, alpha_min=0.01, T_min=0.01)
    _same(ctx, rec, 0.01, u, w, h)


@pytest.mark.parametrize("w,h", [(180, 140), (330, 300)])
def test_more_waiting_hits_than_a_column_holds(ctx, w, h):
    """400 faint proxies of nearly one place: hundreds of hits of a ray lie
    within the bounds of all of them, more than its column takes."""
    rng = np.random.default_rng(84)
    rec = _records(400, 1e-3 * rng.normal(size=(400, 3)), 0.3 + 1e-4 * rng.random((400, 1)), 0.03, 84)
    st = _same(ctx, rec, 0.005, view(w, h, k=8, T_min=0.001, alpha_min=0.005).uniforms, w, h)
    assert st["handed"] > 1000


def test_lists_that_do_not_fit(ctx):
    """3,500 proxies that each cover the whole image need more list entries
    (1.75 million for 500 bins) than a launch has at first; the next one has them."""
    rng = np.random.default_rng(85)
    d = rng.normal(size=(3500, 3))
    rec = _records(3500, 3.0 * d / np.linalg.norm(d, axis=1, keepdims=True) + (0.0, 0.0, -3.0), 4.0, 0.02, 85)
    w, h = 320, 200
    u = view(w, h, pos=(0.0, 0.0, 30.0), k=16, T_min=0.01, hfov=3.0).uniforms
    from gtrace.tracer import Context
    with Context(0) as c2:
        g = Scene(c2, rec, 0.01)
        ref, _ = oracle.Scene(rec, 0.01, "f32").render(u, w, h)
        handed = []
        for _ in range(2):
            img, st = c2.render(g, u, w, h, stats=True)
            assert np.array_equal(_bits(img), ref.view(np.uint32))
            handed.append(st["handed"])
        assert handed[0] > 0
        g.close()


@pytest.mark.parametrize("case", ["sheared", "t_min", "t_max"])
def test_views_the_lists_do_not_serve(ctx, case):
    """A sheared camera and a negative t_min take the hierarchy kernels; a
    finite t_max does not."""
    pg = small_scene(n=2500, seed=86)
    w, h = 210, 150
    m = look_at((0.3, 0.4, 4.0)).reshape(4, 4).copy()
    kw = dict(k=6, alpha_min=0.01, T_min=0.01)
    if case == "sheared":
        m[0, :3] += 0.1 * m[2, :3]
    elif case == "t_min":
        kw["t_min"] = -0.5
    else:
        kw["t_max"] = 4.1
    _same(ctx, pg.gaussiansBuffer, 0.01, pack_uniforms(m.reshape(16), w, h, **kw), w, h)


def test_antialiased_frames_and_batch_graph(ctx):
    """Jittered frames blended by the list tracer, and a batch of two scenes
    replayed from its graph with other scenes and cameras."""
    pa, pb = small_scene(n=2000, seed=87), small_scene(n=3000, seed=88)
    ga, gb = Scene(ctx, pa.gaussiansBuffer, 0.01), Scene(ctx, pb.gaussiansBuffer, 0.02)
    oa, ob = oracle.Scene(pa.gaussiansBuffer, 0.01, "f32"), oracle.Scene(pb.gaussiansBuffer, 0.02, "f32")
    w, h = 173, 151
    acc, ref = np.zeros((h, w, 4), np.float32), np.zeros((w * h, 4), np.float32)
    for f in range(2):
        u = view(w, h, k=5, accumulated_frames=f).uniforms
        ctx.render(ga, u, w, h, out=acc, antialias=True)
        oa.render_accum(u, w, h, ref)
        assert np.array_equal(_bits(acc), ref.view(np.uint32)), f
    for (s0, o0), (s1, o1), x in [((ga, oa), (gb, ob), 0.0), ((gb, ob), (ga, oa), 1.5)]:
        views = [(s0, view(150, 90, pos=(x, 0.5, 4.0), k=4).uniforms, 150, 90),
                 (s1, view(130, 110, pos=(1.0, x, 3.5), k=9).uniforms, 130, 110)]
        outs, st = ctx.render_batch(views)
        for (_, u, ww, hh), o, out in zip(views, (o0, o1), outs):
            assert np.array_equal(_bits(out), o.render(u, ww, hh)[0].view(np.uint32))
        assert st["rays"] == 150 * 90 + 130 * 110


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("w,h", [(170, 145), (350, 280)])
def test_checkpoint_and_gradients(ctx, mode, w, h):
    from test_backward_gpu import _check, _ref_grad
    pg = small_scene(n=1200, seed=89)
    rec = pg.gaussiansBuffer
    u = view(w, h, k=5, T_min=0.002).uniforms
    s = Scene(ctx, rec, 0.01)
    img = ctx.render(s, u, w, h, checkpoint=True)
    ref, _ = oracle.Scene(rec, 0.01, "f32").render(u, w, h)
    assert np.array_equal(_bits(img), ref.view(np.uint32))
    g = np.random.default_rng(12).normal(size=(h, w, 4)).astype(np.float32)
    got, info = ctx.backward(s, u, w, h, g, mode=mode)
    assert info["used_mode"] == mode
    _check(got, _ref_grad(rec, 0.01, u, w, h, g))
