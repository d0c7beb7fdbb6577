"""Room for the per-view proxy lists (gt_stream.cu, gt_api.cu): lists whose
lengths pass 2^32 together, and buffers that grow to what launches needed.  The hierarchy kernels' image of the same view is
the reference (bit-equal to the oracle, test_parity_gpu.py, test_packet_gpu.py)."""
import numpy as np
import pytest

from conftest import small_scene, view
from gtrace.tracer import Context, Scene
from gtrace.uniforms import look_at, pack_uniforms

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).reshape(-1, 4).view(np.uint32)


def test_more_list_entries_than_32_bits_count():
    """135,000 proxies that each cover all 32,768 bins of a 2^20 x 1 image:
    4.4e9 list entries.  The proxies lie one behind another (0.007 apart, 50 to
    1,050 from the camera, a field of view of 1 degree), so a ray ends at the
    first few."""
    n, w, h = 135_000, 1 << 20, 1
    rng = np.random.default_rng(91)
    rec = np.zeros((n, 80), np.float32)
    rec[:, 0:2] = 0.5 * rng.normal(size=(n, 2))
    rec[:, 2] = -np.linspace(50.0, 1050.0, n)
    rec[:, 4:7] = 4.0
    rec[:, 8] = 1.0
    rec[:, 12] = 0.6
    rec[:, 16:19] = rng.normal(size=(n, 3))
    u = pack_uniforms(look_at((0.0, 0.0, 0.0), (0.0, 0.0, -1.0)), w, h, hfov=1.0, k=4, alpha_min=0.01, T_min=0.02)
    u.view(np.float32)[17] = u.view(np.float32)[16]  # (anisotropic pixels)
    with Context(0) as c:
        s = Scene(c, rec, 0.01)
        got = [c.render(s, u, w, h) for _ in range(2)]
        c.set_tune(s, u, w, h, kbuf=64, blocks_per_sm=8, block_threads=128)
        ref = c.render(s, u, w, h)
        s.close()
    assert (ref[..., :3].max(axis=-1) > 0).mean() > 0.5
    for img in got:
        assert np.array_equal(_bits(img), _bits(ref))


W, H = 320, 200


def _wide_proxies(n):
    """Proxies that each cover the whole image, one behind another, and the view
    that shows them: a ray ends at the third or fourth."""
    rng = np.random.default_rng(92)
    rec = np.zeros((n, 80), np.float32)
    rec[:, 0:2] = 0.3 * rng.normal(size=(n, 2))
    rec[:, 2] = -np.linspace(50.0, 500.0, n)
    rec[:, 4:7] = 4.0
    rec[:, 8] = 1.0
    rec[:, 12] = 0.9
    rec[:, 16:19] = rng.normal(size=(n, 3))
    return rec, view(W, H, pos=(0.0, 0.0, 0.0), target=(0.0, 0.0, -1.0), k=4, T_min=0.01, hfov=1.5).uniforms


# 3,500 proxies in 500 bins: 1.75 million entries, room for 1.4 million at
# first: the rays of more than 80 bins (128 each) go to the warp-per-ray kernel,
# and once all fit, those at the launch's end
@pytest.mark.parametrize("how", ["another view between", "queued"])
def test_a_need_is_kept_and_told_without_waiting(how):
    rec, u = _wide_proxies(3500)
    small = view(64, 48, pos=(0.0, 0.0, 0.0), target=(0.0, 0.0, -1.0), k=4, hfov=1.5).uniforms
    with Context(0) as c:
        s = Scene(c, rec, 0.01)
        out = c.device_alloc(W * H * 16)
        if how == "queued":
            for _ in range(2):
                c.render_device(s, u, W, H, out, asynchronous=True)
            c.synchronize()
        else:
            assert c.render_device(s, u, W, H, out)["handed"] > 10_000
            c.render_device(s, small, 64, 48, out)
        assert c.render_device(s, u, W, H, out)["handed"] < 4_000
        c.device_free(out)
        s.close()


def test_every_ray_is_handed_over_once():
    """Thousands of faint proxies about one place: more rays give up their
    waiting hits than the hand-over buffer takes (a quarter of them)."""
    rng = np.random.default_rng(93)
    n = 3500
    d = rng.normal(size=(n, 3))
    rec = np.zeros((n, 80), np.float32)
    rec[:, 0:3] = 3.0 * d / np.linalg.norm(d, axis=1, keepdims=True) + (0.0, 0.0, -3.0)
    rec[:, 4:7] = 4.0
    rec[:, 8] = 1.0
    rec[:, 12] = 0.02
    u = view(W, H, pos=(0.0, 0.0, 30.0), k=16, T_min=0.01, hfov=3.0).uniforms
    with Context(0) as c:
        s = Scene(c, rec, 0.01)
        st = c.render(s, u, W, H, stats=True)[1]
        s.close()
    assert W * H // 4 < st["handed"] <= W * H == st["rays"]


def test_lists_that_cannot_be_had():
    """A batch whose lists need more memory than the GPU has left renders
    without them, and replays its graph instead of asking again each time; once
    memory is freed it has them."""
    import torch
    rec = small_scene(n=60_000, seed=94).gaussiansBuffer
    with Context(0) as c:
        s = Scene(c, rec, 0.01)
        u = view(160, 150, k=6, alpha_min=0.2, T_min=0.2).uniforms
        out = c.device_alloc(160 * 150 * 16)
        views = [(s, u, 160, 150, out)] * 40
        ref = np.empty((150, 160, 4), np.float32)
        with_lists = c.render_batch(views, device_outputs=True)[1]
        c.memcpy(ref.ctypes.data, out, ref.nbytes, 1)
    with Context(0) as c:
        s = Scene(c, rec, 0.01)
        out = c.device_alloc(160 * 150 * 16)
        views = [(s, u, 160, 150, out)] * 40
        # 40 x 60,000 proxies: 1.5 GB of lists
        ballast = c.device_alloc(torch.cuda.mem_get_info(0)[0] - (1 << 30))
        launches = []
        for _ in range(4):
            n0 = c.launch_count()
            st = c.render_batch(views, device_outputs=True)[1]
            launches.append(c.launch_count() - n0)
        img = np.empty_like(ref)
        c.memcpy(img.ctypes.data, out, img.nbytes, 1)
        assert np.array_equal(_bits(img), _bits(ref))
        assert st["proxy_tests"] != with_lists["proxy_tests"]
        assert launches[1:] == [1, 1, 1]
        c.device_free(ballast)
        again = c.render_batch(views, device_outputs=True)[1]
        c.memcpy(img.ctypes.data, out, img.nbytes, 1)
        assert np.array_equal(_bits(img), _bits(ref))
        assert abs(again["proxy_tests"] - with_lists["proxy_tests"]) < 0.1 * with_lists["proxy_tests"]


def test_lists_make_room_for_other_buffers():
    """With little memory left, a buffer of the program's own, then a larger
    image, are had at the lists' cost; views and gradients stay the same."""
    import torch
    rec = small_scene(n=60_000, seed=94).gaussiansBuffer
    w, h = 160, 150
    u = view(w, h, k=6, alpha_min=0.2, T_min=0.2).uniforms
    g = np.random.default_rng(94).normal(size=(h, w, 4)).astype(np.float32)
    with Context(0) as c:
        s = Scene(c, rec, 0.01)
        out = c.device_alloc(w * h * 16)
        views = [(s, u, w, h, out)] * 40
        ballast = c.device_alloc(torch.cuda.mem_get_info(0)[0] - (3 << 30))
        ref = c.render(s, u, w, h)
        grad = c.backward(s, u, w, h, g, mode=1)[0]
        assert c.render_batch(views, device_outputs=True)[1]["rays"] == 40 * w * h  # (1.5 GB of lists)
        more = c.device_alloc(torch.cuda.mem_get_info(0)[0] + (1 << 29))
        img = np.empty_like(ref)
        assert c.render_batch(views, device_outputs=True)[1]["rays"] == 40 * w * h
        c.memcpy(img.ctypes.data, out, img.nbytes, 1)
        assert np.array_equal(_bits(img), _bits(ref))
        got = c.backward(s, u, w, h, g, mode=1)[0]
        assert np.abs(got - grad).max() <= 1e-4 * np.abs(grad).max()  # (sums in another order)
        c.device_free(more)
        c.device_free(ballast)
        s.close()
