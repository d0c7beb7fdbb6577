"""Images in host memory: the trace kernels write them directly only where they
are page-locked from the first byte to the last."""
import numpy as np
import pytest

from conftest import small_scene, view
from gtrace._lib import GTraceError
from gtrace.tracer import Scene
from gtrace.uniforms import with_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(60, 40), (260, 200)])  # a warp per ray, lists
@pytest.mark.parametrize("antialias", [False, True])
@pytest.mark.parametrize("locked", ["first", "last", "all"])
def test_partly_locked_images(ctx, w, h, antialias, locked):
    """Partly locked: CUDA refuses the copy from the staging image (an error, and
    the context stays usable) or takes it; the image is right or untouched."""
    import torch
    s = Scene(ctx, small_scene(n=1500, seed=96).gaussiansBuffer, 0.01)
    u = view(w, h, k=6).uniforms
    frames = range(2) if antialias else [0]
    ref = np.zeros((h, w, 4), np.float32)
    for f in frames:
        ctx.render(s, with_fields(u, accumulated_frames=f), w, h, out=ref, antialias=antialias)
    page = 4096
    buf = np.zeros(ref.nbytes + 2 * page, np.uint8)
    at = -buf.ctypes.data % page
    img = buf[at:at + ref.nbytes].view(np.float32).reshape(h, w, 4)
    half = ref.nbytes // 2 // page * page
    start, size = {"first": (0, half), "last": (half, ref.nbytes - half), "all": (0, ref.nbytes)}[locked]
    rt = torch.cuda.cudart()
    assert int(rt.cudaHostRegister(img.ctypes.data + start, size, 0)) == 0
    try:
        try:
            for f in frames:
                ctx.render(s, with_fields(u, accumulated_frames=f), w, h, out=img, antialias=antialias)
            assert np.array_equal(img, ref)
        except GTraceError:
            assert locked != "all"
        ctx.synchronize()
    finally:
        rt.cudaHostUnregister(img.ctypes.data + start)
    assert np.array_equal(ctx.render(s, u, w, h), ctx.render(s, u, w, h))
    s.close()
