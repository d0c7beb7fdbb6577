"""Uploads from host buffers that are page-locked in part."""
import numpy as np
import pytest

from conftest import small_scene, view
from gtrace.tracer import Scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2000, 20000])  # below and above one direct copy (4 MB)
@pytest.mark.parametrize("locked", ["first", "last", "all"])
def test_partly_locked_records(ctx, n, locked):
    import torch
    rec = np.ascontiguousarray(small_scene(n=n, seed=95).gaussiansBuffer, np.float32).reshape(-1)
    u = view(48, 40, k=6).uniforms
    s = Scene(ctx, rec.reshape(-1, 80), 0.01)
    ref = ctx.render(s, u, 48, 40)
    s.close()
    page = 4096
    buf = np.empty(rec.nbytes + 2 * page, np.uint8)
    at = -buf.ctypes.data % page
    host = buf[at:at + rec.nbytes].view(np.float32)
    host[:] = rec
    half = rec.nbytes // 2 // page * page
    start, size = {"first": (0, half), "last": (half, rec.nbytes - half), "all": (0, rec.nbytes)}[locked]
    rt = torch.cuda.cudart()
    assert int(rt.cudaHostRegister(host.ctypes.data + start, size, 0)) == 0
    try:
        s = Scene(ctx, host.reshape(-1, 80), 0.01)
        assert np.array_equal(ctx.render(s, u, 48, 40), ref)
        s.close()
    finally:
        rt.cudaHostUnregister(host.ctypes.data + start)
