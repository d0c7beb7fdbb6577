"""The scene build's kernels at the sizes where they can go wrong: hierarchy
clustering around a warp's and a node's cluster counts (16, 32), the one-pass
record kernel at block edges (64 records), for records of other strides and
for buffers that are not 16-byte aligned.  Hierarchies must satisfy the
invariants of test_bvh_gpu.py; images must be equal bit for bit (a scene's
records do not depend on how its buffer was read)."""
import numpy as np
import pytest

from conftest import small_scene, view
from gtrace.tracer import Scene
from test_bvh_gpu import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 15, 16, 17, 31, 32, 33, 34, 48, 63, 64, 65, 129, 1000])
def test_clustering_sizes(ctx, n):
    pg = small_scene(n=n, seed=90 + n)
    s = Scene(ctx, pg.gaussiansBuffer, 0.01)
    _check(s, pg.gaussiansBuffer, 0.01)
    s.close()


def test_collinear_proxies_of_growing_size(ctx):
    """Sizes and gaps that double from one proxy to the next: every merge's
    best partner is the cluster of all smaller ones."""
    n = 40
    rec = np.zeros((n, 80), np.float32)
    rec[:, 0] = 1.5 ** np.arange(n)
    rec[:, 4:7] = 0.1 * rec[:, 0:1]
    rec[:, 8] = 1.0
    rec[:, 12] = 0.5
    s = Scene(ctx, rec, 0.01)
    _check(s, rec, 0.01)
    s.close()


@pytest.mark.parametrize("n", [1, 63, 64, 65, 700])
@pytest.mark.parametrize("stride,offset", [(320, 4), (336, 0), (112, 0), (84, 4)])
def test_record_strides_and_alignment(ctx, n, stride, offset):
    """The same records at another stride or 4 bytes off a 16-byte boundary
    (the general path) as from a 320-byte aligned buffer."""
    pg = small_scene(n=n, seed=95)
    words = min(stride // 4, 80)
    full = pg.gaussiansBuffer.copy()
    n_sh = min(16, (stride - 64) // 16)
    full[:, 16 + 4 * n_sh:] = 0.0  # the coefficients such a record holds
    rows = np.zeros((n, stride // 4), np.float32)
    rows[:, :words] = full[:, :words]
    dev = ctx.device_alloc(rows.nbytes + 16)
    try:
        ctx.memcpy(dev + offset, rows.ctypes.data, rows.nbytes, 0)
        a = Scene(ctx, None, 0.05, device_ptr=dev + offset, n=n, stride=stride)
        b = Scene(ctx, full, 0.05)
        u = view(60, 44, k=5).uniforms
        np.testing.assert_array_equal(ctx.render(a, u, 60, 44).view(np.uint32),
                                      ctx.render(b, u, 60, 44).view(np.uint32))
        assert a.info()["n_kept"] == b.info()["n_kept"] and a.info()["bounds"] == b.info()["bounds"]
        a.close()
        b.close()
    finally:
        ctx.device_free(dev)


@pytest.mark.parametrize("n", [239, 255, 256, 257, 272, 273, 274, 511, 512, 513])
@pytest.mark.parametrize("spread", [1.0, 0.0])
def test_clustering_tasks_at_block_edges(ctx, n, spread):
    """Nodes whose leaves straddle two blocks of the search for the clusterings
    to start with; with spread 0 all codes are equal and only the positions in
    the sorted order tell the leaves apart."""
    rec = small_scene(n=n, seed=97).gaussiansBuffer.copy()
    rec[:, 0:3] *= spread
    s = Scene(ctx, rec, 0.01)
    _check(s, rec, 0.01)
    s.close()


@pytest.mark.parametrize("n", [2, 1023, 1024, 1025, 2049, 151_551, 151_553, 310_007])
def test_sort_at_block_edges(ctx, n):
    """Stretches of the sort that are full, one short and one over (148 blocks
    of 1,024 pairs), with many equal codes: leaves in Morton order, equal codes
    in the order of the particles."""
    rng = np.random.default_rng(n)
    rec = np.zeros((n, 80), np.float32)
    rec[:, 0:3] = rng.integers(0, 40, size=(n, 3))
    rec[0, 0:3], rec[1, 0:3] = 0.0, 39.0
    rec[:, 4:7] = 0.01
    rec[:, 8] = 1.0
    rec[:, 12] = 0.5
    for fast in (False, True):
        s = Scene(ctx, rec, 0.01, fast_build=fast)
        _, leaves, info = s.export_bvh()
        b = np.asarray(s.info()["bounds"], np.float64).reshape(2, 3)
        s.close()
        u = (rec[:, 0:3] - b[0]) / (b[1] - b[0]) * 1023.0
        assert np.abs(u - np.round(u)).min() > 1e-3  # no cell is decided by rounding
        q, code = np.floor(u).astype(np.uint32), np.zeros(n, np.uint32)
        for bit in range(10):
            for a in range(3):
                code |= ((q[:, a] >> bit) & 1) << (3 * bit + 2 - a)
        assert np.array_equal(leaves, np.argsort(code, kind="stable"))
