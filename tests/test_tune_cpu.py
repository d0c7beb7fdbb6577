"""A tuning result goes back through Context.set_tune as the launch it stands
for (the library behind the context is a stand-in)."""
import ctypes as C
import types

import pytest

from conftest import view
from gtrace import _lib as L
from gtrace.tracer import Context


class _Library:
    """gt_autotune and gt_autotune_batch return `found`; gt_set_tune keeps what it is given."""

    def __init__(self, found):
        self.found = found

    def gt_autotune(self, h, scene, u, w, hh, r):
        C.memmove(r, C.byref(self.found), C.sizeof(self.found))
        return 0

    def gt_autotune_batch(self, h, items, n, r):
        C.memmove(r, C.byref(self.found), C.sizeof(self.found))
        return 0

    def gt_set_tune(self, h, scene, u, w, hh, r):
        self.installed = L.TuneResult.from_buffer_copy(C.cast(r, C.POINTER(L.TuneResult)).contents)
        return 0


@pytest.mark.parametrize("mark", [0, 0x4C495354])
@pytest.mark.parametrize("batch", [False, True])
def test_a_result_goes_back_as_it_came(mark, batch):
    c = Context.__new__(Context)
    c._h = None
    c._lib = _Library(L.TuneResult(32, 8, 8, 4, 1.0, 2.0, 24, 16, 4, mark))
    scene = types.SimpleNamespace(handle=C.c_void_p(1))
    u = view(64, 48).uniforms
    r = c.autotune_batch([(scene, u, 64, 48)]) if batch else c.autotune(scene, u, 64, 48)
    keys = ("blocks_per_sm", "kbuf", "leaf_batch", "block_threads", "handoff_after", "default")
    c.set_tune(scene, u, 64, 48, **{k: r[k] for k in keys if k in r})
    got = c._lib.installed
    assert (got._pad, got.block_threads, got.blocks_per_sm) == (mark, 32, 8)
    assert (got.kbuf, got.leaf_batch, got.handoff_after) == (24, 16, 4)
