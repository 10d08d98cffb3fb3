"""A cancel flag raised late in a mesh, while the dual walk runs."""
import ctypes
import threading
import time

import pytest

from libfive_b200 import ffi, workloads
from libfive_b200.shape import Tape

pytestmark = pytest.mark.gpu

REGION = ffi.Region3(*[ffi.Interval(-1.5, 1.5)] * 3)


def test_cancel_during_the_walk(gpu):
    """64 spheres at depth 10: the walk is the last eighth of some 30 ms.  The
    flag goes up within it (at 94 to 97 % of the call); most of twenty such
    calls end cancelled (a busy host may raise it too late)."""
    lib = ffi.load()
    tape = Tape(workloads.spheres_union(64, seed=1))

    def render(flag):
        m = lib.lfb_render_mesh(tape.ptr, REGION, ffi.MeshSettings(3.0 / 1000, 1e-8, ctypes.pointer(flag)), None)
        if m:
            lib.libfive_mesh_delete(m)
        return bool(m)

    flag = ctypes.c_int32(0)
    for _ in range(4):
        start = time.perf_counter()
        assert render(flag)
        total = time.perf_counter() - start
    cancelled = 0
    for k in range(20):
        flag.value = 0

        def up():
            end = time.perf_counter() + (0.94 + 0.0015 * k) * total
            while time.perf_counter() < end:
                pass
            flag.value = 1

        t = threading.Thread(target=up)
        t.start()
        if not render(flag):
            assert ffi.last_error()[0] == -5     # LFB_E_CANCELLED
            cancelled += 1
        t.join()
    assert cancelled > 10
    flag.value = 0
    assert render(flag)
