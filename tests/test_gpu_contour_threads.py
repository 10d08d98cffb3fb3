"""Slices rendered by several threads at once: the buffers are one call's at
a time, the welding of its segments is not."""
import threading

import pytest

from libfive_b200 import workloads
from libfive_b200.shape import Tape, render_slice
from mesh_compare import same_contours

pytestmark = pytest.mark.gpu

LO, HI = (-1.5, -1.5), (1.5, 1.5)


@pytest.mark.parametrize("threads", [2, 6])
def test_threads(gpu, threads):
    jobs = [(Tape(workloads.spheres_union(8 + 9 * i, seed=i)), 0.05 * i, 3.0 / (100 + 300 * i)) for i in range(threads)]
    want = [render_slice(t, LO, HI, z, f) for t, z, f in jobs]
    got = [None] * threads

    def work(i):
        t, z, f = jobs[i]
        for _ in range(5):
            got[i] = render_slice(t, LO, HI, z, f)

    pool = [threading.Thread(target=work, args=(i,)) for i in range(threads)]
    [t.start() for t in pool]
    [t.join() for t in pool]
    for a, b in zip(got, want):
        assert len(b) > 0 and same_contours(a, b)
