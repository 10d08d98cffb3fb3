"""Device memory of a mesh whose leaf tapes all have too many registers to be
decoded: no room is taken for decoded steps."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = """
import torch
from libfive_b200 import workloads as wl
from libfive_b200.shape import Tape
rng = wl.SplitMix64(3)
s = [wl.sphere([rng.uniform(-1, 1) for _ in range(3)], rng.uniform(0.15, 0.4)) for _ in range(32)]
while len(s) > 1:
    s = [wl.blend_stable(s[i], s[i + 1], 0.1) for i in range(0, len(s), 2)]
tape = Tape(s[0])
tape.render_mesh((-1.5,) * 3, (1.5,) * 3, 3.0)     # constant tables and the like
free = torch.cuda.mem_get_info()[0]
verts, tris = tape.render_mesh((-1.5,) * 3, (1.5,) * 3, 3.0 / 96)
torch.cuda.synchronize()
print(len(tris), (free - torch.cuda.mem_get_info()[0]) >> 20)
"""


def test_no_room_for_steps_that_cannot_be(gpu):
    """32 blends with min, in a process of its own (buffers are kept): the
    mesh takes some 350 MiB, and 36 bytes for each of its arena's 13 M
    clauses would be 450 MiB more."""
    r = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    triangles, mib = map(int, r.stdout.split())
    assert triangles > 100000
    assert mib < 350 + 450 // 2
