"""Meshes of tapes that were made a moment ago, on the batch's own streams,
while the legacy stream is busy: the tapes' uploads are ordered before any
stream's work, so each mesh is the one that a single call gives."""
import pytest
import torch

from libfive_b200 import workloads
from libfive_b200.shape import Tape, render_meshes
from mesh_compare import same_mesh

pytestmark = pytest.mark.gpu

LO, HI = (-1.5, -1.5, -1.5), (1.5, 1.5, 1.5)


# Small tapes (their uploads fit the command buffer) and larger ones.
@pytest.mark.parametrize("prims", [3, 30, 300])
def test_batch_of_fresh_tapes(gpu, prims):
    shapes = [workloads.random_csg(prims, seed=90 + k, size=(0.1, 0.4)) for k in range(8)]
    want = [Tape(s).render_mesh(LO, HI, 3.0 / 32) for s in shapes]
    a = torch.rand(4096, 4096, device="cuda")
    for _ in range(4):
        for _ in range(10):
            a = (a @ a).clamp_(0.0, 1.0)
        got = render_meshes([(Tape(s), LO, HI, 3.0 / 32) for s in shapes], workers=4)
        for g, w in zip(got, want):
            assert same_mesh(*g, *w)
