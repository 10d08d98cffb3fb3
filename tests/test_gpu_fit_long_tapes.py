"""A fit step of long tapes: two or three shapes whose points fill the GPU run
one after another, fewer or more points side by side; the same losses as each
shape alone."""
import numpy as np
import pytest
import torch

from libfive_b200 import workloads
from libfive_b200.fit import BatchedFit
from libfive_b200.shape import Tape

pytestmark = pytest.mark.gpu


# 56,832 and 113,664 points are half a wave and a wave of the backward kernel.
@pytest.mark.parametrize("sizes", [(56832, 56832), (56833, 113664), (56833, 113665), (60000, 60000, 60000)])
def test_two_and_three(gpu, sizes):
    shapes = [workloads.fit_csg_vars(112, seed=90 + j)[:2] for j in range(len(sizes))]
    points = [tuple(torch.from_numpy(a).cuda() for a in workloads.uniform_points(n, seed=n + j))
              for j, n in enumerate(sizes)]
    tapes = [Tape(s, v) for s, v in shapes]
    assert min(t.n_clauses for t in tapes) > 1536
    losses = BatchedFit(tapes, points, lr=1e-2).step().cpu().numpy()
    for j, (s, v) in enumerate(shapes):
        assert BatchedFit([Tape(s, v)], [points[j]], lr=1e-2).step().cpu().numpy()[0] == losses[j]
    assert np.isfinite(losses).all()
