"""The reverse mode's two backward kernels of longer tapes: a call's number
of points chooses, whatever the tape was called with before, and no later
call waits for a compiler."""
import time

import numpy as np
import pytest
import torch

from libfive_b200 import workloads
from libfive_b200.fit import BatchedFit
from libfive_b200.shape import Tape

pytestmark = pytest.mark.gpu

# 1,000, 50,000 and 220,000 points take the form for three blocks an SM (as
# many waves as four blocks have), 120,001 and 300,007 the one for four.
SIZES = (1000, 50000, 120001, 220000, 300007)


def gradient(tape, n):
    p = [np.asarray(a, np.float32) for a in workloads.uniform_points(n, seed=3)]
    g = [np.zeros(n, np.float32) for _ in range(3)]
    gvars = np.zeros(tape.n_vars, np.float32)
    t = time.perf_counter()
    tape.grad(*p, gx=g[0], gy=g[1], gz=g[2], gvars=gvars)
    return time.perf_counter() - t, g, gvars


@pytest.mark.parametrize("order", [SIZES, SIZES[::-1], (120001, 1000, 120001, 220000)])
def test_any_order(gpu, order):
    # more than two segments of 192 clauses
    shape, vals, _ = workloads.fit_csg_vars(48, seed=78)
    tape = Tape(shape, vals)
    assert tape.n_clauses > 384
    first = gradient(tape, order[0])[0]
    for n in order:
        took, got, gvars = gradient(tape, n)
        assert took < 0.5 * first       # the first call compiled for a second
        _, want, _ = gradient(Tape(shape, vals), n)
        for a, b in zip(got, want):
            assert np.array_equal(a, b, equal_nan=True)
        assert np.isfinite(gvars).all()


def test_after_a_fit(gpu):
    """A fit step compiles the form for its own points; a call that wants the
    other one gets it."""
    shape, vals, _ = workloads.fit_csg_vars(48, seed=79)
    tape = Tape(shape, vals)
    points = [tuple(torch.from_numpy(a).cuda() for a in workloads.uniform_points(1000, seed=5))]
    BatchedFit([tape], points, lr=0.0).step()
    for n in (120001, 50000):
        _, got, _ = gradient(tape, n)
        _, want, _ = gradient(Tape(shape, vals), n)
        for a, b in zip(got, want):
            assert np.array_equal(a, b, equal_nan=True)
