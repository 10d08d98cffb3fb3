"""The branches that work sizes choose: a slice's levels on the list kernels
or a thread a cell, a height map's rounds over z slabs, the lanes of a fit
step, and the reverse mode's two backward kernels; each against the oracle
or the same work done one by one."""
import numpy as np
import pytest
import torch

import oracle_ffi
from libfive_b200 import workloads
from libfive_b200.fit import BatchedFit
from libfive_b200.shape import Shape, Tape, render_heightmap, render_slice
from mesh_compare import same_contours
from oracle_ffi import OracleTape

pytestmark = pytest.mark.gpu

X, Y, Z = Shape.X, Shape.Y, Shape.Z


# Depths 1 to 13, whose levels have from 4 to about 80,000 cells: one block a
# cell up to 2,048, one warp a cell below 8,192, one thread a cell above.
@pytest.mark.parametrize("cells", [2, 100, 1500, 6000])
def test_slice_levels(gpu, cells):
    shape = workloads.spheres_union(64, seed=1)
    lo, hi, feature = (-1.5, -1.5), (1.5, 1.5), 3.0 / cells
    got = render_slice(Tape(shape), lo, hi, 0.05, feature, 1e-8)
    want = oracle_ffi.render_contours(OracleTape(shape), lo, hi, 0.05, feature, 1e-8)[0]
    assert len(got) == len(want)
    assert same_contours(got, want)


def test_slice_of_many_registers(gpu):
    # more registers than the list kernels take: a thread a cell throughout.
    # Every part is read twice, the second time in the same order.
    parts = [(X() * (1.0 + 0.001 * i) + Y() * 0.01 * i).square() + Y().square() - 0.5
             for i in range(450)]
    least, most = parts[0], parts[0]
    for p in parts[1:]:
        least = least.min(p)
    for p in parts[1:]:
        most = most.max(p)
    shape = least.max(most - 1.0)
    tape = Tape(shape)
    assert tape.n_regs > 400
    got = render_slice(tape, (-1.5, -1.5), (1.5, 1.5), 0.0, 0.1, 1e-8)
    want = oracle_ffi.render_contours(OracleTape(shape), (-1.5, -1.5), (1.5, 1.5), 0.0, 0.1, 1e-8)[0]
    assert same_contours(got, want)


def undecided():
    """A floor under two slanted bars.  (X + 1) Y - X Y - Y is zero up to
    rounding, but its interval is not, so that the boxes above the floor stay
    undecided and are searched: the rounds run to the last slab."""
    fog = ((X() + 1.0) * Y() - X() * Y() - Y()) * 40.0 + 0.05
    bars = ((X() * 0.5 + Z() - 0.3).abs() - 0.02).max(Y().abs() - 0.1)
    return (Z() + 1.2).min(bars).min(fog)


# One slab, the bounds of the first rounds, and enough for every round.
@pytest.mark.parametrize("nz", [3, 16, 17, 33, 113, 530])
def test_heightmap_rounds(gpu, nz):
    lo, hi, res = (-1.0, -0.9, -1.5), (1.0, 1.0, 1.5), (18, 9, nz / 3.0)
    depth, norm = render_heightmap(Tape(undecided()), lo, hi, res)
    want_depth, want_norm = oracle_ffi.render_heightmap(OracleTape(undecided()), lo, hi, res)
    assert np.array_equal(depth, want_depth)
    assert np.array_equal(norm, want_norm)


# One shape, one lane each, and more shapes than lanes, of uneven sizes.
@pytest.mark.parametrize("count", [1, 2, 8, 9, 19])
def test_fit_side_by_side(gpu, count):
    shapes = [workloads.fit_csg_vars(4 + j % 5, seed=60 + j)[:2] for j in range(count)]
    points = [workloads.uniform_points(1 + 517 * (j % 4), seed=j) for j in range(count)]
    points = [tuple(torch.from_numpy(np.asarray(a, np.float32)).cuda() for a in p) for p in points]
    together = BatchedFit([Tape(s, v) for s, v in shapes], points, lr=1e-2)
    losses = together.step().cpu().numpy()
    for j, (s, v) in enumerate(shapes):
        alone = BatchedFit([Tape(s, v)], [points[j]], lr=1e-2)
        # f and its mean are the same numbers in the same order
        assert alone.step().cpu().numpy()[0] == losses[j]
        a, b = int(together.var_offsets[j]), int(together.var_offsets[j + 1])
        # the first moment is (1 - beta1) times the gradient, a sum of up to
        # 1,552 points in an order that atomics choose: 1,552 roundings of
        # 2^-24 of partial sums, taken to stay below 64 times the largest
        # component
        g, want = together.m[a:b].cpu().numpy(), alone.m[:b - a].cpu().numpy()
        np.testing.assert_allclose(g, want, rtol=0, atol=1552 * 2.0 ** -24 * 64 * np.abs(want).max())


# A tape of more than two segments of 192 clauses, at numbers of points whose
# first call compiles the backward kernel for three blocks an SM (50,000 and
# 300,007), or for four (120,001), and then both.
@pytest.mark.parametrize("sizes", [(50000, 120001, 300007), (120001, 50000)])
def test_gradient_kernels(gpu, sizes):
    shape, vals, _ = workloads.fit_csg_vars(32, seed=77)
    tape, few = Tape(shape, vals), 1000
    assert tape.n_clauses > 384

    def gradient(t, p):
        g = [np.zeros(len(p[0]), np.float32) for _ in range(3)]
        gvars = np.zeros(t.n_vars, np.float32)
        t.grad(*p, gx=g[0], gy=g[1], gz=g[2], gvars=gvars)
        return g

    for n in sizes:
        pts = [np.asarray(a, np.float32) for a in workloads.uniform_points(n, seed=3)]
        got = gradient(tape, pts)
        # the points' own gradients are the same numbers from the kernel that
        # a tape of its own compiles for a few points
        for at in (0, n - few):
            want = gradient(Tape(shape, vals), [a[at:at + few] for a in pts])
            for a, b in zip(got, want):
                assert np.array_equal(a[at:at + few], b, equal_nan=True)
