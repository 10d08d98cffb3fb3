"""Derivatives of long tapes pruned per cell of points, where an operation's
interval ends at a value at which the operation jumps or overflows: the whole
tape's values and partials, bit for bit, taken from calls too small for the
pruned path."""
import numpy as np
import pytest

from libfive_b200 import workloads as wl
from libfive_b200.shape import Shape, Tape, X, Y, Z

pytestmark = pytest.mark.gpu


def long_tape(s):
    """s over a union of spheres that makes the tape too long to be compiled
    and has values between -2 and 4 in the region of the points; the sum
    reads both everywhere."""
    tape = Tape(wl.spheres_union(400, seed=9) + s)
    assert tape.n_clauses > 4096
    return tape


def same_as_whole_tape(tape, p):
    got = tape.derivs(*p)
    parts = [tape.derivs(*[np.ascontiguousarray(c[i:i + 255]) for c in p]) for i in range(0, len(p[0]), 255)]
    want = [np.concatenate([q[k] for q in parts]) for k in range(4)]
    return all(np.array_equal(a.view(np.uint32)[~np.isnan(b)], b.view(np.uint32)[~np.isnan(b)]) and
               np.array_equal(np.isnan(a), np.isnan(b)) for a, b in zip(got, want))


def points_ending_at_zero(sign, zero, n=4096):
    """Half of the points at x = zero, the others on one side of it, so that
    many cells' boxes end there."""
    rng = np.random.default_rng(5)
    x = (sign * rng.uniform(0.0, 0.9, n)).astype(np.float32)
    x[rng.random(n) < 0.5] = zero
    y, z = (rng.uniform(-1.0, 1.0, n).astype(np.float32) for _ in range(2))
    return x, y, z


# min(1 / x, -1) below x = 0 and max(1 / x, 1) above it: the whole tape takes
# the constant at a zero of the other side's sign.
@pytest.mark.parametrize("zero", [0.0, -0.0])
@pytest.mark.parametrize("sign", [-1.0, 1.0])
def test_reciprocal_up_to_zero(gpu, sign, zero):
    r = Shape.new("recip", X())
    tape = long_tape(r.min(-1.0).max(-50.0) if sign < 0 else r.max(1.0).min(50.0))
    assert same_as_whole_tape(tape, points_ending_at_zero(sign, np.float32(zero)))


# inf - inf is NaN at the points of a corner, where both terms overflow; its
# absolute value is never below zero, and so decides against -1 unless the
# interval says that it may be NaN.
def test_difference_of_infinities(gpu):
    d = ((X() * 100.0).exp() - (Y() * 100.0).exp()).abs()
    tape = long_tape(d.min(-1.0) + (-d).max(1.0))
    x, y, z = (np.random.default_rng(a).uniform(0.8, 1.0, 4096).astype(np.float32) for a in range(3))
    assert same_as_whole_tape(tape, (x, y, z))
    # infinite coordinates under a linear difference
    tape = long_tape((X() * 0.8 - Y() * 0.6).square().min(-1.0))
    x[::7], y[::7] = np.inf, np.inf
    assert same_as_whole_tape(tape, (x, y, z))


# log(x) over [lo, 0] is -inf at the points at zero and NaN at the others: as
# a second operand of min it is the value at zero, although the other operand
# is the value elsewhere.
@pytest.mark.parametrize("zero", [0.0, -0.0])
def test_logarithm_up_to_zero(gpu, zero):
    one = Shape.constant(1.0)
    tape = long_tape(one.min(X().log()).max(0.5))
    assert same_as_whole_tape(tape, points_ending_at_zero(-1.0, np.float32(zero)))


# Cells with a few points that have a NaN coordinate, or a NaN constant.
def test_nan_among_others(gpu):
    one = Shape.constant(1.0)
    x, y, z = (np.random.default_rng(a).uniform(-3.0, 0.0, 4096).astype(np.float32) for a in range(3))
    x[100], y[200], z[300] = np.nan, np.nan, np.nan
    assert same_as_whole_tape(long_tape(one.min(X()).max(0.5) + one.min(Y() + Z()).max(-0.5)), (x, y, z))
    nan = Shape.constant(float("nan"))
    assert same_as_whole_tape(long_tape(one.min(X() + nan).max(0.5)), (x, y, z))


UNARY = ("square", "sqrt", "neg", "abs", "recip", "exp", "log", "const-var")
BINARY = ("add", "sub", "mul", "div", "min", "max")
SPECIAL = (0.0, -0.0, 1.0, -1.0, 88.0, 3e38, -3e38, 1e-40, np.inf, -np.inf, np.nan)


def random_tree(rng, depth):
    if depth == 0:
        if rng.random() < 0.2:
            return Shape.constant(float(rng.choice(SPECIAL)))
        # a factor of its own, so that no two subtrees are one
        return (X, Y, Z)[rng.integers(3)]() * float(rng.uniform(0.5, 2.0))
    if rng.random() < 0.35:
        return Shape.new(str(rng.choice(UNARY)), random_tree(rng, depth - 1))
    op = str(rng.choice(BINARY if rng.random() < 0.5 else BINARY[4:]))
    return Shape.new(op, random_tree(rng, depth - 1), random_tree(rng, depth - 1))


# Every operation that the pruned path takes, over constants and coordinates
# at its edges: 500 trees, joined twelve at a time and those one by one.
@pytest.mark.parametrize("seed", [0, 1, 2, 3])
def test_random_trees(gpu, seed):
    rng = np.random.default_rng(seed)
    parts = [random_tree(rng, int(rng.integers(3, 6))) for _ in range(500)]
    parts = [t.min(0.01 * i) if i % 2 else Shape.constant(-0.01 * i).max(t) for i, t in enumerate(parts)]
    for width in (12, 50):
        parts = [parts[i:i + width] for i in range(0, len(parts), width)]
        for p in parts:
            while len(p) > 1:
                p[:2] = [p[0].min(p[1]) if rng.random() < 0.5 else p[0].max(p[1])]
        parts = [p[0] for p in parts]
    tape = Tape(parts[0])
    assert tape.n_clauses > 4096 and tape.n_regs <= 100 and tape.n_choices >= tape.n_clauses // 64
    p = []
    for _ in range(3):
        v = (rng.uniform(-2.0, 2.0, 5000) * (1.0, 1e-3, 100.0, 1e19)[seed]).astype(np.float32)
        at = rng.random(5000) < 0.15
        v[at] = rng.choice(np.array(SPECIAL, np.float32), at.sum())
        p.append(v)
    assert same_as_whole_tape(tape, p)
