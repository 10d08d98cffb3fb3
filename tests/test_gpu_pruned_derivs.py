"""Derivatives of long tapes by pruning them per cell of points: the
interpreter's values and partials bit for bit (the general path, taken by
small calls and by static evaluation), for every count of points around the
cells' sizes and for coordinates that are not finite."""
import numpy as np
import pytest

from libfive_b200 import workloads as wl
from libfive_b200.shape import Shape, Tape, X, Y, Z

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def csg():
    return Tape(wl.random_csg(420, seed=5))     # over 4,096 clauses: never compiled


def general(tape, p):
    """The same points through calls too small for the pruned path."""
    parts = [tape.derivs(*[np.ascontiguousarray(c[i:i + 255]) for c in p]) for i in range(0, len(p[0]), 255)]
    return [np.concatenate([q[k] for q in parts]) for k in range(4)]


def same(a, b):
    return all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) |
               bool(np.all((x.view(np.uint32) == y.view(np.uint32)) | (np.isnan(x) & np.isnan(y))))
               for x, y in zip(a, b))


@pytest.mark.parametrize("n", [255, 256, 257, 4736, 18945, 40001])
def test_counts(gpu, csg, n):
    assert csg.n_clauses > 4096
    p = wl.uniform_points(n, seed=n)
    assert same(csg.derivs(*p), general(csg, p))


@pytest.mark.parametrize("spread", [0.0, 1e-6, 1e-2, 30.0])
def test_spreads(gpu, csg, spread):
    p = [np.float32(0.3) + np.float32(spread) * c for c in wl.uniform_points(3000, seed=2)]
    p = [np.ascontiguousarray(c, np.float32) for c in p]
    assert same(csg.derivs(*p), general(csg, p))


def test_not_finite(gpu, csg):
    p = list(wl.uniform_points(5000, seed=3))
    for k, v in enumerate((np.nan, np.inf, -np.inf, np.float32(3e38), np.float32(-0.0))):
        for a in range(3):
            p[a][100 * (k + 1) + a] = v
    assert same(csg.derivs(*p), general(csg, p))


def test_ties_and_nans_inside(gpu):
    """Points on ties of min and max, and operands that are NaN at points."""
    x, y, z = X(), Y(), Z()
    parts = []
    for i in range(700):
        a = (x - 0.01 * (i % 20)).abs().max((y - 0.05 * (i // 20)).abs()) - 0.01
        b = (x * (0.5 + 0.001 * i) - y).sqrt() if i % 50 == 7 else (z + 0.002 * i).abs() - 0.3
        parts.append(a.min(b) if i % 3 else b.max(a))
    while len(parts) > 1:
        parts = [(parts[i].min(parts[i + 1]) if i % 6 else parts[i].max(-parts[i + 1]))
                 if i + 1 < len(parts) else parts[i] for i in range(0, len(parts), 2)]
    s = parts[0]
    tape = Tape(s)
    assert tape.n_clauses > 4096
    g = (np.arange(30, dtype=np.float32) * np.float32(0.05)) - np.float32(0.5)
    p = [np.ascontiguousarray(c.ravel()) for c in np.meshgrid(g, g, g, indexing="ij")]
    assert same(tape.derivs(*p), general(tape, p))


def test_opcodes_outside_are_left_to_the_interpreter(gpu):
    """A tape with an opcode whose interval rule is only an enclosure."""
    s = wl.random_csg(420, seed=6).min(X().sin() + Shape.constant(2.0))
    tape = Tape(s)
    p = wl.uniform_points(3000, seed=4)
    assert same(tape.derivs(*p), general(tape, p))
