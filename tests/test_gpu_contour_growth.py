"""Slices whose clause lists, pruned tapes, leaf records and segments outgrow
the contourer's buffers, one after another in the same call, against the
oracle."""
import pytest

import oracle_ffi
from libfive_b200 import ffi, workloads
from libfive_b200.shape import Tape, X, Y, render_slice
from mesh_compare import same_contours
from oracle_ffi import OracleTape

pytestmark = pytest.mark.gpu

LO, HI = (-1.5, -1.5), (1.5, 1.5)


def rings(pitch, terms):
    """A lattice of circles under `terms` small bumps: three clauses each,
    and no min or max, so that no cell's list gets shorter."""
    a, b = X() % pitch - pitch / 2, Y() % pitch - pitch / 2
    s = (a.square() + b.square()).sqrt() - pitch * 0.3
    for i in range(terms):
        s = s + (X() * (0.1 + 0.03 * i) + Y()).square() * (1e-4 / (i + 1))
    return s


def check(shape, feature):
    got = render_slice(Tape(shape), LO, HI, 0.05, feature, 1e-8)
    want = oracle_ffi.render_contours(OracleTape(shape), LO, HI, 0.05, feature, 1e-8)[0]
    assert len(want) > 0 and len(got) == len(want)
    assert same_contours(got, want)


# Every one of 4,096 cells branches with a list of 160 clauses, and the slice
# has more leaves and segments than the buffers start with room for.
def test_lists_and_leaves(gpu):
    check(rings(0.03, 30), 3.0 / 512)


# Every buffer from its smallest; lists past their limit are given up, and a
# thread a cell goes on from there.
@pytest.mark.parametrize("shape, feature", [
    (rings(0.3, 20), 3.0 / 128),
    (workloads.spheres_union(64, seed=1), 3.0 / 700),
])
def test_from_the_smallest(gpu, shape, feature):
    lib = ffi.load()
    ffi.check(lib.lfb_debug_set(b"small_capacity", 1))
    try:
        check(shape, feature)
    finally:
        ffi.check(lib.lfb_debug_set(b"small_capacity", 0))
    check(shape, feature)
