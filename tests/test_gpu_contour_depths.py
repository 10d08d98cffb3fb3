"""Slices whose quadtree is deeper than the list kernels' packed coordinates
reach (21 bits an axis): a small circle in a large region."""
import numpy as np
import pytest

import oracle_ffi
from libfive_b200.shape import Tape, X, Y, render_slice
from mesh_compare import same_contours
from oracle_ffi import OracleTape

pytestmark = pytest.mark.gpu


# cells of 2000 / 2^L units; the circle is a few hundred of them around
@pytest.mark.parametrize("levels", [20, 21, 22, 23, 24])
def test_small_circle_in_a_large_region(gpu, levels):
    size = 2000.0 / 2 ** levels
    r = 60 * size
    circle = ((X() - r * 1.3).square() + (Y() + r * 0.7).square()).sqrt() - r
    lo, hi = (-1000.0, -1000.0), (1000.0, 1000.0)
    got = render_slice(Tape(circle), lo, hi, 0.0, size * 1.2, 1e-8)
    want = oracle_ffi.render_contours(OracleTape(circle), lo, hi, 0.0, size * 1.2, 1e-8)[0]
    assert len(want) == 1 and len(want[0]) > 100
    assert len(got) == 1 and same_contours(got, want)
    assert np.abs(np.hypot(got[0][:, 0] - r * 1.3, got[0][:, 1] + r * 0.7) - r).max() < size
