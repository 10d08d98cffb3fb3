"""The leaf kernel's register file, which the tapes of a large mesh choose
(thousands of leaf groups): tapes of up to 8 registers, of 9 to 16, of more,
and mixed, against the oracle's meshes."""
import pytest

from libfive_b200 import workloads as wl
from libfive_b200.shape import Tape, X, Y, Z
from mesh_compare import oracle_mesh, same_mesh
from oracle_ffi import OracleTape

pytestmark = pytest.mark.gpu

LO, HI = (-1.5, -1.5, -1.5), (1.5, 1.5, 1.5)


def spread(n):
    """A smooth shape whose tape needs about n registers at once and has no
    min or max that could shorten it: n terms, each read by a first chain of
    sums and again by a second."""
    parts = [(X() * (1.0 + 0.01 * i) + Y() * 0.1 * i).square() + Z().square() for i in range(n)]
    a, b = parts[0], parts[-1]
    for p in parts[1:]:
        a = (a.square() + p.square()).sqrt()
    for p in parts[:-1]:
        b = (b.square() + p).sqrt()
    return (a + b) * (2.0 / n) - 1.0


SHAPES = {
    "few registers": (lambda: wl.spheres_union(24, seed=3), 0, 8),
    "9 to 16": (lambda: spread(10), 9, 16),
    "more": (lambda: spread(24), 17, 400),
    "9 to 16 and few": (lambda: spread(10).max(wl.sphere([1.3, 0, 0], 0.9)).min(wl.spheres_union(12, seed=3)), 9, 30),
    "more and few": (lambda: spread(24).min(wl.spheres_union(40, seed=3)), 17, 400),
}


@pytest.mark.parametrize("name", sorted(SHAPES))
def test_mesh_is_the_oracles(gpu, name):
    make, least, most = SHAPES[name]
    s = make()
    tape = Tape(s)
    assert least <= tape.n_regs <= most
    v, t = tape.render_mesh(LO, HI, 3.0 / 80)
    ov, ot = oracle_mesh(OracleTape(s), LO, HI, 3.0 / 80)
    assert len(t) > 4 * 2368    # more groups than all run at once
    assert same_mesh(v, t, ov, ot)
