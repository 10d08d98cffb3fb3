"""The leaf stage's fused interpreter steps and its deferred check of
zero-valued samples, against the oracle's meshes: tapes around the sizes of
its buffers, every kind of step, and samples that the check sends back."""
import pytest

from libfive_b200 import workloads as wl
from libfive_b200.shape import Tape, X, Y, Z

pytestmark = pytest.mark.gpu

LO, HI = (-1.5, -1.5, -1.5), (1.5, 1.5, 1.5)


def chain(n):
    """n spheres in a row, each joined to the ones before it: 11 n - 1
    clauses, all of them needed in the coarse cells' tapes."""
    s = None
    for i in range(n):
        c = wl.sphere([-0.9 + 1.8 * i / max(1, n - 1), 0.13 * (-1) ** i, 0.05], 0.31)
        s = c if s is None else s.min(c)
    return s


def many_registers(n):
    """A value that needs about n registers at once: a product of n shifted
    coordinates, all made before the first is used."""
    parts = [(X() * (1.0 + 0.01 * i) + Y() * 0.1 * i).square() + Z().square() for i in range(n)]
    while len(parts) > 1:
        parts = [parts[i].min(parts[i + len(parts) // 2]) for i in range(len(parts) // 2)] + \
            ([parts[-1]] if len(parts) % 2 else [])
    return parts[0] - 0.5


def plateau():
    """Negative below x = -0.2, exactly zero with a zero gradient up to 0.3,
    positive above: the zero samples of the edge search are outside."""
    x = X() + Y().square() * 0.25
    return (x + 0.2).min((x - 0.3).max(0.0))


SHAPES = {
    "one sphere": lambda: chain(1),
    "5 spheres": lambda: chain(5),         # around 56 and 64 clauses and steps
    "6 spheres": lambda: chain(6),
    "20 spheres": lambda: chain(20),       # more steps than one buffer holds
    "8 registers": lambda: many_registers(8),
    "20 registers": lambda: many_registers(20),
    "box": lambda: wl.box([-0.25, 0.25, -0.125], 0.5),      # zeros on the lattice
    "negated": lambda: wl.difference(wl.box([0.1, -0.2, 0.3], 0.7), wl.zcylinder([-0.1, -0.1, 0.0], 0.3, 0.9)),
    "rare steps": lambda: (X().square() + Y().square() * 0.5 + (Z() / (X().square() + 2.0)).square()).sqrt()
    .max(1.0 - (X() + 1.1)) - 0.8,
    "immediates": lambda: ((0.3 - X()).max(-0.4).min(0.9).abs() * 1.5 + Y().abs() * 0.75 + (-Z()).abs()) - 0.8,
    "plateau": plateau,
    "plateau and sphere": lambda: plateau().max(wl.sphere([0, 0, 0], 1.1)),
}


@pytest.mark.parametrize("name", sorted(SHAPES))
@pytest.mark.parametrize("cells", [1, 2, 5, 24])
def test_mesh_is_the_oracles(gpu, name, cells):
    from mesh_compare import oracle_mesh, same_mesh
    from oracle_ffi import OracleTape
    s = SHAPES[name]()
    v, t = Tape(s).render_mesh(LO, HI, 3.0 / cells)
    ov, ot = oracle_mesh(OracleTape(s), LO, HI, 3.0 / cells)
    assert same_mesh(v, t, ov, ot)
    if cells == 24:
        assert len(t) > 0


def test_plateau_with_small_buffers(gpu):
    """No room for the deferred samples: every group with one is searched again."""
    from libfive_b200 import ffi
    from mesh_compare import oracle_mesh, same_mesh
    from oracle_ffi import OracleTape
    s = SHAPES["plateau and sphere"]()
    ffi.check(ffi.load().lfb_debug_set(b"small_capacity", 1))
    try:
        v, t = Tape(s).render_mesh(LO, HI, 0.125)
    finally:
        ffi.check(ffi.load().lfb_debug_set(b"small_capacity", 0))
    ov, ot = oracle_mesh(OracleTape(s), LO, HI, 0.125)
    assert len(t) > 0 and same_mesh(v, t, ov, ot)
