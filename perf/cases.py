"""The work that programs have this library do, as cases to be timed.

A case is a dict of plain values.  `listed()` gives the ones that stand for
the library's uses, `draw(rng)` one more of the same ranges, `prepare` what a
program holds before the call (trees, tapes, points on the GPU), `run` one
pass through the public entry points, `work` what such a pass cannot do
without and `exact` its result in 64 bits.

Two things every case follows.  A program builds its tape once and calls it
many times: the evaluation cases keep one tape per shape and get new points
(or new free variables) with every seed, while the meshing cases get a new
tree with every seed, since a program that meshes has edited its model.  The
mesher and the contourer number vertices, triangles and contours in the order
in which the GPU finishes them, so the same call gives the same mesh in
another order: `run` takes such a result on to the GPU, as a program that
goes on with it there does, and sorts it there (`one_order`).
"""
import math
import random

import numpy as np
import torch

from libfive_b200 import shape as lf
from libfive_b200 import workloads as wl
from libfive_b200.fit import BatchedFit

LOWER, UPPER = (-1.5, -1.5, -1.5), (1.5, 1.5, 1.5)
SIDE = 3.0


def listed():
    return [
        # A preview of a small part while its author edits it: the smallest
        # mesh, all latency.
        {"name": "mesh part 24 preview", "kind": "mesh", "model": "part", "n": 24, "cells": 30},
        # The 64-sphere union at 64 voxels per unit.
        {"name": "mesh spheres 64", "kind": "mesh", "model": "spheres", "n": 64, "cells": 192},
        # An ordinary assembly at an odd resolution.
        {"name": "mesh part 300", "kind": "mesh", "model": "part", "n": 300, "cells": 333},
        # The large CSG: 2,000 primitives, octree to depth 10.
        {"name": "mesh csg 2000", "kind": "mesh", "model": "csg", "n": 2000, "cells": 1024},
        # Many models of uneven size in one call, each at its own resolution.
        {"name": "mesh batch 16", "kind": "batch", "count": 16, "n_lo": 8, "n_hi": 1000, "cells_lo": 64,
         "cells_hi": 384},
        # One layer of a print: a slice of a large model at a fine step.
        {"name": "slice csg 1000", "kind": "slice", "n": 1000, "cells": 2048},
        # A rendered view: depth and normals.
        {"name": "heightmap 512", "kind": "heightmap", "n": 32, "voxels": 512},
        # A few thousand probe points: latency and one launch.
        {"name": "values 1000", "kind": "values", "model": "spheres", "n": 64, "points": 1000},
        # A lattice's worth of points.
        {"name": "values 2097152", "kind": "values", "model": "spheres", "n": 64, "points": 2097152},
        # Values and derivatives over a tape far too long to be compiled whole.
        {"name": "derivs csg 1500", "kind": "derivs", "model": "csg", "n": 1500, "points": 100003},
        # Loss and gradient with respect to every free variable.
        {"name": "loss grad 64", "kind": "grad", "n": 64, "points": 1000000},
        # One step of fitting several shapes' free variables to points.
        {"name": "fit 6", "kind": "fit", "shapes": 6, "n": 24, "points": 65536},
    ]


def log_between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("mesh", "mesh", "mesh", "batch", "slice", "heightmap", "values", "derivs", "grad", "fit"))
    if kind == "mesh":
        model = rng.choice(("part", "spheres", "csg"))
        n = log_between(rng, 8, {"part": 600, "spheres": 128, "csg": 2000}[model])
        return {"kind": kind, "model": model, "n": n,
                "cells": log_between(rng, 24, {"part": 500, "spheres": 250, "csg": 1000}[model])}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(4, 16), "n_lo": 8, "n_hi": log_between(rng, 64, 1000),
                "cells_lo": 32, "cells_hi": log_between(rng, 64, 384)}
    if kind == "slice":
        return {"kind": kind, "n": log_between(rng, 16, 1000), "cells": log_between(rng, 100, 2048)}
    if kind == "heightmap":
        return {"kind": kind, "n": rng.randint(8, 32), "voxels": log_between(rng, 64, 512)}
    if kind == "values":
        return {"kind": kind, "model": "spheres", "n": rng.randint(8, 64), "points": log_between(rng, 100, 2000000)}
    if kind == "derivs":
        model = rng.choice(("spheres", "csg"))
        n = rng.randint(8, 64) if model == "spheres" else log_between(rng, 400, 1500)
        return {"kind": kind, "model": model, "n": n,
                "points": log_between(rng, 1000, 2000000 if model == "spheres" else 100000)}
    if kind == "grad":
        return {"kind": kind, "n": rng.randint(8, 64), "points": log_between(rng, 10000, 1000000)}
    return {"kind": kind, "shapes": rng.randint(2, 6), "n": rng.randint(8, 24),
            "points": log_between(rng, 4096, 65536)}


# Models, as plain data, so that a shape and its values in 64 bits come from
# the same numbers: ("sphere", c, r), ("box", c, s), ("cyl", c, r, h) and
# (operator, a, b).


def uniform3(rng, a):
    return [rng.uniform(-a, a) for _ in range(3)]


def pairwise(nodes, operator):
    """The nodes joined by a balanced tree of operators."""
    while len(nodes) > 1:
        nodes = [(operator(), nodes[i], nodes[i + 1]) if i + 1 < len(nodes) else nodes[i]
                 for i in range(0, len(nodes), 2)]
    return nodes[0]


def spheres_model(n, rng):
    return pairwise([("sphere", uniform3(rng, 1.0), rng.uniform(0.1, 0.35)) for _ in range(n)],
                    lambda: "union")


def feature(i, rng, size):
    c, s = uniform3(rng, 1.0), rng.uniform(*size)
    if i % 3 == 0:
        return ("sphere", c, s)
    if i % 3 == 1:
        return ("box", c, s)
    return ("cyl", c, s, rng.uniform(*size))


def csg_model(n, rng):
    """Random CSG with the weights of workloads.CSG_WEIGHTS."""
    names = ("union", "blend", "difference", "intersection")
    return pairwise([feature(i, rng, (0.02, 0.2)) for i in range(n)],
                    lambda: rng.choices(names, wl.CSG_WEIGHTS)[0])


def part_model(n, rng):
    """A block with bosses added to it and holes taken out of it."""
    add = [("box", [0.0, 0.0, 0.0], 0.7)]
    cut = []
    for i in range(n - 1):
        (add if i % 2 else cut).append(feature(i // 2, rng, (0.05, 0.25)))
    body = pairwise(add, lambda: rng.choices(("union", "blend"), (0.9, 0.1))[0])
    return ("difference", body, pairwise(cut, lambda: "union")) if cut else body


def model_of(case, rng):
    return {"spheres": spheres_model, "csg": csg_model, "part": part_model}[case.get("model", "csg")](case["n"], rng)


def build(node, leaf, join):
    return leaf(node) if node[0] in ("sphere", "box", "cyl") else join(
        node[0], build(node[1], leaf, join), build(node[2], leaf, join))


def to_shape(node):
    def leaf(p):
        return {"sphere": wl.sphere, "box": wl.box, "cyl": wl.zcylinder}[p[0]](*p[1:])

    def join(name, a, b):
        return {"union": wl.union, "blend": wl.blend_stable, "difference": wl.difference,
                "intersection": wl.intersection}[name](a, b)

    return build(node, leaf, join)


def blend64(a, b, m=0.05):
    k = 2.75 / m ** 2
    return torch.minimum(a, b) - torch.log1p(torch.exp(-k * (a - b).abs())) / k


def to_double(node, x, y, z):
    """The model's values at points, in 64 bits."""
    def f32(v):
        return float(np.float32(v))

    def leaf(p):
        d = [x - f32(p[1][0]), y - f32(p[1][1]), z - f32(p[1][2])]
        if p[0] == "sphere":
            return (d[0] ** 2 + d[1] ** 2 + d[2] ** 2).sqrt() - f32(p[2])
        if p[0] == "box":
            return torch.maximum(torch.maximum(d[0].abs(), d[1].abs()), d[2].abs()) - f32(p[2])
        return torch.maximum((d[0] ** 2 + d[1] ** 2).sqrt() - f32(p[2]), d[2].abs() - f32(p[3]))

    def join(name, a, b):
        if name == "blend":
            return blend64(a, b)
        return {"union": torch.minimum, "intersection": torch.maximum}[name](a, b) \
            if name != "difference" else torch.maximum(a, -b)

    return build(node, leaf, join)


def points_in(n, seed, near=1.5):
    """n float32 points on the GPU, uniform in a cube."""
    g = torch.Generator("cuda").manual_seed(seed)
    return [torch.rand(n, generator=g, device="cuda") * (2 * near) - near for _ in range(3)]


TAPES = {}


def kept(key, make):
    """What a program builds once for a model and keeps."""
    if key not in TAPES:
        TAPES[key] = make()
    return TAPES[key]


# Free-variable shapes: spheres (cx, cy, cz, r), joined pairwise by blends.


def variable_shape(n):
    """(tape, for each of its variables the place of it in [cx, cy, cz, r] * n)."""
    variables, spheres = [], []
    x, y, z = lf.X(), lf.Y(), lf.Z()
    for _ in range(n):
        cx, cy, cz, r = (lf.Shape.var() for _ in range(4))
        variables += [cx, cy, cz, r]
        spheres.append(((x - cx).square() + (y - cy).square() + (z - cz).square()).sqrt() - r)
    while len(spheres) > 1:
        spheres = [wl.blend_stable(spheres[i], spheres[i + 1]) if i + 1 < len(spheres) else spheres[i]
                   for i in range(0, len(spheres), 2)]
    tape = lf.Tape(spheres[0])
    at = {v.id(): i for i, v in enumerate(variables)}
    return tape, [at[i] for i in tape.var_ids()], variables


def sphere_parameters(n, seed):
    rng = random.Random(seed)
    return [v for _ in range(n) for v in uniform3(rng, 1.0) + [rng.uniform(0.1, 0.35)]]


def values64(params, x, y, z):
    """The blended spheres' values in 64 bits; params: [n, 4]."""
    f = [((x - p[0]) ** 2 + (y - p[1]) ** 2 + (z - p[2]) ** 2).sqrt() - p[3] for p in params]
    while len(f) > 1:
        f = [blend64(f[i], f[i + 1]) if i + 1 < len(f) else f[i] for i in range(0, len(f), 2)]
    return f[0]


def prepare(case, seed):
    kind = case["kind"]
    rng = random.Random(seed)
    if kind == "mesh":
        return {"case": case, "tape": lf.Tape(to_shape(model_of(case, rng))), "step": SIDE / case["cells"],
                "room": mesh_room(depth_of(case["cells"]))}
    if kind == "batch":
        jobs = []
        for i in range(case["count"]):
            # sizes spread over the whole range by place, the models by seed
            t = i / max(1, case["count"] - 1)
            n = int(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** t)
            u = (i * 0.6180339887) % 1.0
            cells = int(case["cells_lo"] * (case["cells_hi"] / case["cells_lo"]) ** u)
            model = part_model(n, rng) if i % 2 else csg_model(n, rng)
            jobs.append((lf.Tape(to_shape(model)), LOWER, UPPER, SIDE / cells))
        return {"case": case, "jobs": jobs, "room": mesh_room(10)}
    if kind == "slice":
        return {"case": case, "tape": lf.Tape(to_shape(csg_model(case["n"], rng))), "z": rng.uniform(-0.5, 0.5),
                "step": SIDE / case["cells"],
                "room": room(*[200 * 2 ** depth_of(case["cells"])] * 2, 2)}
    if kind == "heightmap":
        # the view moves over the model with the seed
        tape = kept(("heightmap", case["n"]), lambda: lf.Tape(to_shape(spheres_model(case["n"], random.Random(7)))))
        at = uniform3(rng, 0.2)
        return {"case": case, "tape": tape, "lower": [LOWER[a] + at[a] for a in range(3)],
                "upper": [UPPER[a] + at[a] for a in range(3)], "res": case["voxels"] / SIDE}
    if kind in ("values", "derivs"):
        tape = kept((kind, case["model"], case["n"]), lambda: lf.Tape(to_shape(model_of(case, random.Random(7)))))
        p = points_in(case["points"], seed)
        out = [torch.empty_like(p[0]) for _ in range(1 if kind == "values" else 4)]
        return {"case": case, "tape": tape, "points": p, "out": out}
    if kind == "grad":
        tape, order, _ = kept(("grad", case["n"]), lambda: variable_shape(case["n"]))
        params = sphere_parameters(case["n"], seed)
        p = points_in(case["points"], seed, 1.2)
        return {"case": case, "tape": tape, "points": p,
                "vars": torch.tensor([params[i] for i in order], dtype=torch.float32, device="cuda"),
                "f": torch.empty_like(p[0]), "g": [torch.empty_like(p[0]) for _ in range(3)],
                "gvars": torch.empty(len(order), device="cuda"), "loss": torch.empty(1, device="cuda")}
    # fit: the shapes are kept, their points and starting values come from the seed
    shapes = kept(("fit", case["shapes"], case["n"]), lambda: [variable_shape(case["n"]) for _ in range(case["shapes"])])
    start, points = [], []
    for k, (tape, order, variables) in enumerate(shapes):
        params = sphere_parameters(case["n"], seed * 100 + k)
        start.append(torch.tensor([params[i] for i in order], dtype=torch.float32, device="cuda"))
        points.append(points_in(case["points"], seed * 100 + k, 1.2))
    fit = BatchedFit([s[0] for s in shapes], points)
    return {"case": case, "fit": fit, "start": start, "out": [torch.empty_like(v) for v in start]}


def one_order(points, cells):
    """Points sorted by their coordinates and cells (rows of point numbers)
    as sorted rows of the points' places in that order; a triangle may start
    at any of its corners, a segment only at its first."""
    order = torch.arange(len(points), device=points.device)
    for a in reversed(range(points.shape[1])):
        order = order[torch.sort(points[order, a], stable=True).indices]
    points = points[order]
    new = torch.ones(len(points), dtype=torch.int64, device=points.device)
    new[1:] = (points[1:] != points[:-1]).any(1)
    rank = torch.empty_like(new)
    rank[order] = torch.cumsum(new, 0) - 1
    r = rank[cells]
    first, rest = r[:, 0], r[:, 1]
    if r.shape[1] == 3:
        rest = rest << 32 | r[:, 2]
        for i in (1, 2):   # the corner to start at: the least in order
            f, g = r[:, i], r[:, (i + 1) % 3] << 32 | r[:, (i + 2) % 3]
            less = (f < first) | ((f == first) & (g < rest))
            first, rest = torch.where(less, f, first), torch.where(less, g, rest)
    by = torch.sort(rest, stable=True).indices
    by = by[torch.sort(first[by], stable=True).indices]
    first, rest = first[by], rest[by]
    columns = [first, rest >> 32, rest & 0xffffffff] if r.shape[1] == 3 else [first, rest]
    return points, torch.stack(columns, 1).int()


def room(points, cells, dim):
    """Buffers of one size for whatever this call brings; the rest stays 0."""
    return [torch.zeros(points, dim, device="cuda"), torch.zeros(cells, dim, dtype=torch.int32, device="cuda")]


def depth_of(cells):
    return math.ceil(math.log2(cells))


def mesh_room(depth):
    t = min(40 * 4 ** depth, 24_000_000) + 4096
    return room(t // 2, t, 3)


def fill(buffers, parts):
    """The parts' points and cells, one after another, in the buffers."""
    for buffer, pieces in zip(buffers, zip(*parts)):
        at = 0
        for piece in pieces:
            buffer[at:at + len(piece)] = piece   # fails when there is no room
            at += len(piece)
    return buffers + [np.array([[len(p), len(c)] for p, c in parts])]


def mesh_on_gpu(verts, tris):
    return one_order(torch.from_numpy(verts).cuda(), torch.from_numpy(tris.view(np.int32)).cuda().long())


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "mesh":
        return fill(state["room"], [mesh_on_gpu(*state["tape"].render_mesh(LOWER, UPPER, state["step"]))])
    if kind == "batch":
        return fill(state["room"], [mesh_on_gpu(*m) for m in lf.render_meshes(state["jobs"])])
    if kind == "slice":
        cs = lf.render_slice(state["tape"], LOWER[:2], UPPER[:2], state["z"], state["step"])
        if not cs:
            return fill(state["room"], [(np.zeros((0, 2)), np.zeros((0, 2)))])
        ends = np.cumsum([len(c) for c in cs]) - 1
        a = np.delete(np.arange(ends[-1] + 1), ends)
        points, segments = one_order(torch.from_numpy(np.concatenate(cs)).cuda(),
                                     torch.from_numpy(np.stack([a, a + 1], 1)).cuda())
        # a closed contour repeats its first point, wherever that was
        return fill(state["room"], [(torch.unique_consecutive(points, dim=0), segments)])
    if kind == "heightmap":
        return lf.render_heightmap(state["tape"], state["lower"], state["upper"], state["res"])
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "values":
        return state["tape"].values(*state["points"], out=state["out"][0], stream=stream)
    if kind == "derivs":
        return state["tape"].derivs(*state["points"], *state["out"], stream=stream)
    if kind == "grad":
        from libfive_b200 import ffi
        tape, v = state["tape"], state["vars"]
        ffi.check(ffi.load().lfb_tape_set_vars_device(tape.ptr, v.data_ptr(), v.numel(), stream), "set variables")
        state["gvars"].zero_()
        tape.loss_grad(*state["points"], state["f"], *state["g"], gvars=state["gvars"], loss=state["loss"],
                       stream=stream)
        return {"f": state["f"], "g": state["g"], "gvars": state["gvars"], "loss": state["loss"]}
    # fit: one step from the starting values and cleared moments
    from libfive_b200 import ffi
    fit = state["fit"]
    for tape, v in zip(fit.tapes, state["start"]):
        ffi.check(ffi.load().lfb_tape_set_vars_device(tape.ptr, v.data_ptr(), v.numel(), stream), "set variables")
    fit.t = 0
    fit.m.zero_()
    fit.v.zero_()
    losses = fit.step()
    return {"losses": losses, "m": fit.m, "v": fit.v}


# Clauses of a primitive with its operator, and the triangles of a mesh per
# square of its cells along an edge of the region, as these models have them.
CLAUSES = 11
TRIANGLES = {"spheres": 10.0, "part": 9.0, "csg": 9.0}


def mesh_work(model, n, cells):
    """Outputs written once; each crossed edge's search (four rounds of 14
    samples, two gradients) and each cell's corner through one primitive."""
    cells = 2.0 ** depth_of(cells)
    t = TRIANGLES[model] * cells ** 2
    return {"bytes": t * 12 + t / 2 * 12 + n * CLAUSES * 8, "flops": (t / 2 * (4 * 14 + 2 * 4) + t / 2) * CLAUSES}


def work(case):
    kind = case["kind"]
    if kind == "mesh":
        return mesh_work(case["model"], case["n"], case["cells"])
    if kind == "batch":
        n, c = (case["n_lo"] * case["n_hi"]) ** 0.5, (case["cells_lo"] * case["cells_hi"]) ** 0.5
        w = mesh_work("part", n, c)
        return {k: v * case["count"] for k, v in w.items()}
    if kind == "slice":
        segments = 20.0 * 2.0 ** depth_of(case["cells"])
        return {"bytes": segments * 8 + case["n"] * CLAUSES * 8,
                "flops": segments * (4 * 16 + 2 * 4) * CLAUSES + case["n"] * CLAUSES * 2}
    if kind == "heightmap":
        pixels = case["voxels"] ** 2
        return {"bytes": pixels * 8, "flops": pixels * 6 * CLAUSES}
    p = case["points"]
    if kind == "values":
        return {"bytes": 16 * p, "flops": p * case["n"] * CLAUSES}
    if kind == "derivs":
        return {"bytes": 28 * p, "flops": 4 * p * case["n"] * CLAUSES}
    if kind == "grad":
        return {"bytes": 28 * p, "flops": 4 * p * case["n"] * (CLAUSES + 5)}
    return {"bytes": case["shapes"] * (12 * p + case["n"] * 4 * 16),
            "flops": 4 * case["shapes"] * p * case["n"] * (CLAUSES + 5)}


def loss_gradient64(params, points):
    """mean f^2 of the blended spheres with its gradients, in 64 bits."""
    n = len(points[0])
    leaf = torch.tensor(params, dtype=torch.float32, device="cuda").double().reshape(-1, 4).requires_grad_()
    f_all, g_all, loss = [], [], 0.0
    for at in range(0, n, 50000):
        p = [q[at:at + 50000].double().requires_grad_() for q in points]
        f = values64(list(leaf), *p)
        part = (f * f).sum() / n
        part.backward()
        loss += part.detach()
        f_all.append(f.detach())
        g_all.append([q.grad for q in p])
    return torch.cat(f_all), [torch.cat([g[a] for g in g_all]) for a in range(3)], leaf.grad.reshape(-1), loss


def exact(case, seed):
    kind = case["kind"]
    if kind in ("values", "derivs"):
        node = model_of(case, random.Random(7))
        points = points_in(case["points"], seed)
        outs = []
        for at in range(0, case["points"], 20000):
            p = [q[at:at + 20000].double().requires_grad_(kind == "derivs") for q in points]
            f = to_double(node, *p)
            if kind == "derivs":
                f.sum().backward()
            outs.append([f.detach()] + ([q.grad for q in p] if kind == "derivs" else []))
        outs = [torch.cat([o[k] for o in outs]) for k in range(len(outs[0]))]
        return outs[0] if kind == "values" else tuple(outs)
    if kind == "grad":
        _, order, _ = kept(("grad", case["n"]), lambda: variable_shape(case["n"]))
        f, g, gp, loss = loss_gradient64(sphere_parameters(case["n"], seed), points_in(case["points"], seed, 1.2))
        return {"f": f, "g": g, "gvars": gp[torch.tensor(order, device="cuda")], "loss": loss.reshape(1)}
    if kind == "fit":
        shapes = kept(("fit", case["shapes"], case["n"]), lambda: [variable_shape(case["n"]) for _ in range(case["shapes"])])
        losses, m = [], []
        for k, (_, order, _) in enumerate(shapes):
            _, _, gp, loss = loss_gradient64(sphere_parameters(case["n"], seed * 100 + k),
                                             points_in(case["points"], seed * 100 + k, 1.2))
            losses.append(loss)
            m.append(gp[torch.tensor(order, device="cuda")])
        m = torch.cat(m)
        return {"losses": torch.stack(losses), "m": (1 - 0.9) * m, "v": (1 - 0.999) * m * m}
    return None   # meshes, contours and images: no plain 64-bit form
