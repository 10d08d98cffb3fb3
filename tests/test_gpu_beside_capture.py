"""Calls while a CUDA graph is being captured on another stream, in which they
take no part: free variables set, derivatives on a stream of their own."""
import numpy as np
import pytest
import torch

from libfive_b200 import workloads
from libfive_b200.shape import Tape

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
def test_set_vars_in_an_open_capture(gpu, mode):
    shape, vals, _ = workloads.fit_csg_vars(12, seed=3)
    tape = Tape(shape, vals)
    p = [torch.from_numpy(a).cuda() for a in workloads.uniform_points(1000, seed=1)]
    out = torch.empty_like(p[0])
    tape.values(*p, out=out, stream=torch.cuda.current_stream().cuda_stream)
    moved = workloads.perturbed(vals, 0.05, seed=4)
    want = Tape(shape, moved).values(*[a.cpu().numpy() for a in p])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode=mode):
        tape.values(*p, out=out, stream=torch.cuda.current_stream().cuda_stream)
        tape.set_vars(moved)
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), want, equal_nan=True)


# A long tape's derivatives on a stream of its own: the pruned path allocates.
@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
def test_long_derivatives_beside_an_open_capture(gpu, mode):
    tape, short = Tape(workloads.random_csg(420, seed=5)), Tape(workloads.spheres_union(8, seed=1))
    assert tape.n_clauses > 4096
    p = [torch.from_numpy(a).cuda() for a in workloads.uniform_points(4000, seed=1)]
    out = [torch.empty_like(p[0]) for _ in range(5)]
    short.values(*p, out=out[4], stream=torch.cuda.current_stream().cuda_stream)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode=mode):
        short.values(*p, out=out[4], stream=torch.cuda.current_stream().cuda_stream)
        for _ in range(2):
            tape.derivs(*p, *out[:4], stream=side.cuda_stream)
    torch.cuda.synchronize()
    want = tape.derivs(*[a.cpu().numpy() for a in p])
    for a, b in zip(out, want):
        assert np.array_equal(a.cpu().numpy(), b, equal_nan=True)
