"""Free variables set while a CUDA graph is being captured on a stream: a
host call that takes no part in the capture."""
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
