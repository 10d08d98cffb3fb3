"""A fit step captured in a CUDA graph, and steps of other fits while the
capture is open."""
import numpy as np
import pytest
import torch

from libfive_b200 import workloads
from libfive_b200.fit import BatchedFit
from libfive_b200.shape import Tape

pytestmark = pytest.mark.gpu


def make(seed, n=2000):
    shapes = [workloads.fit_csg_vars(6 + j, seed=seed + j)[:2] for j in range(3)]
    points = [tuple(torch.from_numpy(a).cuda() for a in workloads.uniform_points(n, seed=seed + j)) for j in range(3)]
    return BatchedFit([Tape(s, v) for s, v in shapes], points, lr=1e-2)


def test_step_while_another_is_captured(gpu):
    a, b, twin = make(10), make(20), make(20)
    a.step()      # kernels compiled, scratch there
    b.step()
    want = [twin.step().cpu().numpy().copy() for _ in range(2)]
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="relaxed"):
        captured = a.step(stream=torch.cuda.current_stream().cuda_stream)
        with torch.cuda.stream(side):
            second = b.step(stream=side.cuda_stream)
    torch.cuda.synchronize()
    # the variables after one step differ in the last bits between the two
    # (the gradient is a sum in an order that atomics choose): 2^-24 of
    # partial sums of 2,000 points, on losses near one
    np.testing.assert_allclose(second.cpu().numpy(), want[1], rtol=2000 * 2.0 ** -24, atol=0)
    # the captured step runs at each replay: the losses of the variables as
    # the steps before left them
    graph.replay()
    torch.cuda.synchronize()
    one = captured.cpu().numpy().copy()
    assert np.isfinite(one).all()
    graph.replay()
    torch.cuda.synchronize()
    assert not np.array_equal(captured.cpu().numpy(), one)


def test_captured_step(gpu):
    """After one step outside nothing is allocated or compiled in a capture."""
    a, twin = make(30), make(30)
    a.step()
    want = [twin.step().cpu().numpy().copy() for _ in range(2)]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = a.step(stream=torch.cuda.current_stream().cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    np.testing.assert_allclose(captured.cpu().numpy(), want[1], rtol=2000 * 2.0 ** -24, atol=0)
