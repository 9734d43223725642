"""Cooperative steps recorded by a caller's stream capture: after one call that
made the plan, a captured call replays to the bits of the same steps made
directly; a context whose first call falls into a capture takes the launch
engine's route, which refuses to prepare its launches there."""
import numpy as np
import pytest

from mantiis_gb300 import MantiisError, Solver, default_params, generate_disks

pytestmark = pytest.mark.gpu


def solver(levels):
    n = 128
    pore = generate_disks(n, 4, 10, 0.65, 3, open_x_edges=True)
    p = default_params(multiblock=int(levels > 1), max_allowed_level=2, edge_fine=int(levels > 1))
    return Solver(pore, np.where(pore == 1, 0.05, 0.0), np.where(pore == 1, 7.73, 0.0), p)


@pytest.mark.parametrize("levels", [1, 2])
def test_captured_steps_replay(levels):
    import torch

    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    direct, s = solver(levels), solver(levels)
    direct.advance_graph(2)
    direct.advance_graph(4)
    s.set_stream(stream.cuda_stream)
    s.advance_graph(2)
    s.sync()
    with torch.cuda.graph(graph, stream=stream):
        s.advance_graph(4)
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(s.cells(with_f=True)["f"], direct.cells(with_f=True)["f"])


def test_first_call_in_a_capture_is_refused():
    import torch

    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    s = solver(1)
    s.set_stream(stream.cuda_stream)
    s.sync()
    with torch.cuda.graph(graph, stream=stream):
        with pytest.raises(MantiisError):
            s.advance_graph(4)
        torch.zeros(1, device="cuda")  # the capture itself goes on
    torch.cuda.synchronize()
    direct = solver(1)
    direct.advance_graph(4)
    s.advance_graph(4)
    assert np.array_equal(s.cells(with_f=True)["f"], direct.cells(with_f=True)["f"])
