"""Cooperative steps recorded by a caller's stream capture and replayed more than
once: only what every replay runs from the recorded parity is recorded; the rest is
refused, and the capture goes on."""
import numpy as np
import pytest

from mantiis_gb300 import MantiisError, Solver, default_params, generate_disks

pytestmark = pytest.mark.gpu


def solver(levels):
    pore = generate_disks(128, 4, 10, 0.65, 3, open_x_edges=True)
    p = default_params(multiblock=int(levels > 1), max_allowed_level=2, edge_fine=int(levels > 1))
    return Solver(pore, np.where(pore == 1, 0.05, 0.0), np.where(pore == 1, 7.73, 0.0), p)


def populations(s):
    return s.cells(with_f=True)["f"]


def recorded(s, before, steps):
    """The graph of a captured call, and the error that the call raised."""
    import torch

    stream, graph, error = torch.cuda.Stream(), torch.cuda.CUDAGraph(), None
    s.set_stream(stream.cuda_stream)
    for n in before:
        s.advance_graph(n)
    s.sync()
    with torch.cuda.graph(graph, stream=stream):
        torch.zeros(1, device="cuda")
        try:
            s.advance_graph(steps)
        except MantiisError as e:
            error = e
    torch.cuda.synchronize()
    return graph, error


@pytest.mark.parametrize("levels", [1, 2])
@pytest.mark.parametrize("before,steps,replays", [((2,), 4, 3), ((2, 1), 2, 3), ((4, 1), 1, 1)])
def test_replays(levels, before, steps, replays):
    import torch

    direct, s = solver(levels), solver(levels)
    for n in before:
        direct.advance_graph(n)
    graph, error = recorded(s, before, steps)
    assert error is None
    for _ in range(replays):
        graph.replay()
        torch.cuda.synchronize()
        direct.advance_graph(steps)
        assert np.array_equal(populations(s), populations(direct))


@pytest.mark.parametrize("levels", [1, 2])
@pytest.mark.parametrize("before,steps", [((4, 2), 3), ((0,), 4), ((0,), 3)])
def test_refused(levels, before, steps):
    direct, s = solver(levels), solver(levels)
    _, error = recorded(s, before, steps)
    assert error is not None and "capture" in str(error)
    # nothing of the refused call has run or been counted
    for n in (*before, steps):
        direct.advance_graph(n)
    s.advance_graph(steps)
    assert s.time == direct.time and np.array_equal(populations(s), populations(direct))
