"""Cooperative launches against launches per phase over calls longer than one launch
(500 steps), runs that stop on their tolerance within, at the end of and after a batch
of steps and go on, and batches whose images are groups of their own."""
import numpy as np
import pytest

from mantiis_gb300 import Batch, Solver, default_params, generate_disks

pytestmark = pytest.mark.gpu


def solver(n, levels=1, seed=5, **kw):
    pore = generate_disks(n, max(2, n // 40), max(4, n // 14), 0.65, seed, open_x_edges=True)
    p = default_params(dx=1e-9, multiblock=int(levels > 1), max_allowed_level=max(2, levels), edge_fine=int(levels > 1), **kw)
    return Solver(pore, np.where(pore == 1, 0.05, 0.0), np.where(pore == 1, 7.73, 0.0), p)


def close(a, b, n):
    # FP64 sums of up to n^2 non-negative terms in another order
    return len(a) == len(b) and np.allclose(a, b, rtol=n * n * 2.0 ** -52, atol=0.0)


@pytest.mark.parametrize("n,levels", [(64, 1), (128, 2)])
def test_long_calls(n, levels):
    out = []
    for engine in (0, 1):
        s = solver(n, levels, tol=0.0)
        s.set_engine(engine)
        assert s.run(1101) == 1101
        s.advance(777)
        s.advance_graph(1003)
        assert s.run(3) == 3
        out.append((s.cells(with_f=True)["f"], s.residuals(), s.time))
    assert out[0][2] == out[1][2] and close(out[0][1], out[1][1], n) and np.array_equal(out[0][0], out[1][0])


def test_stops_on_tolerance():
    n = 64
    ref = solver(n, tol=0.0)
    ref.set_engine(0)
    ref.run(1200)
    r = ref.residuals()
    lowest = np.minimum.accumulate(r)
    for target in (7, 999, 1000, 1001, 1150):  # batches of run are 1000 steps
        # the first step from there on whose residual is the lowest so far: a tolerance picks it
        stop = next(k for k in range(target, 1200) if r[k - 1] < lowest[k - 2])
        tol = float(np.sqrt(r[stop - 1] * lowest[stop - 2]))
        out = []
        for engine in (0, 1):
            s = solver(n, tol=tol)
            s.set_engine(engine)
            assert s.run(1200) == stop
            s.advance_graph(5)
            s.advance(4)
            out.append((s.cells(with_f=True)["f"], s.residuals(), s.time))
            s.close()
        assert out[0][2] == out[1][2] and close(out[0][1], out[1][1], n) and np.array_equal(out[0][0], out[1][0])


def test_groups_of_one_image():
    solo, own = ([solver(1300, 1, seed) for seed in (3, 4)] for _ in range(2))  # populations of 61 MB each
    b = Batch(own)
    b.advance(9)
    b.advance(5)
    b.sync()
    assert b.launches == 4
    for s, g in zip(solo, own):
        s.set_engine(0)
        s.advance_graph(14)
        assert s.time == g.time and np.array_equal(s.cells(with_f=True)["f"], g.cells(with_f=True)["f"])
