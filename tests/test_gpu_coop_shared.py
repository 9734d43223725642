"""Default contexts that step at the same time: those that would take turns at the whole
GPU for nothing take launches per phase while another's steps are in flight, and
cooperative launches again when they are alone.  States are the same bits."""
import threading

import numpy as np
import pytest

from mantiis_gb300 import Batch, Solver, default_params, generate_disks

pytestmark = pytest.mark.gpu


def solver(n, levels=1, seed=5, **kw):
    pore = generate_disks(n, max(3, n // 100), max(8, n // 20), 0.62, seed, open_x_edges=True)
    p = default_params(dx=1e-9, tol=0.0, multiblock=int(levels > 1), max_allowed_level=max(2, levels),
                       edge_fine=int(levels > 1), **kw)
    return Solver(pore, np.where(pore == 1, 0.05, 0.0), np.where(pore == 1, 7.73, 0.0), p)


def populations(s):
    return s.cells(with_f=True)["f"]


def launches_of(s, steps):
    l0 = s.launches
    s.advance_graph(steps)
    return s.launches - l0


def test_route_follows_other_contexts():
    # some 10 ms of steps in flight, against the microseconds of the calls after them
    large, mid, small = solver(1024), solver(320), solver(100)
    b = Batch([solver(256, 2), solver(256, 2, 6)])
    for s in (large, mid, small):
        s.advance_graph(4)
        s.sync()
    b.advance(9)
    b.sync()
    assert launches_of(mid, 100) == 1  # alone
    mid.sync()
    large.advance_graph(1000)
    assert launches_of(mid, 100) > 1 and launches_of(small, 100) == 1
    l0 = b.launches
    b.advance(40)  # many images' launches would be slower than turns of 32 steps
    assert b.launches - l0 == 2
    for s in (large, mid, small, b):
        s.sync()
    assert launches_of(mid, 100) == 1
    mid.sync()
    # steps of the batch are others' to a context outside of it
    b.advance(1001)
    assert launches_of(mid, 50) > 1
    mid.sync()
    b.sync()
    ref = solver(320)
    ref.set_engine(0)
    ref.advance_graph(354)
    assert np.array_equal(populations(mid), populations(ref))


@pytest.mark.parametrize("n,levels", [(128, 1), (320, 1), (256, 2)])
def test_threads(n, levels):
    ref = [solver(n, levels, 5 + i) for i in range(3)]
    par = [solver(n, levels, 5 + i) for i in range(3)]

    def step(s):
        for _ in range(5):
            s.run(40)
            s.advance_graph(21)
            s.advance(7)
        s.sync()

    for s in ref:
        s.set_engine(0)
        step(s)
    threads = [threading.Thread(target=step, args=(s,)) for s in par]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s, r in zip(par, ref):
        assert s.time == r.time
        a, b = s.residuals(), r.residuals()
        # FP64 sums of up to n^2 non-negative terms in another order
        assert len(a) == len(b) and np.allclose(a, b, rtol=n * n * 2.0 ** -52, atol=0.0)
        assert np.array_equal(populations(s), populations(r))


def test_contexts_come_and_go_on_threads():
    def live(seed):
        for k in range(6):
            with solver(100, 1, seed + k) as s:
                s.advance_graph(30)
                s.run(10)

    threads = [threading.Thread(target=live, args=(10 * i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    with solver(320) as s:
        s.advance_graph(4)
        s.sync()
        assert launches_of(s, 20) == 1
