"""Calls that change between cooperative launches and launches per phase: short calls
of images beyond the L2, few steps of a batch of few images.  States are the bits of
the launch engine's whichever way each call goes, and each goes the way it should."""
import numpy as np
import pytest

from mantiis_gb300 import Batch, Solver, default_params, generate_disks

pytestmark = pytest.mark.gpu


def solver(n, levels=1, seed=5, **kw):
    pore = generate_disks(n, max(3, n // 40), max(8, n // 14), 0.65, seed, open_x_edges=True)
    p = default_params(dx=1e-9, tol=0.0, multiblock=int(levels > 1), max_allowed_level=max(2, levels),
                       edge_fine=int(levels > 1), **kw)
    return Solver(pore, np.where(pore == 1, 0.05, 0.0), np.where(pore == 1, 7.73, 0.0), p)


def populations(s):
    return s.cells(with_f=True)["f"]


def test_short_calls_of_a_large_image():
    n = 2000  # populations of 144 MB, more than the L2
    a, b = solver(n), solver(n, plain_path=2)
    b.set_engine(0)
    for call, steps, launches in [("advance_graph", 1, None), ("advance_graph", 2, None), ("advance_graph", 3, 1),
                                  ("advance", 2, None), ("advance", 3, 1), ("run", 2, None), ("run", 3, 2),
                                  ("advance_graph", 1, None), ("advance_graph", 2, None), ("advance", 5, 1)]:
        l0 = a.launches
        for s in (a, b):
            getattr(s, call)(steps)
        assert a.launches - l0 == launches if launches else a.launches - l0 > steps, (call, steps)
    assert a.time == b.time
    ra, rb = a.residuals(), b.residuals()
    # FP64 sums of up to n^2 non-negative terms in another order
    assert len(ra) == len(rb) and np.allclose(ra, rb, rtol=n * n * 2.0 ** -52, atol=0.0)
    assert np.array_equal(populations(a), populations(b))
    a.close()
    b.close()


def test_single_steps_of_run():
    for n, coop in ((100, True), (1100, False)):  # populations of 0.4 / 44 MB, a quarter of the L2 is 34
        a, b = solver(n), solver(n, plain_path=2)
        b.set_engine(0)
        l0 = a.launches
        for steps in (1, 1, 4, 1):
            assert a.run(steps) == b.run(steps) == steps
        # a cooperative launch and the read pass for each call, or launches per phase
        assert (a.launches - l0 == 2 * 4) == coop
        assert np.array_equal(populations(a), populations(b))


@pytest.mark.parametrize("shapes", [[(128, 1), (64, 2)], [(128, 1), (64, 1)], [(64, 1)] * 13, [(256, 2), (100, 1), (128, 2)]])
def test_few_steps_of_a_batch(shapes):
    solo = [solver(n, l, 20 + i) for i, (n, l) in enumerate(shapes)]
    grouped = [solver(n, l, 20 + i) for i, (n, l) in enumerate(shapes)]
    for s in solo:
        s.set_engine(0)
    b = Batch(grouped)
    levels = sum(s.info["max_level"] for s in grouped)
    many = 8 if levels > len(shapes) else 4
    for steps in (1, 2, 3, 4, 8, 1, 6, 7, 2):
        l0 = b.launches
        b.advance(steps)
        b.sync()
        assert (b.launches - l0 == 1) == (levels > 12 or steps % 2 == 1 or steps >= many), steps
        for s in solo:
            s.advance_graph(steps)
    for s, g in zip(solo, grouped):
        assert s.time == g.time and np.array_equal(populations(s), populations(g))
    b.close()


def test_groups_do_not_depend_on_staging():
    # buffers that downloads and uploads leave behind are no part of what a step touches
    shapes = [(1100, 1)] * 4  # two of 44 MB to a group
    out = []
    for staged in (False, True):
        ss = [solver(n, l, i, plain_path=2) for i, (n, l) in enumerate(shapes)]
        if staged:
            for s in ss:
                c = s.cells(with_f=True)
                s.set_equilibrium(c["rho"], c["ux"], c["uy"])
        b = Batch(ss)
        b.advance(9)
        b.sync()
        out.append(b.launches)
        b.close()
    assert out == [2, 2]
