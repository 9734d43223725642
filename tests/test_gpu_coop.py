"""Transport steps in cooperative launches (the default) against the launches per
phase, bit for bit, where the split of the cells can go wrong: fewer warps of
cells than SMs, odd sides, void and solid x seams (cells whose neighbours wrap),
one to three levels (interface rows with special sources among them), every
collision and wall model, single steps, calls that begin at either parity, and
batches of more levels than one launch takes."""
import numpy as np
import pytest

from mantiis_gb300 import Batch, Solver, default_params, generate_disks, pore_properties

pytestmark = pytest.mark.gpu


def image(n, seed, porosity=0.65, open_edges=True):
    pore = generate_disks(n, max(2, n // 40), max(3, n // 14), porosity, seed, open_x_edges=open_edges)
    lp, ku = pore_properties(pore, 1.0, 1.0)
    return pore, np.where(pore == 1, 0.1 * ku / ku[pore == 1].mean(), 0.0), lp


def start(s, seed=1):
    r = np.random.default_rng(seed)
    rho = s.info["rho_in"] * (1.0 + 1e-6 * r.uniform(-1, 1, s.n_cells))
    s.set_equilibrium(rho, 1e-6 * r.uniform(0, 1, s.n_cells), 1e-6 * r.uniform(-1, 1, s.n_cells))


CASES = [
    # n, levels, collision, wall, open x edges
    (24, 1, 2, 2, True),
    (33, 1, 0, 1, False),
    (131, 1, 1, 2, True),
    (300, 1, 1, 0, False),
    (301, 1, 2, 1, True),
    (64, 2, 2, 2, True),
    (128, 2, 0, 2, False),
    (256, 3, 2, 2, False),
    (256, 3, 2, 1, True),
    (256, 2, 1, 0, True),
]


@pytest.mark.parametrize("n,levels,collision,wall,open_edges", CASES)
def test_engines_agree(n, levels, collision, wall, open_edges):
    img = image(n, 5, open_edges=open_edges)
    p = default_params(dx=1e-9, collision=collision, wall=wall, multiblock=int(levels > 1),
                       max_allowed_level=max(2, levels), edge_fine=int(levels > 1), tol=0.0)
    out = []
    for engine in (0, 1):
        s = Solver(*img, p)
        s.set_engine(engine)
        start(s)
        l0 = s.launches
        for steps in (1, 2, 1):
            assert s.run(steps) == steps
        s.advance(3)
        s.advance_graph(3)
        s.advance_graph(1)
        assert s.run(5) == 5
        launches = s.launches - l0
        c = s.cells(with_f=True)
        out.append((c["f"], s.residuals(), launches))
        s.close()
    assert np.isfinite(out[0][0]).all() and np.array_equal(out[0][0], out[1][0])
    # FP64 sums of up to n^2 terms in another order
    assert len(out[0][1]) == len(out[1][1])
    assert np.allclose(out[0][1], out[1][1], rtol=n * n * 2.0 ** -52, atol=0.0)
    assert out[1][2] < out[0][2]  # the cooperative launches did run


def test_residuals_every_third_step():
    img = image(100, 6)
    p = default_params(dx=1e-9, check_every=3, tol=0.0)
    out = []
    for engine in (0, 1):
        s = Solver(*img, p)
        s.set_engine(engine)
        start(s)
        for steps in (4, 1, 9, 2):
            s.advance(steps)
        out.append((s.cells(with_f=True)["f"], s.residuals()))
        s.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert len(out[0][1]) == len(out[1][1]) > 3
    assert np.allclose(out[0][1], out[1][1], rtol=100 * 100 * 2.0 ** -52, atol=0.0)


def test_batch_of_several_groups():
    # 45 levels: more than one launch's 40
    shapes = [(64, 2), (40, 1), (128, 2), (33, 1)] * 7 + [(256, 3)]
    imgs = [image(n, 20 + i) for i, (n, _) in enumerate(shapes)]
    prm = [default_params(dx=1e-9, multiblock=int(l > 1), max_allowed_level=max(2, l), edge_fine=int(l > 1))
           for _, l in shapes]
    solo = [Solver(*a, p) for a, p in zip(imgs, prm)]
    grouped = [Solver(*a, p) for a, p in zip(imgs, prm)]
    for i, (s, g) in enumerate(zip(solo, grouped)):
        s.set_engine(0)
        start(s, i)
        start(g, i)
        s.advance_graph(12)
    b = Batch(grouped)
    for steps in (1, 4, 7):
        b.advance(steps)
    b.sync()
    assert 0 < b.launches <= 3 * 2
    for s, g in zip(solo, grouped):
        assert s.time == g.time
        assert np.array_equal(s.cells(with_f=True)["f"], g.cells(with_f=True)["f"])
    b.close()
