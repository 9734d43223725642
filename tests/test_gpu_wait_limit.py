"""A grid barrier whose wait runs out (a limit of one poll: most blocks give up at once)
is reported by every image that the launch steps, once, and the contexts stay usable."""
import numpy as np
import pytest

from mantiis_gb300 import SIM_ADSORPTION, Batch, MantiisError, Solver, default_params, generate_disks, lib

pytestmark = pytest.mark.gpu

E_DEVICE = -4


def solver(n=128, seed=3, **kw):
    pore = generate_disks(n, 4, 10, 0.65, seed, open_x_edges=True)
    return Solver(pore, np.where(pore == 1, 0.05, 0.0), np.where(pore == 1, 7.73, 0.0), default_params(tol=0.0, **kw))


def limit(s, polls):
    assert lib().mgpu_set_wait_limit(s._h, polls) == 0


def gives_up(call):
    with pytest.raises(MantiisError) as e:
        call()
    assert e.value.code == E_DEVICE and "wait" in str(e.value)


def restart(s):
    rho = np.full(s.n_cells, s.info["rho_in"])
    s.set_equilibrium(rho, np.full(s.n_cells, 1e-6), np.zeros(s.n_cells))


@pytest.mark.parametrize("sim", [0, SIM_ADSORPTION])
def test_one_context(sim):
    s, fresh = solver(simulation=sim), solver(simulation=sim)
    limit(s, 1)
    gives_up(lambda: s.run(20))
    s.sync()  # reported once
    s.advance_graph(20)
    gives_up(s.sync)
    if sim:  # the density of the previous step is state too: not compared
        return
    limit(s, 0)
    restart(s)
    restart(fresh)
    s.advance_graph(20)
    fresh.advance_graph(20)
    s.sync()
    assert np.array_equal(s.cells(with_f=True)["f"], fresh.cells(with_f=True)["f"])


def test_every_image_of_a_group():
    images = [solver(n, 3 + i) for i, n in enumerate((128, 64, 100))]
    b = Batch(images)
    limit(images[0], 1)
    b.advance(20)
    for s in images:
        gives_up(s.sync)
    b.sync()
    b.advance(20)
    gives_up(b.sync)
    b.sync()  # every image's word was cleared
    b.close()
