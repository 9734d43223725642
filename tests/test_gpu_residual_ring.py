"""Residuals every k-th step over calls that are longer than the ring of residual
slots (8192): those not read yet must not be cleared or written over by later
steps of the call, whichever engine steps."""
import numpy as np
import pytest

from mantiis_gb300 import SIM_ADSORPTION, Solver, default_params, generate_disks, pore_properties

pytestmark = pytest.mark.gpu

N = 24


def history(engine, steps, call, **kw):
    pore = generate_disks(N, 2, 4, 0.65, 6, open_x_edges=True)
    lp, ku = pore_properties(pore, 1.0, 1.0)
    kn = np.where(pore == 1, 0.1 * ku / ku[pore == 1].mean(), 0.0)
    with Solver(pore, kn, lp, default_params(dx=1e-9, tol=0.0, **kw)) as s:
        s.set_engine(engine)
        for _ in range(steps // call):
            s.advance(call)
        return s.cells(with_f=True)["f"], s.residuals()


@pytest.mark.parametrize("every", [3, 4, 100])
@pytest.mark.parametrize("engine", [0, 1])
def test_transport(engine, every):
    steps = 20000
    f0, r0 = history(0, steps, 2000, check_every=every)
    f1, r1 = history(engine, steps, steps, check_every=every)
    # the residual of step j is known after step j + 1
    assert len(r0) == len(r1) == (steps - 1) // every
    assert np.isfinite(r0).all() and np.isfinite(r1).all()
    # FP64 sums of up to N^2 non-negative terms in another order
    assert np.allclose(r0, r1, rtol=N * N * 2.0 ** -52, atol=0.0)
    assert np.array_equal(f0, f1)


def test_adsorption():
    steps, every = 20000, 4
    kw = dict(simulation=SIM_ADSORPTION, psi_form=1, g_ff=-0.25, g_fs=-1.5, rho_psi=0.5, rho_init=0.5, fbody=0.0,
              check_every=every)
    f0, r0 = history(1, steps, 2000, **kw)
    f1, r1 = history(1, steps, steps, **kw)
    assert len(r0) == len(r1) == steps // every
    assert np.array_equal(r0, r1) and np.array_equal(f0, f1)  # maxima: no order of summation
