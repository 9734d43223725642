"""The adsorption engine that keeps each block's cells for many steps against the
launches per pass, bit for bit, where its split of the cells can go wrong: fewer
warps of cells than SMs, shares that are not whole warps, a void x seam (cells
whose neighbours wrap), more cells than the blocks' shared memory holds, single
steps and calls that begin at either parity."""
import numpy as np
import pytest

from mantiis_gb300 import SIM_ADSORPTION, Solver, default_params, generate_disks, pore_properties

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,porosity,psi_form", [(24, 0.8, 1), (40, 0.7, 0), (131, 0.6, 1), (333, 0.65, 0),
                                                 (1024, 0.92, 1)])
def test_engines_agree(n, porosity, psi_form):
    pore = generate_disks(n, max(2, n // 40), max(3, n // 16), porosity, 11, open_x_edges=True)
    lp, ku = pore_properties(pore, 1.0, 1.0)
    kw = dict(psi_form=1, rho_psi=0.5, g_ff=-0.25, g_fs=-1.5, rho_init=0.5, fbody=0.0) if psi_form else {}
    p = default_params(dx=1e-9, simulation=SIM_ADSORPTION, tol=0.0, **kw)
    kn = np.where(pore == 1, 0.1 * ku / ku[pore == 1].mean(), 0.0)
    out = []
    for engine in (0, 1):
        s = Solver(pore, kn, lp, p)
        s.set_engine(engine)
        rho0 = s.params.rho_init or s.info["rho_in"]
        rho = rho0 * (1.0 + 1e-3 * np.random.default_rng(5).uniform(-1, 1, s.n_cells))
        s.set_equilibrium(rho, np.zeros_like(rho), np.zeros_like(rho))
        for steps in (1, 2, 1, 5, 16):
            assert s.run(steps) == steps
        c = s.cells(with_f=True)
        out.append([c["f"], c["rho"], c["ux"], c["uy"], s.residuals()])
        s.close()
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)
