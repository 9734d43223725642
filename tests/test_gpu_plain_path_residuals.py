"""The residual of a step is the same sum whichever plain-cell kernel steps, also where
the pipelined one (plain_path 1) takes several tiles to a block."""
import numpy as np
import pytest

from mantiis_gb300 import Solver, default_params, generate_disks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,levels", [(200, 1), (900, 1), (1024, 2)])
def test_residuals(n, levels):
    pore = generate_disks(n, max(3, n // 100), max(8, n // 25), 0.65, 5, open_x_edges=True)
    kn, lp = np.where(pore == 1, 0.05, 0.0), np.where(pore == 1, 7.73, 0.0)
    out = []
    for path in (0, 1, 2):
        p = default_params(dx=1e-9, tol=0.0, plain_path=path, multiblock=int(levels > 1), max_allowed_level=2,
                           edge_fine=int(levels > 1))
        with Solver(pore, kn, lp, p) as s:
            s.run(5)
            s.advance(4)
            out.append((s.residuals(), s.cells(with_f=True)["f"]))
    for r, f in out[1:]:
        # FP64 sums of up to n^2 non-negative terms in another order
        assert len(r) == len(out[0][0]) and np.allclose(r, out[0][0], rtol=n * n * 2.0 ** -52, atol=0.0)
        assert np.array_equal(f, out[0][1])
