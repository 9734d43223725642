"""The pore-property pipeline where its tiles can go wrong: images around a tile's
44 rows and 512 columns (of the padded width 3n), skeleton branches and wide
void regions whose fronts cross many tiles and launches, against the host code
bit for bit."""
import numpy as np
import pytest

from mantiis_gb300 import generate_disks, pore_properties, pore_properties_gpu

pytestmark = pytest.mark.gpu


def check(pore):
    lp_h, kn_h = pore_properties(pore, 2e-9, 6e-9)
    lp_g, kn_g, iters = pore_properties_gpu(pore, 2e-9, 6e-9, return_iterations=True)
    assert np.array_equal(lp_g, lp_h) and np.array_equal(kn_g, kn_h)
    return iters


@pytest.mark.parametrize("n", [4, 5, 32, 33, 43, 44, 45, 64, 87, 88, 89, 132, 170, 171, 257])
def test_sides_around_tiles(n):
    if n < 24:
        pore = (np.random.default_rng(n).random((n, n)) < 0.7).astype(np.int32)
    else:
        pore = generate_disks(n, 2, max(3, n // 10), 0.65, n, open_x_edges=True)
    assert check(pore) >= 1


@pytest.mark.parametrize("n", [200, 345])
def test_wide_voids(n):
    # one void with a few solid specks: fronts of n / 2 iterations
    pore = np.ones((n, n), np.int32)
    pore[0] = pore[-1] = 0
    pore[n // 3, n // 4:n // 4 + 3] = 0
    pore[2 * n // 3, n // 2] = 0
    assert check(pore) > n // 4
    # a comb of thin channels: many skeleton branches
    comb = np.zeros((n, n), np.int32)
    comb[n // 2 - 4:n // 2 + 4] = 1
    comb[5:-5, ::7] = 1
    check(comb)
