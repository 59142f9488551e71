"""Binning: lattices past the size where a scan block adds up the tiles before its own
(2.1M cells), and cells that hold many particles."""
import numpy as np
import pytest

from swc import scenes

pytestmark = pytest.mark.gpu


def run(swc_mod, s):
    liq = swc_mod.DualParticleSphLiquid(s, warm_start="zero")
    liq.initialize()
    rho0 = np.array(liq.realInfo()[0])
    st = liq.advance(s.dt)
    out = rho0, st["n_virtual"], liq.getParticles()[0], np.array(liq.realInfo()[0])
    liq.close()
    return out


@pytest.mark.parametrize("cells", [(1000, 2048), (2900, 2900)])
def test_block_in_the_last_cells_of_a_large_lattice(swc_mod, cells):
    s = scenes.projection_block_2d(n=40, seed=3).rounded_to_float32()
    shift = [(c - g) * s.grid_spacing for c, g in zip(cells, s.grid_size)]
    far = s.copy(grid_size=(*cells, 1)[:len(s.grid_size)],
                 grid_origin=tuple(o - d for o, d in zip(s.grid_origin, shift)) + tuple(s.grid_origin[2:]))
    a, b = run(swc_mod, s), run(swc_mod, far)
    # the same particles in the same order of cells: FP32 sums of the same terms
    np.testing.assert_allclose(b[0], a[0], rtol=1e-6)
    assert a[1] == b[1]
    np.testing.assert_allclose(b[2], a[2], rtol=0, atol=1e-7)
    np.testing.assert_allclose(b[3], a[3], rtol=1e-5)


def test_order_within_full_cells(swc_mod):
    """Up to dozens of particles in a cell, whose order follows from their ids alone."""
    s = scenes.projection_block_2d(n=40, seed=5)
    rng = np.random.default_rng(1)
    pos = s.positions.copy()
    pos[:1200] = pos[rng.integers(0, 60, 1200)] + rng.uniform(-2e-3, 2e-3, (1200, 2))
    s = s.copy(positions=pos).rounded_to_float32()
    a, b = run(swc_mod, s), run(swc_mod, s)
    for u, v in zip(a, b):
        assert np.array_equal(u, v)
    x, h = s.positions, 4 * s.particle_radius
    d = np.linalg.norm(x[:, None] - x[None], axis=2) / h
    w = np.where(d < 0.5, 6 * (d ** 3 - d ** 2) + 1, np.where(d < 1, 2 * (1 - d) ** 3, 0)).sum(1)
    rho = s.mass * 40 / (7 * np.pi * h ** 2) * w
    # FP32 sums of some hundred terms of one sign
    np.testing.assert_allclose(a[0], rho, rtol=2e-5)
