"""Node lattices whose last brick along x holds only a few nodes, with liquid up to the
lattice's last corner: the virtual gather of the empty brick slots must not walk cell
rows past the lattice (nor read past the cell ranges in the last row)."""
import numpy as np
import pytest

from swc import scenes
from test_gpu_parity import TOL_V, make_pair, rel, sync_oracle

pytestmark = pytest.mark.gpu


# n + 7 nodes per axis: 17 and 33 of a 16-wide brick column (2D), 17 and 26 of an 8-wide one (3D)
@pytest.mark.parametrize("dim,n", [(2, 10), (2, 26), (3, 10), (3, 19)])
def test_mostly_empty_last_brick(swc_mod, oracle_mod, dim, n):
    build = scenes.projection_block_2d if dim == 2 else scenes.projection_block_3d
    s, liq, ref = make_pair(swc_mod, oracle_mod, build(n=n, seed=n))
    sync_oracle(liq, ref)
    ref.set_pressure(np.zeros(0))
    assert liq.advance(s.dt)["status"] == 0
    ref.advance(s.dt)
    gv, ov = liq.virtual(), ref.virtual()
    assert np.array_equal(gv["node"], ov["node"])
    np.testing.assert_allclose(gv["rho"], ov["rho"], rtol=2e-5, atol=1e-6 * np.abs(ov["rho"]).max())
    np.testing.assert_allclose(gv["vol"], ov["vol"], rtol=2e-5, atol=1e-6 * np.abs(ov["vol"]).max())
    np.testing.assert_allclose(gv["div"], ov["div"], rtol=0, atol=1e-4 * np.abs(ov["div"]).max())
    assert rel(liq.getParticles()[1], ref.particles()[1]) < TOL_V
