"""Particle counts on both sides of each change in how a pass shares its work: lanes per
particle pair (density, viscosity), lanes per node pair (virtual gather), pieces of a brick
and lanes per particle (pressure gradient)."""
import numpy as np
import pytest

from swc import scenes
from test_gpu_parity import TOL_V, rel, sync_oracle

pytestmark = pytest.mark.gpu


# n^dim particles.  3D: 8 lanes per pair up to 32,768 particles, 4 up to 65,536, 2 up to
# 131,072; gather 4 lanes up to 48,000 and 2 up to 290,000; gradient 2 x 2 up to 262,144.
# 2D: 4 lanes per pair up to 65,536, 2 up to 131,072; gather and gradient as in 3D.
@pytest.mark.parametrize("dim,n", [(3, 3), (3, 31), (3, 33), (3, 37), (3, 41), (3, 51), (3, 65), (3, 67),
                                   (2, 5), (2, 221), (2, 257), (2, 363), (2, 513), (2, 541)])
def test_splits_follow_the_oracle(swc_mod, oracle_mod, dim, n):
    build = scenes.projection_block_2d if dim == 2 else scenes.projection_block_3d
    s = build(n=n, seed=n).rounded_to_float32()
    liq = swc_mod.DualParticleSphLiquid(s, warm_start="zero", max_iterations=4, keep_virtual_velocity=True)
    ref = oracle_mod.Oracle(s, max_iterations=4)
    liq.initialize()
    ref.initialize()
    sync_oracle(liq, ref)
    ref.set_pressure(np.zeros(0))
    liq.advance(s.dt)  # ends at the cap of 4 iterations
    ref.advance(s.dt)
    gv, ov = liq.virtual(), ref.virtual()
    assert np.array_equal(gv["node"], ov["node"])
    # FP32 sums of at most a few hundred terms (2e-5), and the rounding of the FP32 positions
    # after their step, a few ulp in units of the spacing.  Nodes whose only particles lie on
    # the edge of the support amplify that without limit: the oracle itself moves by 3.6% there
    # for half an ulp, at up to 1.4e-4 of the nodes.
    x = liq.getParticles()[0]
    shift = np.abs(x).max() * 2.0 ** -24 / (np.ptp(x[:, 0]) / max(n - 1, 1))
    for f in ("rho", "vol"):
        off = np.abs(gv[f] - ov[f]) > (2e-5 + 8 * shift) * np.abs(ov[f]) + 1e-6 * np.abs(ov[f]).max()
        assert off.mean() < 1e-3, (f, off.mean())
    np.testing.assert_allclose(gv["div"], ov["div"], rtol=0, atol=1e-4 * np.abs(ov["div"]).max())
    assert rel(liq.getParticles()[1], ref.particles()[1]) < TOL_V
    liq.close()


# sand: 8 lanes per particle up to 114,688 particles (2D: 65,536), then one
@pytest.mark.parametrize("dim,scale,low,high", [(3, 10, 1, 7 << 14), (3, 84, 1, 7 << 14), (3, 92, (7 << 14) + 1, 1 << 18),
                                                (2, 16, 1, 1 << 16), (2, 500, (1 << 16) + 1, 1 << 18)])
def test_sand_splits_follow_the_oracle(swc_mod, oracle_mod, dim, scale, low, high):
    from test_gpu_sand import _check_step, _pair

    s = scenes.sand_contact_block(dim, scale=scale, seed=scale, wall_depth=12 / (4 * scale))
    assert low <= s.positions.shape[0] <= high, s.positions.shape
    g, o = _pair(s, oracle_mod, swc_mod)
    for _ in range(2):
        _check_step(g, o, s.dt)


@pytest.mark.parametrize("dim", [2, 3])
def test_sand_more_contacts_than_a_list(swc_mod, oracle_mod, dim):
    """60 particles within a radius: 59 contacts each, past the 32 that the lanes share."""
    from test_gpu_sand import _check_step, _pair

    s = scenes.sand_contact_block(dim, scale=16, seed=2, wall_depth=12 / 64)
    rng = np.random.default_rng(4)
    s.positions[:60] = s.positions.mean(axis=0) + rng.uniform(-0.5, 0.5, (60, dim)) * s.radius
    g, o = _pair(s, oracle_mod, swc_mod)
    _check_step(g, o, s.dt)
