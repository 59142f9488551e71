"""The resident CG solve and the row passes at the brick counts where their forms change.

The solution is held against the block-per-brick operator kernel (k_true_residual): the
residual b - A x evaluated with it agrees with the recursive one to FP32 rounding, and
|x| relative errors of the product would show in it at once."""
import numpy as np
import pytest

from swc import scenes

pytestmark = pytest.mark.gpu


def bricks_2d(n):
    return scenes.projection_block_2d(n=n, seed=n)


def bricks_3d(n):
    return scenes.projection_block_3d(n=n, seed=n)


# active bricks on 152 SMs: one and a few (one cluster, lattices of up to 100 bricks or 27 in
# 3D); more; 3D up to 3 per block in groups of four warps and
# past that in groups of two, with one more than a whole round; 2D up to 8 per block in
# groups of two warps and past that single warps
@pytest.mark.parametrize("build,n,low,high", [
    (bricks_2d, 9, 1, 4), (bricks_2d, 121, 60, 100), (bricks_2d, 170, 101, 144), (bricks_2d, 601, 1217, 1700),
    (bricks_3d, 9, 8, 8), (bricks_3d, 45, 305, 456), (bricks_3d, 52, 457, 608), (bricks_3d, 60, 609, 800), (bricks_3d, 96, 2129, 2500)])
def test_solve_at_brick_counts(swc_mod, build, n, low, high):
    s = build(n).rounded_to_float32()
    liq = swc_mod.DualParticleSphLiquid(s, warm_start="zero", tolerance=1e-5, compute_true_residual=True)
    liq.initialize()
    for _ in range(2):
        st = liq.advance(s.dt)
        assert low <= st["active_bricks"] <= high, st
        assert st["status"] == 0 and st["rel_residual"] < 1e-5
        # recursive and true residual part by FP32 rounding of x, d and q alone: |A||x| 2^-24
        # per iteration, below 2e-6 |b| for these solves
        assert abs(st["true_rel_residual"] - st["rel_residual"]) < 2e-6, st
    # the diagonal of the row pass: A applied to a unit vector of one node gives alpha_hat there
    v = liq.virtual()
    k = int(np.argmax(v["alpha_hat"]))
    e = np.zeros(v["node"].shape[0])
    e[k] = 1.0
    assert liq.applyOperator(e)[k] == pytest.approx(v["alpha_hat"][k], rel=1e-6)
    liq.close()


@pytest.mark.parametrize("n,tol,cap", [(1, 1e-5, -1), (2, 1e-12, 200), (4, 1e-5, -1)])
def test_small_systems_follow_the_oracle(swc_mod, oracle_mod, n, tol, cap):
    """A few nodes around 1, 8 and 64 particles: the first two stall in the reference's own
    iteration (A is not symmetric) and end at the cap, with the same residual (its relative
    difference is that of two FP32 / FP64 runs of a contracting iteration, far below 1%)."""
    s = bricks_3d(n).rounded_to_float32()
    liq = swc_mod.DualParticleSphLiquid(s, warm_start="zero", tolerance=tol, max_iterations=cap)
    ref = oracle_mod.Oracle(s, tolerance=tol, max_iterations=cap)
    liq.initialize()
    ref.initialize()
    ref.set_pressure(np.zeros(0))
    st = liq.advance(s.dt)
    ref.advance(s.dt)
    o = ref.stats()
    assert (st["status"], st["n_virtual"]) == (o["status"], ref.num_virtual())
    assert abs(st["cg_iterations"] - o["iterations"]) <= 1
    if o["status"]:
        assert st["rel_residual"] == pytest.approx(o["rel_residual"], rel=1e-2)


@pytest.mark.parametrize("n", [9, 25])
def test_residual_that_vanishes_in_one_step(swc_mod, n):
    """alpha0 a million times the largest diagonal: A is alpha0 times the identity but for
    rows of at most 1e-6 alpha0, so one step takes r down to 1e-6 of itself and its norm
    comes from r - alpha q itself, not from the cancelling sums.  Bound: the rows' 1e-6
    (within a factor 2 after the move) and two FP32 roundings of r."""
    s = bricks_3d(n).rounded_to_float32()
    liq = swc_mod.DualParticleSphLiquid(s, warm_start="zero", tolerance=1e-5, compute_true_residual=True)
    liq.initialize()
    sc = liq.scalars()
    liq.setScalars(sc["rho0"], 1e6 * sc["alpha0"], sc["kappa"])
    st = liq.advance(s.dt)
    assert (st["status"], st["cg_iterations"]) == (0, 1), st
    assert 0 < st["rel_residual"] < 2e-6 + 2.0**-22
    assert abs(st["true_rel_residual"] - st["rel_residual"]) < 2.0**-22
    liq.close()


@pytest.mark.parametrize("build,n", [(bricks_2d, 9), (bricks_2d, 121), (bricks_3d, 9), (bricks_3d, 60)])
@pytest.mark.parametrize("tol,cap,status", [(2.0, -1, 0), (1e-6, 0, 1)])
def test_solves_that_end_at_their_start(swc_mod, build, n, tol, cap, status):
    """A start within the tolerance, and a cap of no iterations: x stays the start (0), whose
    residual is b itself, so both norms are sums of the same terms."""
    s = build(n).rounded_to_float32()
    liq = swc_mod.DualParticleSphLiquid(s, warm_start="zero", tolerance=tol, max_iterations=cap)
    liq.initialize()
    st = liq.advance(s.dt)
    assert st["status"] == status and st["cg_iterations"] == 0
    assert st["rhs_norm"] == pytest.approx(np.linalg.norm(liq.virtual()["div"]), rel=1e-6)
    assert st["rel_residual"] == 1.0 and st["initial_rel_residual"] == 1.0
    assert not np.any(liq.virtual()["p"])
    # and the next one runs as usual
    st = liq.advance(s.dt)
    assert st["n_virtual"] == liq.virtual()["node"].shape[0]
    liq.close()
