"""The norm that ends a solve is that of the residual the solve holds."""
import numpy as np
import pytest

from swc import scenes

pytestmark = pytest.mark.gpu

# one cluster and the blocks of the SMs, in 2D and 3D, with the stencil's rows summed as in
# applyOperator's kernel (few bricks a block)
SIZES = [(2, 9), (2, 170), (3, 9), (3, 25), (3, 45)]


def context(swc_mod, dim, n, **kw):
    s = (scenes.projection_block_2d if dim == 2 else scenes.projection_block_3d)(n=n, seed=n).rounded_to_float32()
    liq = swc_mod.DualParticleSphLiquid(s, warm_start="zero", **kw)
    liq.initialize()
    return s, liq


@pytest.mark.parametrize("dim,n", SIZES)
@pytest.mark.parametrize("cap,tol", [(1, 1e-5), (-1, 0.9)])
@pytest.mark.parametrize("factor", [1.0, 30.0, 1e3])
def test_reported_residual_is_the_stored_one(swc_mod, dim, n, cap, tol, factor):
    """One iteration from zero, ended by its cap or by the tolerance: x = alpha b, r = b - alpha q
    with q = A b and alpha = |b|^2 / b.q, all in FP32 from sums far longer.  From applyOperator's
    q (the same additions) r is rebuilt to the bit, and its norm agrees with the reported one
    to the 44 bits of the sums.  (A prediction from the sums is off by the rounding of r,
    2^-31 and more.)  `factor` times alpha0 leaves quotients of the norms on both sides of the line
    between prediction and measurement."""
    s, liq = context(swc_mod, dim, n, max_iterations=cap, tolerance=tol)
    sc = liq.scalars()
    liq.setScalars(sc["rho0"], factor * sc["alpha0"], sc["kappa"])
    st = liq.project()
    if cap < 0 and st["cg_iterations"] != 1:
        pytest.skip("one step does not reach the tolerance")
    assert st["cg_iterations"] == 1
    L = np.longdouble
    b = liq.virtual()["div"].astype(np.float32)
    q = liq.applyOperator(b.astype(np.float64)).astype(np.float32)
    alpha = np.float32((b.astype(L) ** 2).sum() / (b.astype(L) * q.astype(L)).sum())
    r = (b.astype(L) - L(alpha) * q.astype(L)).astype(np.float32)
    rel = np.sqrt((r.astype(L) ** 2).sum() / (b.astype(L) ** 2).sum())
    assert abs(float(st["rel_residual"] / rel - 1)) < 2.0**-40
    liq.close()


@pytest.mark.parametrize("dim,n", SIZES)
@pytest.mark.parametrize("factor", [3.0, 10.0, 30.0, 300.0, 3e3])
def test_quotients_around_the_line(swc_mod, dim, n, factor):
    """Solves whose norms fall by a factor around and far past the line in every iteration end
    within the tolerance, true and recursive residual apart by the rounding of x and r."""
    s, liq = context(swc_mod, dim, n, tolerance=1e-5, compute_true_residual=True)
    sc = liq.scalars()
    liq.setScalars(sc["rho0"], factor * sc["alpha0"], sc["kappa"])
    st = liq.project()
    assert st["status"] == 0 and st["rel_residual"] < 1e-5, st
    assert abs(st["true_rel_residual"] - st["rel_residual"]) < 2e-6, st
    liq.close()
