"""swc_time_kernel: every kernel is timed on any state of a context, and leaves it as it was."""
import numpy as np
import pytest

from swc import _lib, scenes

pytestmark = pytest.mark.gpu

SOLVE = (0, 1, 6)  # product, meeting, step of the CG solve


def block(dim, n):
    return (scenes.projection_block_2d if dim == 2 else scenes.projection_block_3d)(n=n, seed=n).rounded_to_float32()


@pytest.mark.parametrize("dim,n", [(2, 9), (2, 170), (3, 9), (3, 25)])
def test_solve_phases_without_a_right_hand_side(swc_mod, dim, n):
    """At rest without gravity b = 0 and the solve itself makes no iteration; the timed one makes
    as many as asked for all the same, and so it does on a context that has made no step."""
    s = block(dim, n)
    s = s.copy(velocities=np.zeros_like(s.velocities))
    s.enable_gravity = False
    liq = swc_mod.DualParticleSphLiquid(s, warm_start="zero", tolerance=1e-5)
    liq.initialize()
    for k in range(2):
        for which in SOLVE:
            assert 0 < liq.timeKernel(which, 7) < 10.0  # ms
        st = liq.advance(s.dt)
        assert (st["status"], st["cg_iterations"], st["rhs_norm"]) == (0, 0, 0.0)
        assert not np.any(liq.virtual()["p"])
    liq.close()


@pytest.mark.parametrize("dim,n,reps", [(2, 9, 400), (2, 170, 400), (3, 9, 400), (3, 25, 400)])
def test_solve_phases_far_past_convergence(swc_mod, dim, n, reps):
    """400 iterations are past the point where r = 0 in FP32; the mean of a phase stays that of a
    few iterations (within a factor 4: shared machine), and the context's next steps are those of a
    context that timed nothing."""
    s = block(dim, n)
    liq, twin = (swc_mod.DualParticleSphLiquid(s, warm_start="node", tolerance=1e-5) for _ in range(2))
    for c in (liq, twin):
        c.initialize()
        c.advance(s.dt)
    for which in SOLVE:
        few, many = liq.timeKernel(which, 8), liq.timeKernel(which, reps)
        assert 0.25 < many / few < 4, (which, few, many)
    for which in (2, 4):
        assert liq.timeKernel(which, 3) > 0
    for _ in range(2):
        a, b = liq.advance(s.dt), twin.advance(s.dt)
        assert a["cg_iterations"] == b["cg_iterations"] and a["initial_rel_residual"] == b["initial_rel_residual"]
        assert np.array_equal(liq.getParticles(), twin.getParticles())
    liq.close()
    twin.close()


def test_a_timed_solve_that_fails_is_reported(swc_mod):
    s = block(3, 25)
    liq, twin = (swc_mod.DualParticleSphLiquid(s, warm_start="node", tolerance=1e-5) for _ in range(2))
    for c in (liq, twin):
        c.initialize()
        c.advance(s.dt)
    liq.L.swc_debug_wait_limit(liq.h, 0)
    for which in SOLVE:
        with pytest.raises(swc_mod.SwcError) as e:
            liq.timeKernel(which, 5)
        assert e.value.status == _lib.SWC_CUDA_ERROR
    liq.L.swc_debug_wait_limit(liq.h, -1)
    a, b = liq.advance(s.dt), twin.advance(s.dt)
    assert a["status"] == 0 and a["initial_rel_residual"] == b["initial_rel_residual"]
    assert np.array_equal(liq.getParticles(), twin.getParticles())
    liq.close()
    twin.close()


def test_gradient_after_a_breakdown(swc_mod):
    """A step whose solve broke down left its gradient pass out; timed, the pass is whole (a pass
    that returns at once takes a fiftieth)."""
    s = block(3, 60)
    liq = swc_mod.DualParticleSphLiquid(s, warm_start="zero", tolerance=1e-5)
    liq.initialize()
    liq.advance(s.dt)
    whole = liq.timeKernel(3, 5)
    v = s.velocities.copy()
    v[:, 0] = np.nan
    liq.setParticles(s.positions, v)
    with pytest.raises(swc_mod.SwcError) as e:
        liq.project()  # (an advance would move the particles out of every node's reach)
    assert e.value.status == _lib.SWC_NAN_DETECTED
    assert liq.timeKernel(3, 5) > 0.3 * whole
    liq.close()
