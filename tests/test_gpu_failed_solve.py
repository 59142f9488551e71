"""A CG solve whose blocks give up waiting for one another: the wait limit is set to a single
look (swc_debug_wait_limit), so some block's wait runs out at the first meeting and the
kernel returns its status; nothing hangs.

The step returns SWC_CUDA_ERROR with the velocities not projected, and its half-made
solution starts nothing: the context goes on as one whose step ended with p = 0."""
import os

import numpy as np
import pytest

from swc import _lib, learn, scenes

pytestmark = pytest.mark.gpu

MODEL = os.path.join(os.path.dirname(learn.__file__), "models", "warm_start.npz")


def block(dim, n):
    """A block without walls (with p = 0 its gradient pass adds nothing), past the sizes whose
    solve is one cluster."""
    s = (scenes.projection_block_2d if dim == 2 else scenes.projection_block_3d)(n=n, seed=n).rounded_to_float32()
    z = np.zeros((0, dim))
    return s.copy(boundary_positions=z, boundary_normals=z, boundary_velocities=z)


def context(swc_mod, s, mode):
    liq = swc_mod.DualParticleSphLiquid(s, warm_start=mode, tolerance=1e-5)
    if mode == "learned":
        liq.setMlp(*learn.load_model(MODEL))
    liq.initialize()
    return liq


def fail(swc_mod, liq, step):
    liq.L.swc_debug_wait_limit(liq.h, 0)
    with pytest.raises(swc_mod.SwcError) as e:
        step()
    assert e.value.status == _lib.SWC_CUDA_ERROR
    liq.L.swc_debug_wait_limit(liq.h, -1)


@pytest.mark.parametrize("dim,n", [(2, 170), (3, 25), (3, 60)])
@pytest.mark.parametrize("mode", ["prefix", "node", "zero", "extrapolate", "learned"])
def test_failed_solve_is_contained(swc_mod, dim, n, mode):
    s = block(dim, n)
    liq, twin = context(swc_mod, s, mode), context(swc_mod, s, mode)
    for _ in range(4):
        assert liq.advance(s.dt)["status"] == twin.advance(s.dt)["status"] == 0
    fail(swc_mod, liq, lambda: liq.advance(s.dt))
    # the twin's step: a solve of no iterations from zero
    twin.setSolverOptions(warm_start="zero", max_iterations=0)
    assert twin.advance(s.dt)["status"] == _lib.SWC_CG_NOT_CONVERGED
    twin.setSolverOptions(warm_start=mode, max_iterations=-1)
    assert np.array_equal(liq.getParticles(), twin.getParticles())
    assert not np.any(liq.virtual()["p"])
    # and on: the next start is zero, the history begins again
    for k in range(4):
        a, b = liq.advance(s.dt), twin.advance(s.dt)
        assert a["status"] == 0 and (k or a["initial_rel_residual"] == 1.0)
        for key in ("cg_iterations", "initial_rel_residual", "rel_residual", "warm_start_used"):
            assert a[key] == b[key], (k, key)
        assert np.array_equal(liq.getParticles(), twin.getParticles())
    # a projection that fails, several times, and a context initialized again
    for _ in range(3):
        fail(swc_mod, liq, liq.project)
    for c in (liq, twin):
        c.setParticles(s.positions, s.velocities)
        c.initialize()
        assert c.advance(s.dt)["status"] == 0
    assert np.array_equal(liq.getParticles(), twin.getParticles())
    liq.close()
    twin.close()


def test_failed_solve_logs_no_features(swc_mod):
    s = block(3, 25)
    liq = swc_mod.DualParticleSphLiquid(s, warm_start="node", tolerance=1e-5, keep_features=True)
    liq.initialize()
    liq.advance(s.dt)
    assert liq.features()[0].shape[0] == liq.numVirtual()
    fail(swc_mod, liq, lambda: liq.advance(s.dt))
    with pytest.raises(swc_mod.SwcError) as e:
        liq.features()
    assert e.value.status == _lib.SWC_BAD_ARG
    liq.advance(s.dt)
    assert np.isfinite(liq.features()[1]).all()
    liq.close()
