"""Solves at other scales of length and velocity than the scenes' own (centimetres, 0.1 m/s):
the sums of the iteration hold over the whole FP32 range that r.r does."""
import numpy as np
import pytest

from swc import scenes

pytestmark = pytest.mark.gpu


def block(dim, n, length=1.0, velocity=1.0):
    s = (scenes.projection_block_2d if dim == 2 else scenes.projection_block_3d)(n=n, seed=n).rounded_to_float32()
    t = s.copy(positions=s.positions * length, velocities=s.velocities * velocity,
               boundary_positions=s.boundary_positions * length)
    t.particle_radius *= length
    t.grid_spacing *= length
    t.grid_origin = tuple(o * length for o in s.grid_origin)
    t.mass *= length**dim
    t.boundary_mass *= length**dim
    t.enable_gravity = False
    return t


# one cluster and the blocks of the SMs, in 2D and 3D
SIZES = [(2, 9), (2, 170), (3, 9), (3, 25)]


# (3D at 2^-18: the FP32 kernel sums themselves end there)
@pytest.mark.parametrize("dim,n,length", [(d, n, f) for d, n in SIZES for f in (2.0**-12, 2.0**-16, 2.0**-18, 2.0**10)
                                          if d == 2 or f > 2.0**-18])
def test_scale_of_length(swc_mod, oracle_mod, dim, n, length):
    """Spacings from 38 nm to 10 m, one projection, against the oracle: alpha0 goes from 1e-2
    to 5e13 and D from 1e-2 to 1e7, so q = A d up to 1e20.  True and recursive residual part by
    |A||x| 2^-24 an iteration, below 2e-6 |b| (as at the scenes' own scale)."""
    s = block(dim, n, length=length)
    liq = swc_mod.DualParticleSphLiquid(s, warm_start="zero", tolerance=1e-5, compute_true_residual=True)
    ref = oracle_mod.Oracle(s, tolerance=1e-5)
    liq.initialize()
    ref.initialize()
    ref.set_pressure(np.zeros(0))
    st = liq.project()
    ref.project()
    o = ref.stats()
    assert st["status"] == 0 and st["rel_residual"] < 1e-5, st
    assert abs(st["true_rel_residual"] - st["rel_residual"]) < 2e-6, st
    assert abs(st["cg_iterations"] - o["iterations"]) <= 1
    liq.close()


@pytest.mark.parametrize("dim,n", SIZES)
@pytest.mark.parametrize("velocity", [2.0**-20, 2.0**46, 2.0**50])
def test_scale_of_velocity(swc_mod, dim, n, velocity):
    """Everything up to p is linear in the velocities, and a power of two scales without
    rounding: the same iterations, and p to the bit."""
    out = []
    for g in (1.0, velocity):
        s = block(dim, n, velocity=g)
        liq = swc_mod.DualParticleSphLiquid(s, warm_start="zero", tolerance=1e-5)
        liq.initialize()
        st = liq.project()
        assert st["status"] == 0, st
        out.append((st["cg_iterations"], st["rel_residual"], liq.virtual()["p"] / g))
        liq.close()
    assert out[0][:2] == out[1][:2]
    assert np.array_equal(out[0][2], out[1][2])


@pytest.mark.parametrize("dim,n", SIZES)
@pytest.mark.parametrize("velocity", [1.0, 1e5, 1e7, 1e12])
def test_tolerance_zero(swc_mod, dim, n, velocity):
    """Tolerance 0 runs down to the rule's own floor, |r| < 2.2e-16, from any |b|: up to 31
    decades below it.  x is at its FP32 limit long before (true residual below 2e-6 |b|, as at
    the other tolerances), so p is that of the unscaled velocities to the same measure."""
    s = block(dim, n, velocity=velocity)
    liq = swc_mod.DualParticleSphLiquid(s, warm_start="zero", tolerance=0.0, max_iterations=1500,
                                        compute_true_residual=True)
    liq.initialize()
    st = liq.project()
    assert st["status"] == 0, st
    assert st["rel_residual"] * st["rhs_norm"] < 2.3e-16
    assert 0 < st["true_rel_residual"] < 2e-6, st
    liq.close()
