"""Training data of a step whose solve broke down is refused, not mixed with the last step's."""
import numpy as np
import pytest

from swc import _lib, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n", [(2, 9), (2, 170), (3, 25)])
def test_no_features_of_a_breakdown(swc_mod, dim, n):
    s = (scenes.projection_block_2d if dim == 2 else scenes.projection_block_3d)(n=n, seed=n).rounded_to_float32()
    liq = swc_mod.DualParticleSphLiquid(s, warm_start="zero", tolerance=1e-5, keep_features=True)
    liq.initialize()
    liq.project()
    f, t = liq.features()
    assert np.isfinite(f).all() and np.any(t)
    v = s.velocities.copy()
    v[:, 0] = np.nan
    liq.setParticles(s.positions, v)
    with pytest.raises(swc_mod.SwcError) as e:
        liq.project()
    assert e.value.status == _lib.SWC_NAN_DETECTED
    with pytest.raises(swc_mod.SwcError) as e:
        liq.features()
    assert e.value.status == _lib.SWC_BAD_ARG
    # and a good step is logged again
    liq.setParticles(s.positions, s.velocities)
    liq.project()
    f, t = liq.features()
    assert np.isfinite(f).all() and np.any(t)
    liq.close()
