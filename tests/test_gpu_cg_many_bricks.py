"""The CG solve where a group of warps owns more than four bricks, whose neighbour tables are
then filled again in every product, and solves of several contexts at once."""
import threading

import numpy as np
import pytest

from swc import scenes

pytestmark = pytest.mark.gpu


# more than 152 SMs x 16 groups x 4 bricks in 2D, 152 x 14 x 4 in 3D
@pytest.mark.parametrize("dim,n,low,high,cap", [(2, 1600, 9729, 12000, 30), (3, 160, 8513, 10500, 12)])
def test_fifth_brick_of_a_group(swc_mod, dim, n, low, high, cap):
    """The recursive residual against the true one, which other kernels evaluate: apart by
    |A||x| 2^-24 an iteration, below 2e-6 |b|, where a wrong neighbour would show at once."""
    s = (scenes.projection_block_2d if dim == 2 else scenes.projection_block_3d)(n=n, seed=n).rounded_to_float32()
    liq = swc_mod.DualParticleSphLiquid(s, warm_start="zero", tolerance=1e-5, max_iterations=cap,
                                        compute_true_residual=True)
    liq.initialize()
    for _ in range(2):
        st = liq.advance(s.dt)
        assert low <= st["active_bricks"] <= high, st
        assert st["cg_iterations"] <= cap and st["rel_residual"] < 0.1
        assert abs(st["true_rel_residual"] - st["rel_residual"]) < 2e-6, st
    liq.close()


def run(swc_mod, s, mode, steps, start=None):
    liq = swc_mod.DualParticleSphLiquid(s, warm_start=mode, tolerance=1e-5)
    liq.initialize()
    if start is not None:
        start.wait()
    its = [liq.advance(s.dt)["cg_iterations"] for _ in range(steps)]
    out = its, liq.getParticles()
    liq.close()
    return out


def test_contexts_at_work_together(swc_mod):
    """Four contexts, a thread and a stream each, among them one whose solve is a cluster: each
    solve outside a cluster wants every SM, so they take turns, and every context ends where it
    ends alone, to the bit."""
    jobs = [(scenes.projection_block_3d(n=25, seed=1), "node"), (scenes.projection_block_3d(n=60, seed=2), "prefix"),
            (scenes.projection_block_2d(n=170, seed=3), "extrapolate"), (scenes.dam_break_2d(seed=4), "node")]
    jobs = [(s.rounded_to_float32(), mode) for s, mode in jobs]
    alone = [run(swc_mod, s, mode, 20) for s, mode in jobs]
    together, errors = [None] * len(jobs), []
    start = threading.Barrier(len(jobs))

    def work(k):
        try:
            together[k] = run(swc_mod, *jobs[k], 20, start)
        except Exception as e:  # noqa: BLE001  (shown below)
            errors.append((k, e))
            start.abort()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors, errors
    for a, b in zip(alone, together):
        assert a[0] == b[0]
        assert np.array_equal(a[1], b[1])
