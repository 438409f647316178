"""Contact pairs of a scene do not depend on its unit of length: the queries' FP32
filters only drop pairs that the exact tests drop, also where their squares leave
the range of FP32."""
import numpy as np
import pytest

from hobakv1_gb300 import hobak, scenes
from oracle import oracle

pytestmark = pytest.mark.gpu


def pressed(N, scale):
    """Two cubes, the upper one turned about y and pressed into the lower one."""
    s = scenes.two_cubes_scene(N, gap=0.0, offset=0.03, seed=1)
    rng = np.random.default_rng(1)
    up = np.arange(s.nv) >= s.nv // 2
    s.x0 = rng.normal(size=s.rest.shape) * 0.01 / N
    p = s.rest[up]
    c, d = np.cos(0.7), np.sin(0.7)
    q = p.copy()
    q[:, 0] = 0.5 + c * (p[:, 0] - 0.5) + d * (p[:, 2] - 0.5)
    q[:, 2] = 0.5 - d * (p[:, 0] - 0.5) + c * (p[:, 2] - 0.5)
    s.x0[up] += q - p
    s.x0[up, 1] -= 0.004
    s.rest = s.rest * scale
    s.x0 = s.x0 * scale
    return s


# powers of two: the FP64 tests see the same numbers.  Edges of 0.2: squares of
# FP32 overflow from 2^66 on (1.4e19), everything does at 2^70
@pytest.mark.parametrize("power", [-10, 0, 40, 63, 65, 66, 67, 68, 70, 90])
def test_pairs_at_every_scale(power):
    scale, eps = 2.0 ** power, 2e-2
    s = pressed(5, scale)
    b = hobak.BATCH([s], hobak.solver_opts(integrator=hobak.INTEGRATOR_POSITION, max_iters=3))
    b.set_collisions(0, True, eps * scale, 1e2, 1e-3)
    b.set_edge_collisions(0, True)
    sim = oracle.Sim(s, precond=1, integrator="position")
    sim.set_collisions(True, eps * scale, 1e2, 1e-3, ee=True)
    pairs, _ = b.collision_pairs(0, detect_now=True)
    assert len(pairs) > 40 and np.array_equal(pairs, sim.vf_pairs()[0])
    b.step(1)
    sim.step(1)
    quads = b.edge_pairs(0)
    assert len(quads) > 80 and np.array_equal(quads, sim.ee_pairs())
    b.close()
