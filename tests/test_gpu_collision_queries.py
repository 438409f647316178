"""The collision queries' candidate filters against the oracle's scans over all
pairs: faces pressed together, just within and just beyond the collision
distance, crossed by rotation, and scenes of one batch that overlap in space."""
import numpy as np
import pytest

from hobakv1_gb300 import hobak, scenes
from oracle import oracle

pytestmark = pytest.mark.gpu


def pressed(N, gap, seed, turn):
    """Two cubes, the upper one turned about y and shifted so that its bottom
    face is `gap` above the lower cube's top (negative: into it)."""
    s = scenes.two_cubes_scene(N, gap=0.0, offset=0.03, seed=seed)
    rng = np.random.default_rng(seed)
    up = np.arange(s.nv) >= s.nv // 2
    s.x0 = rng.normal(size=s.rest.shape) * 0.01 / N
    p = s.rest[up]
    c, d = np.cos(turn), np.sin(turn)
    q = p.copy()
    q[:, 0] = 0.5 + c * (p[:, 0] - 0.5) + d * (p[:, 2] - 0.5)
    q[:, 2] = 0.5 - d * (p[:, 0] - 0.5) + c * (p[:, 2] - 0.5)
    s.x0[up] += q - p
    s.x0[up, 1] += gap
    return s


@pytest.mark.parametrize("N,gap,eps,turn", [(3, 0.0, 1e-2, 0.0), (4, 0.008, 1e-2, 0.3), (5, -0.004, 2e-2, 0.7),
                                            (7, 0.0099, 1e-2, 0.1), (6, 0.0, 0.1, 0.5), (9, 0.0005, 1e-3, 0.2)])
def test_pairs_equal_the_scan_over_all(N, gap, eps, turn):
    group = [pressed(N, gap, seed, turn) for seed in (1, 2)]  # both scenes at the same place
    b = hobak.BATCH(group, hobak.solver_opts(integrator=hobak.INTEGRATOR_POSITION))
    sims = []
    for k, s in enumerate(group):
        b.set_collisions(k, True, eps, 1e2, 1e-3)
        b.set_edge_collisions(k, True)
        sim = oracle.Sim(s, precond=1, integrator="position")
        sim.set_collisions(True, eps, 1e2, 1e-3, ee=True)
        sims.append(sim)
    n = 0
    for k, sim in enumerate(sims):
        pairs, _ = b.collision_pairs(k, detect_now=True)
        assert np.array_equal(pairs, sim.vf_pairs()[0])
        n += len(pairs)
    b.step(1)
    for k, sim in enumerate(sims):
        sim.step(1)
        quads = sim.ee_pairs()
        assert np.array_equal(b.edge_pairs(k), quads)
        n += len(quads)
    assert n > 0
