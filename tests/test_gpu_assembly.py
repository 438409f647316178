"""The system matrix's symmetric assembly (each block above the diagonal summed
once and written to both places) on a mesh whose vertex order is random: a
row's neighbours lie on both sides of it and in other 32-vertex slices."""
import dataclasses

import numpy as np
import pytest

from hobakv1_gb300 import hobak, scenes
from oracle import oracle

pytestmark = pytest.mark.gpu


def shuffled(N):
    s = scenes.config2_scene(N, "snh")
    order = np.random.default_rng(N).permutation(s.nv)  # new vertex k was vertex order[k]
    place = np.argsort(order)
    return dataclasses.replace(s, rest=s.rest[order].copy(), tets=place[s.tets].astype(np.int32),
                               pinned=np.sort(place[s.pinned]).astype(np.int32), x0=s.x0[order].copy(),
                               v0=s.v0[order].copy())


# 8 vertices in one slice, 27 (a partial one), 64 (two full ones), 512 (sixteen)
@pytest.mark.parametrize("N", [1, 2, 3, 7])
@pytest.mark.parametrize("integrator,name", [(hobak.INTEGRATOR_VELOCITY, "velocity"),
                                             (hobak.INTEGRATOR_POSITION, "position"),
                                             (hobak.INTEGRATOR_NEWMARK, "newmark")],
                         ids=["velocity", "position", "newmark"])
# every solve ends below 1e-8 of its right-hand side in both; the mixed matrix is FP32
@pytest.mark.parametrize("precision,bound", [(hobak.PRECISION_FP64, 1e-8), (hobak.PRECISION_MIXED, 1e-6)],
                         ids=["fp64", "mixed"])
def test_shuffled_mesh_matches_oracle(N, integrator, name, precision, bound):
    s = shuffled(N)
    b = hobak.BATCH([s], hobak.solver_opts(precision=precision, integrator=integrator))
    sim = oracle.Sim(s, precond=hobak.PRECOND_BLOCK_JACOBI, integrator=name)
    b.step(3)
    sim.step(3)
    x = b.get_state(0)[0] + s.rest.reshape(-1)
    xo = sim.state()[0] + s.rest.reshape(-1)
    assert np.linalg.norm(x - xo) < bound * np.linalg.norm(xo)
    b.close()
