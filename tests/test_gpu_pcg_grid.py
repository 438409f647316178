"""The tile path's one-launch PCGs (pcg_grid.cu; pcg_rows.cu for small FP64
batches) against its loop of two kernels
(solver.cu): a batch with more scenes than the GPU has SMs takes the loop, the
scene alone takes the one launch, and both give the same bits."""
import numpy as np
import pytest

from hobakv1_gb300 import hobak, scenes

pytestmark = pytest.mark.gpu


def moving(N, material, seed):
    s = scenes.config2_scene(N, material)
    rng = np.random.default_rng(seed)
    s.v0 = rng.normal(size=s.rest.shape) * 0.1
    s.v0[s.pinned] = 0.0
    return s


# vertices (N + 1)^3 against tiles of 128 (64): less than one tile, exactly one
# or four of them, ragged; 14, 15 and 16: more CTAs of 32 vertices in FP64
# than tiles, the last such size and the first past it; 27, 34 and 40: two, three and four tiles a CTA
@pytest.mark.parametrize("N", [1, 3, 4, 7, 9, 14, 15, 16, 27, 34, 40])
@pytest.mark.parametrize("precision", [hobak.PRECISION_FP64, hobak.PRECISION_MIXED], ids=["fp64", "mixed"])
def test_one_launch_equals_the_loop(N, precision):
    s = moving(N, "snh" if N % 2 else "arap", N)
    tiny = [scenes.config1_scene(1) for _ in range(200)]  # one CTA each: more than one per SM
    opts = hobak.solver_opts(precision=precision, max_iters=60 if N > 10 else 1000)
    for tile in (128, 64) if N < 10 else (128,):
        out = []
        for group in ([s], [s] + tiny):
            b = hobak.BATCH(group, opts)
            b.set_tuning(tile_vertices=tile)
            st = b.step(2)[0]
            out.append((st, *b.get_state(0)))
            b.close()
        assert out[0][0] == out[1][0]
        assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])


@pytest.mark.parametrize("precision", [hobak.PRECISION_FP64, hobak.PRECISION_MIXED], ids=["fp64", "mixed"])
# 63 CTAs of 32 vertices, and past 152; at the larger distance a CTA of 128 vertices
# has more contact incidences (309) than threads
@pytest.mark.parametrize("N,eps", [(9, 1e-2), (13, 1e-2), (13, 6e-2)])
def test_one_launch_equals_the_loop_in_contact(N, eps, precision):
    s = scenes.two_cubes_scene(N, offset=0.05)
    tiny = [scenes.config1_scene(1) for _ in range(200)]
    out = []
    for group in ([s], [s] + tiny):
        b = hobak.BATCH(group, hobak.solver_opts(precision=precision, integrator=hobak.INTEGRATOR_POSITION))
        b.set_collisions(0, True, eps, 1e3, 1e-3)
        b.set_edge_collisions(0, True)
        st = b.step(3)[0]
        assert len(b.collision_pairs(0)[0]) > 50 and len(b.edge_pairs(0)) > 50
        out.append((st, *b.get_state(0)))
        b.close()
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])


def test_scenes_of_one_batch_end_apart():
    """Stiff, soft, resting and parked scenes in one launch: each as alone."""
    group = scenes.config4_scenes(6, 5, 9)
    group[2].gravity = (0.0, 0.0, 0.0)  # right-hand side zero: done at its start
    b = hobak.BATCH(group)
    b.set_active(4, False)
    b.step(3)
    for k, s in enumerate(group):
        alone = hobak.BATCH([s])
        if k == 4:
            alone.set_active(0, False)
        alone.step(3)
        assert np.array_equal(b.get_state(k)[0], alone.get_state(0)[0]), k
