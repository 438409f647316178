"""The loop of two kernels on scenes too large for one launch, in FP32: past 64
groups of 512 vertices (tiles of 64) or 512 (tiles of 128) a scene's sums are
formed by several CTAs, below that by one."""
import numpy as np
import pytest

from hobakv1_gb300 import hobak, scenes

pytestmark = pytest.mark.gpu


# 97,336 vertices: 191 groups; 117,649: 230; 274,625: 537 (the last
# segments with 31, 6 and 25 groups; one CTA for 48^3 with tiles of 128)
@pytest.mark.parametrize("N,tile", [(45, 64), (48, 64), (48, 128), (64, 128)])
def test_large_scenes_match_fp64(N, tile):
    s = scenes.config2_scene(N, "arap")
    rng = np.random.default_rng(N)
    s.x0 = rng.normal(size=s.rest.shape) * 0.01 / N
    s.x0[s.pinned] = 0.0
    s.dt = 1.0 / 300.0
    out = {}
    for precision in (hobak.PRECISION_FP64, hobak.PRECISION_MIXED):
        b = hobak.BATCH([s], hobak.solver_opts(precision=precision))
        b.set_tuning(tile_vertices=tile)
        start = b.snapshot()
        before = b.launch_count()
        stats = b.step(1)[0]
        assert b.launch_count() - before > 2 * stats[0]  # two kernels an iteration: the loop
        out[precision] = b.get_state(0)[0] + s.rest.reshape(-1)
        assert stats[1] == 1
        for _ in range(3):  # the same bits whichever CTAs come last
            b.restore(start)
            assert b.step(1)[0] == stats
            assert np.array_equal(b.get_state(0)[0] + s.rest.reshape(-1), out[precision])
        b.close()
    x64, x32 = out[hobak.PRECISION_FP64], out[hobak.PRECISION_MIXED]
    # both solves end below 1e-8 of their right-hand side; the mixed matrix is FP32
    assert np.linalg.norm(x32 - x64) < 1e-6 * np.linalg.norm(x64)
