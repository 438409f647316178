"""The one-launch PCGs on what the Kuhn cubes with tiles of 128 do not reach:
tiles of 64 at every number of them per CTA, rows far longer than a cube's 15
blocks, and clusters beside the one launch.  Against the loop of two kernels (the
same scene beside more scenes than the GPU has SMs), to the bit; launch counts say
which of the two ran."""
import dataclasses

import numpy as np
import pytest

from hobakv1_gb300 import hobak, scenes
from oracle import oracle

pytestmark = pytest.mark.gpu


def moving(s, seed):
    rng = np.random.default_rng(seed)
    s.v0 = rng.normal(size=s.rest.shape) * 0.1
    s.v0[s.pinned] = 0.0
    return s


def tower(layers, sides, material="snh"):
    """A round tower around an axis whose vertices neighbour every vertex of two
    rings: rows of 2 sides + 3 blocks."""
    n = sides + 1
    a = 2 * np.pi * np.arange(sides) / sides
    ring = np.stack([np.cos(a), 0 * a, np.sin(a)], axis=1)
    layer = np.concatenate([np.zeros((1, 3)), ring])
    h = 2 * np.pi / sides
    rest = np.concatenate([layer + [0.0, h * j, 0.0] for j in range(layers)])
    tets = []
    for j in range(layers - 1):
        for i in range(sides):
            v = sorted([j * n, j * n + 1 + i, j * n + 1 + (i + 1) % sides])
            w = [k + n for k in v]
            tets += [(v[0], v[1], v[2], w[2]), (v[0], v[1], w[1], w[2]), (v[0], w[0], w[1], w[2])]
    tets = np.array(tets, dtype=np.int32)
    flip = scenes.tet_volumes(rest, tets) < 0
    tets[flip] = tets[flip][:, [0, 2, 1, 3]]
    x0 = np.zeros_like(rest)
    x0[:, 1] = -0.02 * rest[:, 1]
    return dataclasses.replace(scenes.config2_scene(2, material), rest=rest, tets=tets,
                               pinned=np.arange(n, dtype=np.int32), x0=x0, v0=np.zeros_like(rest), dt=0.2)


def alone_and_in_the_loop(s, opts, **tuning):
    tiny = [scenes.config1_scene(1) for _ in range(200)]
    out = []
    for group in ([s], [s] + tiny):
        b = hobak.BATCH(group, opts)
        b.set_tuning(**tuning)
        before = b.launch_count()
        st = b.step(2)[0]
        out.append((st, b.launch_count() - before, *b.get_state(0)))
        b.close()
    (st, one, x, v), (stL, loop, xL, vL) = out
    assert st == stL and np.array_equal(x, xL) and np.array_equal(v, vL)
    assert one < 60 and loop - one >= 2 * st[0] >= 40  # without an iteration's kernels, and with them
    return x


# 10,648 vertices: 2 tiles of 64 a CTA, ..., 74,088: 8 (whole groups); 4,913: one
# tile a CTA, the first size past the thread-per-row kernel in FP64
@pytest.mark.parametrize("N", [16, 21, 27, 31, 34, 37, 39, 41])
@pytest.mark.parametrize("precision", [hobak.PRECISION_FP64, hobak.PRECISION_MIXED], ids=["fp64", "mixed"])
def test_tiles_of_64(N, precision):
    s = moving(scenes.config2_scene(N, "arap"), N)
    alone_and_in_the_loop(s, hobak.solver_opts(precision=precision, max_iters=40), tile_vertices=64)


# rows of 51 blocks: a thread per row in FP64, and a thread per vertex where 80% of
# the SMs have a CTA of 128 of them (16,000 vertices); of 99, too long for the first
# one's shared memory
@pytest.mark.parametrize("layers,sides", [(40, 24), (640, 24), (330, 48)])
@pytest.mark.parametrize("precision", [hobak.PRECISION_FP64, hobak.PRECISION_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("tile", [64, 128])
def test_long_rows(layers, sides, precision, tile):
    s = tower(layers, sides)
    x = alone_and_in_the_loop(s, hobak.solver_opts(precision=precision), tile_vertices=tile)
    if precision == hobak.PRECISION_FP64:
        sim = oracle.Sim(s, precond=hobak.PRECOND_BLOCK_JACOBI, integrator="velocity")
        sim.step(2)
        # every solve ends below 1e-8 of its right-hand side in both
        assert np.linalg.norm(x - sim.state()[0]) < 1e-8 * np.linalg.norm(sim.state()[0] + s.rest.reshape(-1))


@pytest.mark.parametrize("precision", [hobak.PRECISION_FP64, hobak.PRECISION_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("sizes,clusters", [((9, 12, 20, 7), (4, -1, -1, 1)), ((24, 10, 8), (-1, 2, -1)),
                                            ((8, 9, 3), (2, -1, -1))])
def test_clusters_beside_the_one_launch(sizes, clusters, precision):
    """Each scene as alone on its own path, also after the scenes' paths are swapped
    and swapped back."""
    group = [moving(scenes.config2_scene(N, "snh"), N) for N in sizes]
    opts = hobak.solver_opts(precision=precision)

    def run(b, k, path):
        b.set_tuning(cluster_pcg=1)
        for i, p in zip(k, path):
            b.set_scene_cluster(i, p)

    b = hobak.BATCH(group, opts)
    start = b.snapshot()
    others = tuple(-1 if c > 0 else 16 for c in clusters)
    for path in (clusters, others, clusters):
        run(b, range(len(group)), path)
        assert [p > 0 for p in b.pcg_path()] == [p > 0 for p in path]
        b.restore(start)
        before = b.launch_count()
        stats = b.step(2)
        # two kernels an iteration would be more than 80
        assert max(st[0] for st in stats) > 20 and b.launch_count() - before < 60
        for k, s in enumerate(group):
            alone = hobak.BATCH([s], opts)
            run(alone, [0], [path[k]])
            assert alone.step(2)[0] == stats[k]
            assert all(np.array_equal(g, w) for g, w in zip(b.get_state(k), alone.get_state(0)))
            alone.close()
    b.close()


def launches(s, precision, tile, steps=1):
    b = hobak.BATCH([s], hobak.solver_opts(precision=precision))
    b.set_tuning(tile_vertices=tile)
    before = b.launch_count()
    st = b.step(steps)[0]
    n = b.launch_count() - before
    b.close()
    return n, st[0]


@pytest.mark.parametrize("layers,sides,tile,one", [
    (200, 48, 64, False),   # 9,800 vertices: CTAs of 64
    (200, 48, 128, False),  # on half of the SMs
    (330, 48, 128, True),   # 16,170 on 127 of them
    (330, 48, 64, True),    # CTAs of 128 all the same
    (1400, 48, 128, False),  # 68,600: CTAs of 512
])
def test_uneven_rows_choose_the_faster_path_in_fp64(layers, sides, tile, one):
    """Meshes whose rows differ much in length take the one launch in FP64 only
    where it is the faster of the two."""
    s = tower(layers, sides)
    n, iterations = launches(s, hobak.PRECISION_FP64, tile)
    assert (n < 30) == one and (n >= 2 * iterations) == (not one) and iterations > 40


@pytest.mark.parametrize("layers,sides", [(77, 4), (43, 8), (49, 12)])  # 385, 387 and 637 vertices
@pytest.mark.parametrize("tile", [64, 128])
def test_last_cta_of_few_vertices(layers, sides, tile):
    """In FP32 a CTA lists its halo.  The last CTA of a scene may hold one vertex (385
    = 3 x 128 + 1 = 6 x 64 + 1), which has more than four neighbours in other CTAs."""
    s = tower(layers, sides)
    alone_and_in_the_loop(s, hobak.solver_opts(precision=hobak.PRECISION_MIXED), tile_vertices=tile)


def test_cluster_with_a_cta_of_one_vertex():
    """121 vertices in a cluster of 16: eight a CTA and one in the last.  Beside a
    scene whose halo has no room the class gathers from the other CTAs: same bits."""
    s = tower(11, 10)
    out = []
    for group in ([s], [s, scenes.config2_scene(34, "arap")]):
        b = hobak.BATCH(group, hobak.solver_opts(precision=hobak.PRECISION_MIXED))
        b.set_tuning(cluster_pcg=1)
        b.set_scene_cluster(0, 16)
        assert (b.pcg_path() == 16).all()
        st = b.step(2)[0]
        out.append((st, *b.get_state(0)))
        b.close()
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])
