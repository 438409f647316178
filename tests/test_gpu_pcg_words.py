"""The tagged words through which the CTAs of the one-launch PCGs exchange their
partial sums: no word of an earlier solve may pass for one of the running solve,
and none of the running solve may be lost."""
import threading
import time

import numpy as np
import pytest

from hobakv1_gb300 import hobak, scenes

pytestmark = pytest.mark.gpu


def moving(N, seed, **kw):
    s = scenes.config2_scene(N, "snh")
    rng = np.random.default_rng(seed)
    s.v0 = rng.normal(size=s.rest.shape) * 0.1
    s.v0[s.pinned] = 0.0
    for k, v in kw.items():
        setattr(s, k, v)
    return s


def test_words_are_cleared_in_order_with_the_batchs_steps():
    """New solver options restart the solves' count, which clears the words.  The
    next step may follow at once, whatever another thread has queued on the
    default stream meanwhile."""
    import torch
    s = moving(9, 1)
    alone = hobak.BATCH([s])
    alone.step(4)
    want = alone.get_state(0)
    alone.close()
    stop = threading.Event()

    def busy():
        while not stop.is_set():
            torch.cuda._sleep(1_000_000)  # half a millisecond on the default stream
            time.sleep(0.0007)  # (no device-wide wait: the batch may be capturing)

    torch.cuda.init()
    t = threading.Thread(target=busy)
    t.start()
    try:
        for _ in range(25):
            b = hobak.BATCH([s])
            for _ in range(4):
                b.set_solver(b.opts)
                b.step(1)
            got = b.get_state(0)
            b.close()
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    finally:
        stop.set()
        t.join()


def test_a_scene_that_takes_over_another_ones_place():
    """Two FP64 scenes of two CTAs each; the second sits out a step, so that its
    next solve has the number of the first one's last, which took two iterations
    and left words of both.  The first then moves to a cluster and the second
    takes its place in the launch: as alone, to the bit."""
    first = moving(3, 2, dt=1e-7)  # A = M up to 1e-14: one iteration, and the test of its residual
    second = moving(3, 3)
    b = hobak.BATCH([first, second])
    b.set_tuning(cluster_pcg=1)
    for k in (0, 1):
        b.set_scene_cluster(k, -1)
    b.step(2)
    b.set_active(1, False)
    assert b.step(1)[0][0] <= 2
    b.set_active(1, True)
    b.set_scene_cluster(0, 1)
    assert list(b.pcg_path()) == [1, 0]
    st = b.step(1)[1]
    got = b.get_state(1)
    b.close()
    alone = hobak.BATCH([second])
    want = alone.step(3)[0]
    assert st == want
    assert all(np.array_equal(g, w) for g, w in zip(got, alone.get_state(0)))
    alone.close()
