"""The bounded waits of the one-launch PCGs: a wait that runs out ends the step
with HOBAK_ERR_TIMEOUT, and the batch goes on as if it had not been.  A limit of
no polls makes the waits run out: a scene of many CTAs never finds every word
at its first look."""
import numpy as np
import pytest

from hobakv1_gb300 import hobak, scenes
from hobakv1_gb300._lib import HobakError

pytestmark = pytest.mark.gpu
HOBAK_ERR_TIMEOUT = -6  # include/hobak_gpu.h
DEFAULT = 1 << 21


def moving(N):
    s = scenes.config2_scene(N, "snh")
    rng = np.random.default_rng(N)
    s.v0 = rng.normal(size=s.rest.shape) * 0.1
    s.v0[s.pinned] = 0.0
    return s


# a thread per row (32 CTAs of 32 vertices); a thread per vertex in FP64 (4,913
# vertices) and in FP32
@pytest.mark.parametrize("N,precision", [(9, hobak.PRECISION_FP64), (16, hobak.PRECISION_FP64),
                                         (9, hobak.PRECISION_MIXED)], ids=["rows", "grid-fp64", "grid-mixed"])
@pytest.mark.parametrize("integrator", [hobak.INTEGRATOR_VELOCITY, hobak.INTEGRATOR_NEWMARK],
                         ids=["velocity", "newmark"])
@pytest.mark.parametrize("use_graph", [1, 0], ids=["graph", "eager"])
def test_a_wait_that_runs_out_ends_the_step(N, precision, integrator, use_graph):
    s = moving(N)
    b = hobak.BATCH([s], hobak.solver_opts(precision=precision, integrator=integrator, use_graph=use_graph))
    start = b.snapshot()
    want_stats = b.step(2)
    want = b.get_state(0)
    b.restore(start)
    b.set_wait_limit(0)
    with pytest.raises(HobakError) as e:
        b.step(1)
    assert e.value.code == HOBAK_ERR_TIMEOUT
    b.set_wait_limit(DEFAULT)
    b.restore(start)
    assert b.step(2) == want_stats
    assert all(np.array_equal(g, w) for g, w in zip(b.get_state(0), want))
    b.close()


@pytest.mark.parametrize("precision", [hobak.PRECISION_FP64, hobak.PRECISION_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("integrator", [hobak.INTEGRATOR_VELOCITY, hobak.INTEGRATOR_NEWMARK],
                         ids=["velocity", "newmark"])
def test_a_wait_that_ran_out_is_not_lost_in_a_later_solve(precision, integrator):
    """Of several steps, or Newton iterations, enqueued before the host looks."""
    s = moving(9)
    b = hobak.BATCH([s], hobak.solver_opts(precision=precision, integrator=integrator))
    start = b.snapshot()
    for change_options in (False, True):
        b.set_wait_limit(0)
        b.step_async(1)
        b.set_wait_limit(DEFAULT)
        b.restore(start)
        if change_options:
            b.set_solver(b.opts)
        b.step_async(1)  # this one succeeds
        for _ in range(2):  # the same answer until the next step
            with pytest.raises(HobakError) as e:
                b.wait()
            assert e.value.code == HOBAK_ERR_TIMEOUT
        b.restore(start)
        b.step(1)
        b.restore(start)
        b.set_solver(b.opts)
        b.step(1)
        b.restore(start)
    b.close()
