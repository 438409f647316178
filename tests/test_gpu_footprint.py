"""The servers' estimate of a scene's device bytes counts the one-launch PCG's
buffers: it covers the allocation up to 20^3 in both precisions."""
import pytest

from hobakv1_gb300 import hobak, scenes
from hobakv1_gb300.serving import footprint_bytes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 6, 13, 19, 20])
@pytest.mark.parametrize("precision", [hobak.PRECISION_FP64, hobak.PRECISION_MIXED], ids=["fp64", "mixed"])
def test_estimate_covers_the_allocation(N, precision):
    s = scenes.config2_scene(N, "snh")
    b = hobak.BATCH([s], hobak.solver_opts(precision=precision))
    assert footprint_bytes(s, precision) >= b.device_bytes()
    b.close()
