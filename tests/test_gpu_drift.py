"""The resident solve's watch over the storage order's drift: which of the two
solves a scene takes, seen by the kernels a sub-step launches (the kernels per
phase launch three or more an iteration)."""
import numpy as np
import pytest

from conftest import assert_bitwise
from test_gpu_resident import PINNED, scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def E():
    import emerald_b200
    return emerald_b200


def launches(target, step):
    n = target.kernel_launches()
    step()
    return target.kernel_launches() - n


def test_a_new_scene_starts_as_not_drifted(E):
    """Also where the device memory held something else before: here, what
    scenes left there whose lists are cut at 64 (the barrier form, which
    reports the largest drift there is)."""
    kw = dict(support_ratio=2.6, dfsph_max_correction_iterations=3)
    used = [E.Simulation.from_block_scene(scene(E, 60 + k, 50, **kw)) for k in range(24)]
    for sim in used:
        sim.advance("dfsph_p", 1)
    for sim in used[::2]:
        sim.close()
    sc = scene(E, 512, 512)
    a = E.Simulation.from_block_scene(sc)
    b = E.Simulation.from_block_scene(sc)
    b.set_tuning(PINNED)
    for sim in (a, b):
        sim.advance("dfsph_p", 1)
    resident = launches(a, lambda: a.advance("dfsph_p", 1))
    assert 2 * resident < launches(b, lambda: b.advance("dfsph_p", 1))
    for sim in [a, b] + used[1::2]:
        sim.close()
