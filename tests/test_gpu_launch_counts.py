"""The number of kernels a simulation says it has launched."""
import pytest

from test_gpu_drift import launches
from test_gpu_resident import PINNED, scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def E():
    import emerald_b200
    return emerald_b200


@pytest.mark.parametrize("graphs", (True, False))
def test_a_re_sort_is_four_launches(E, graphs):
    """Keys, the sort, the permutation and its commit: every sixteenth
    sub-step has them beside what the others have."""
    sim = E.Simulation.from_block_scene(scene(E, 97, 61))
    sim.set_graphs(graphs)
    counts = [launches(sim, lambda: sim.advance("dfsph_p", 1)) for _ in range(34)]
    assert counts[16] == counts[17] + 4 and counts[32] == counts[33] + 4
    assert len(set(counts[1:16] + counts[17:32])) == 1


def test_frames_of_either_solve_count_their_own(E):
    """A frame with the kernels per phase counts the same after a frame with
    the resident solve as in a simulation that never ran it, and the other way
    about."""
    sc = scene(E, 97, 61)
    a, b, c = (E.Simulation.from_block_scene(sc) for _ in range(3))
    a.frame("dfsph_p")
    b.set_tuning(PINNED)
    c.frame("dfsph_p")
    b.frame("dfsph_p")
    a.set_tuning(PINNED)
    assert launches(a, lambda: a.frame("dfsph_p")) == launches(b, lambda: b.frame("dfsph_p"))
    c.frame("dfsph_p")
    a.set_tuning()
    b.set_tuning()
    want = launches(c, lambda: c.frame("dfsph_p"))
    assert launches(a, lambda: a.frame("dfsph_p")) == want
    assert launches(b, lambda: b.frame("dfsph_p")) == want


def test_timing_with_and_without_the_resident_solve(E):
    """Timed sub-steps run the kernels per phase unless the caller asks for
    the solve they would run untimed."""
    sim = E.Simulation.from_block_scene(scene(E, 97, 61))
    sim.enable_timing(True)
    sim.advance("dfsph_p", 1)
    assert "dfsph_density" in sim.kernel_times() and "solve" not in sim.kernel_times()
    sim.enable_timing(True, resident=True)
    sim.advance("dfsph_p", 1)
    assert "solve" in sim.kernel_times() and "dfsph_density" not in sim.kernel_times()
    sim.enable_timing(False)
