"""What the autotuner leaves behind for the resident solve: it is left out only
where it was timed and lost, for that method, precision and size class. Seen by
the kernels a sub-step launches."""
import pytest

from test_gpu_drift import launches
from test_gpu_resident import PINNED, scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def E():
    import emerald_b200
    return emerald_b200


def takes_resident(E, sim, sc, method):
    """Against the launches of the kernels per phase on the same scene."""
    sim.advance(method, 1)
    n = launches(sim, lambda: sim.advance(method, 1))
    pinned = E.Simulation.from_block_scene(sc)
    pinned.set_tuning(PINNED)
    pinned.advance(method, 1)
    phases = launches(pinned, lambda: pinned.advance(method, 1))
    pinned.close()
    return n + 10 < phases


def test_another_method_is_not_affected(E):
    """IISPH does not cover 34 tiles a share, DFSPH_P and IISPH_AP do."""
    sc = scene(E, 400, 400)
    sim = E.Simulation.from_block_scene(sc)
    assert takes_resident(E, sim, sc, "dfsph_p")
    sim.advance("iisph", 1)
    sim.autotune("iisph")
    assert not takes_resident(E, sim, sc, "iisph")
    assert takes_resident(E, sim, sc, "dfsph_p")
    assert takes_resident(E, sim, sc, "iisph_ap")
    sim.close()


def test_a_scene_it_does_not_cover_says_nothing_of_its_size_class(E):
    """810,000 particles (171 tiles a share) are above the limit of DFSPH_P,
    577,600 (122) in the same size class are not."""
    sc = scene(E, 900, 900)
    big = E.Simulation.from_block_scene(sc)
    big.advance("dfsph_p", 1)
    big.autotune("dfsph_p")
    assert not takes_resident(E, big, sc, "dfsph_p")
    big.close()
    sc = scene(E, 760, 760)
    sim = E.Simulation.from_block_scene(sc)
    assert takes_resident(E, sim, sc, "dfsph_p")
    sim.close()


def test_unpinning_returns_to_the_resident_solve(E):
    sc = scene(E, 97, 61)
    sim = E.Simulation.from_block_scene(sc)
    assert takes_resident(E, sim, sc, "dfsph_p")
    sim.set_tuning(PINNED)
    assert not takes_resident(E, sim, sc, "dfsph_p")
    sim.set_tuning()
    assert takes_resident(E, sim, sc, "dfsph_p")
    sim.close()
