"""The resident solve where a scene or a call is out of the ordinary, against
the launch-per-phase kernels, which a pinned tuning selects: the same bits and
the same statistics."""
import numpy as np
import pytest

from conftest import assert_bitwise
from scenes import F
from test_gpu_resident import ARRAYS, METHODS, PINNED, scene

pytestmark = pytest.mark.gpu

STATS = ("pressure_iterations", "divergence_iterations", "error_average", "error_max",
         "divergence_error_average", "divergence_error_max", "error_average_exact",
         "divergence_error_average_exact", "dt", "error_flags")


@pytest.fixture(scope="module")
def E():
    import emerald_b200
    return emerald_b200


def empty(E):
    sc = scene(E, 8, 4)
    return sc, np.zeros((0, 2), np.float32)


@pytest.mark.parametrize("method", METHODS)
def test_scene_without_particles_reports_its_loops(E, method):
    """A loop over no particles runs until its exit test passes, and the
    statistics say so."""
    sc, none = empty(E)
    a = E.Simulation(sc.params, sc.solid, none, None, sc.solid_volumes)
    b = E.Simulation(sc.params, sc.solid, none, None, sc.solid_volumes)
    b.set_tuning(PINNED)
    sa, sb = a.advance(method, 2), b.advance(method, 2)
    assert sb["pressure_iterations"] > 0
    for key in STATS:
        assert sa[key] == sb[key], (key, sa[key], sb[key])


@pytest.mark.parametrize("method", ("dfsph_p", "iisph"))
def test_batch_with_a_scene_without_particles(E, method):
    sc, none = empty(E)
    big = scene(E, 70, 60)
    got = []
    for pinned in (False, True):
        b = E.Batch(8192, 4096, 4)
        if pinned:
            b.set_tuning(PINNED)
        ids = [b.add_scene(sc.params, sc.solid, none, None, sc.solid_volumes),
               b.add_block_scene(big)]
        b.step(method, 2)
        got.append(([b.stats(k) for k in ids], b.state(ids[1])))
        b.close()
    for sa, sb in zip(got[0][0], got[1][0]):
        for key in STATS:
            if key.endswith("exact"):
                # summed in double, in another order
                assert abs(sa[key] - sb[key]) <= 1e-12 * max(1.0, abs(sb[key])), key
            else:
                assert sa[key] == sb[key], (key, sa[key], sb[key])
    for x, y in zip(got[0][1], got[1][1]):
        assert_bitwise(x, y, method)


@pytest.mark.parametrize("method", METHODS)
@pytest.mark.parametrize("nx,ny,ratio", [(300, 241, 1.0), (60, 50, 2.0), (60, 50, 2.6),
                                         (150, 130, 2.6)])
def test_no_iterations_at_all(E, method, nx, ny, ratio):
    """Loops capped at none, with many blocks and in the barrier form (lists
    cut at 64): no exchange orders the blocks, so what a block reads of its
    neighbours' velocities has to come before they integrate."""
    sc = scene(E, nx, ny, support_ratio=ratio, dfsph_max_correction_iterations=0,
               iisph_max_pressure_iterations=0)
    # (what only an iteration writes is left out)
    arrays = [name for name in ARRAYS[method]
              if (method, name) not in (("dfsph_p", "density_stars"), ("iisph", "sum_dij_pjs"))]
    b = E.Simulation.from_block_scene(sc)
    b.set_tuning(PINNED)
    b.advance(method, 2)
    want = [b.array(name) for name in arrays], b.state()
    for _ in range(4):
        a = E.Simulation.from_block_scene(sc)
        a.advance(method, 2)
        for name, x, y in zip("xv", a.state(), want[1]):
            assert_bitwise(x, y, "%s %s" % (method, name))
        for name, y in zip(arrays, want[0]):
            assert_bitwise(a.array(name), y, "%s %s" % (method, name))
        a.close()
    b.close()


@pytest.mark.parametrize("method", METHODS)
def test_arrays_nothing_has_written_are_zero(E, method):
    """Also where the device memory held something else before."""
    used = [E.Simulation.from_block_scene(scene(E, 60 + d, 50)) for d in range(8)]
    for sim in used:
        for m in METHODS:
            sim.advance(m, 1, stats=False)
    for sim in used[::2]:
        sim.close()
    sc = scene(E, 60, 50, dfsph_max_correction_iterations=0, iisph_max_pressure_iterations=0)
    sim = E.Simulation.from_block_scene(sc)
    fresh = E.Simulation.from_block_scene(sc)
    for name in ARRAYS[method]:
        if name != "pressures":                    # of the method the scene runs
            assert not fresh.array(name).any(), name
    sim.advance(method, 1)
    if method == "iisph":
        assert not sim.array("sum_dij_pjs").any()
    if method == "dfsph_p":
        assert not sim.array("density_stars").any()
