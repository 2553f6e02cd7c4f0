"""The resident solve (one cooperative launch per sub-step) against the
launch-per-phase kernels, which a pinned tuning selects: positions,
velocities, the solver's arrays, iteration counts and error statistics are the
same bits. Both run the same per-particle functions in list order, so nothing
is tolerated."""
import numpy as np
import pytest

from conftest import assert_bitwise
from scenes import F

pytestmark = pytest.mark.gpu

PINNED = dict(apply=1, divergence=4, iisph_sum=4, iisph_beta=4)
METHODS = ("dfsph_p", "iisph", "iisph_ap", "iisph_pseudo_ap", "pcisph")
ARRAYS = {
    "dfsph_p": ("densities", "density_stars", "alphas", "divergence_kappas", "density_kappas"),
    "iisph": ("densities", "pressures", "density_stars", "aiis", "diis", "sum_dij_pjs"),
    "iisph_ap": ("densities", "pressures", "density_stars", "aiis", "pressure_accelerations"),
    "iisph_pseudo_ap": ("densities", "pressures", "density_stars", "aiis",
                        "pressure_accelerations"),
    "pcisph": ("densities", "pressures", "pressure_forces", "velocity_external_forces",
               "position_stars", "velocity_stars"),
}


@pytest.fixture(scope="module")
def E():
    import emerald_b200
    return emerald_b200


def scene(E, nx, ny, **kw):
    args = dict(time_per_step_flicks=1411200, sub_steps=4, iisph_max_pressure_iterations=20,
                iisph_error_average_threshold=F(0.001),
                dfsph_divergence_error_average_threshold=F(0.001),
                dfsph_density_error_average_threshold=F(0.0005),
                dfsph_max_correction_iterations=30)
    args.update(kw)
    return E.BlockScene(nx, ny=ny, dx=F(1.0 / (2 * max(nx, ny))), seed=nx + 7 * ny, **args)


def compare(E, sc, method, steps, forces=None):
    a = E.Simulation.from_block_scene(sc)
    b = E.Simulation.from_block_scene(sc)
    b.set_tuning(PINNED)
    for sim in (a, b):
        if forces is not None:
            sim.set_forces(forces)
    for k in range(2):
        sa, sb = a.advance(method, steps), b.advance(method, steps)
        for key in ("pressure_iterations", "divergence_iterations", "error_average", "error_max",
                    "divergence_error_average", "divergence_error_max", "dt", "error_flags"):
            assert sa[key] == sb[key], (key, sa[key], sb[key])
        # summed in double, in another order
        for key in ("error_average_exact", "divergence_error_average_exact"):
            assert abs(sa[key] - sb[key]) <= 1e-12 * max(1.0, abs(sb[key])), key
        for name, x, y in zip("xv", a.state(), b.state()):
            assert_bitwise(x, y, "%s %s" % (method, name))
        for name in ARRAYS[method]:
            assert_bitwise(a.array(name), b.array(name), "%s %s" % (method, name))
    a.close()
    b.close()


# one lane, one warp, a warp and a lane; a tile more or less than a block's
# least share of four; several blocks with a ragged end; one and several
# tiles a warp; more lists than the shared memory holds (the last one)
@pytest.mark.parametrize("nx,ny", [(1, 1), (8, 4), (11, 3), (31, 4), (43, 3), (97, 61), (300, 241),
                                   (420, 330)])
@pytest.mark.parametrize("method", METHODS)
def test_sizes(E, method, nx, ny):
    compare(E, scene(E, nx, ny), method, 3)


@pytest.mark.parametrize("nx,ny", [(601, 430), (700, 640)])
def test_lists_beyond_shared_memory(E, nx, ny):
    compare(E, scene(E, nx, ny), "dfsph_p", 5)


@pytest.mark.parametrize("method", METHODS)
def test_compensated(E, method):
    compare(E, scene(E, 120, 77, precision=E.PRECISION_COMPENSATED), method, 3)


@pytest.mark.parametrize("method", METHODS)
@pytest.mark.parametrize("ratio", [2.0, 2.6])
def test_long_and_cut_lists(E, method, ratio):
    """About 45 neighbours each, and more than the 64 a list keeps (cut lists
    are not symmetric, and particles near the walls have more than 32 boundary
    neighbours): the barrier form, with several blocks."""
    compare(E, scene(E, 60, 50, support_ratio=ratio, dfsph_max_correction_iterations=3,
                     iisph_max_pressure_iterations=3), method, 1)


@pytest.mark.parametrize("method", METHODS)
def test_caps_and_forces(E, method):
    """Loops capped at one iteration and at none, under a force whose value
    depends on position and velocity."""
    for cap in (1, 0):
        compare(E, scene(E, 70, 40, dfsph_max_correction_iterations=cap,
                         iisph_max_pressure_iterations=cap), method, 2,
                forces=[(E.FORCE_GRAVITY, 9.81), (E.FORCE_POLE, 1e-5, 0.3, 0.2),
                        (E.FORCE_DRAG, 0.1, 0.01)])


@pytest.mark.parametrize("method", ("dfsph_p", "iisph_ap"))
def test_batch_of_many_shares(E, method):
    """A batch with more shares than blocks: blocks take further shares, and
    every scene ends where it ends alone; one scene is paused for a while."""
    scenes = [scene(E, 40 + 13 * (k % 9), 30 + 17 * (k % 5)) for k in range(24)]
    scenes += [scene(E, 330, 301), scene(E, 5, 4)]
    b = E.Batch(sum(-(-len(s.fluid) // 128) * 128 for s in scenes),
                sum(-(-len(s.solid) // 128) * 128 for s in scenes), len(scenes))
    ids = [b.add_block_scene(s) for s in scenes]
    b.step(method, 2)
    b.set_active(ids[3], False)
    b.step(method, 1)
    b.set_active(ids[3], True)
    b.step(method, 2)
    for k in (0, 3, 7, 23, 24, 25):
        sim = E.Simulation.from_block_scene(scenes[k])
        sim.set_tuning(PINNED)
        sim.advance(method, 4 if k == 3 else 5)
        for name, x, y in zip("xv", b.state(ids[k]), sim.state()):
            assert_bitwise(x, y, "%s scene %d %s" % (method, k, name))
        sim.close()
    b.close()
