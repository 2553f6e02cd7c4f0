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


def mixing(E, n):
    """The default dam break: sixty sub-steps a frame that mix the particles
    within a few of them."""
    return E.BlockScene(n, dx=np.float32(1 / (2 * n)), seed=1)


def per_step(target, step, count):
    return [launches(target, step) for _ in range(count)]


@pytest.mark.parametrize("graphs", (True, False))
@pytest.mark.parametrize("method,n", [("dfsph_p", 440), ("iisph_ap", 400), ("iisph", 330),
                                      ("pcisph", 270)])
def test_drift_and_back(E, method, n, graphs):
    """A mixing flow, advanced without statistics: sub-steps go over to the
    kernels per phase, and back once the storage has been sorted; the bits are
    those of the kernels per phase throughout."""
    sc = mixing(E, n)
    a = E.Simulation.from_block_scene(sc)
    b = E.Simulation.from_block_scene(sc)
    a.set_graphs(graphs)
    b.set_tuning(PINNED)
    resident = min(per_step(a, lambda: a.advance(method, 1, stats=False), 3))
    a.advance(method, 60, stats=False)
    counts = per_step(a, lambda: a.advance(method, 1, stats=False), 180)
    # (a re-sort adds four)
    taken = ["resident" if c <= resident + 4 else "per phase" for c in counts]
    assert taken.count("per phase") >= 16        # from one re-sort to the next
    assert any(x == "per phase" and y == "resident" for x, y in zip(taken, taken[1:]))
    b.advance(method, 243, stats=False)
    for name, x, y in zip("xv", a.state(), b.state()):
        assert_bitwise(x, y, "%s %s" % (method, name))
    a.close()
    b.close()


def test_drift_in_frames_and_batches(E):
    sc = mixing(E, 440)
    a = E.Simulation.from_block_scene(sc)
    p = E.Simulation.from_block_scene(sc)
    p.set_tuning(PINNED)
    steps = 0
    for _ in range(2):
        a.frame("dfsph_p")
        steps += p.frame("dfsph_p")["sub_steps"]
    got = launches(a, lambda: a.frame("dfsph_p"))
    n = p.kernel_launches()
    steps += p.frame("dfsph_p")["sub_steps"]
    want = p.kernel_launches() - n
    assert 2 * got > want
    last = p.frame("dfsph_p")["sub_steps"]
    a.frame("dfsph_p")
    for name, x, y in zip("xv", a.state(), p.state()):
        assert_bitwise(x, y, "frames " + name)
    # the same scene in a batch, beside a small one
    small = mixing(E, 40)
    b = E.Batch(1 << 18, 1 << 15, 2)
    ids = [b.add_block_scene(sc), b.add_block_scene(small)]
    b.step("dfsph_p", steps)
    got = launches(b, lambda: b.step("dfsph_p", last))
    assert 2 * got > want
    for name, x, y in zip("xv", b.state(ids[0]), p.state()):
        assert_bitwise(x, y, "batch " + name)
    b.close()


def test_a_scene_after_a_drifted_one(E):
    """In the slot of a scene that had drifted, a new one starts with the
    resident solve, its particles sorted first."""
    sc = scene(E, 512, 512)
    b = E.Batch(1 << 18, 1 << 15, 1)
    sid = b.add_block_scene(mixing(E, 440))
    b.step("dfsph_p", 100)
    b.stats(sid)
    b.remove_scene(sid)
    sid = b.add_block_scene(sc)
    b.step("dfsph_p", 1)
    b.stats(sid)
    resident = per_step(b, lambda: b.step("dfsph_p", 1), 4)
    b.set_tuning(PINNED)
    phases = launches(b, lambda: b.step("dfsph_p", 1))
    assert all(2 * r < phases for r in resident), (resident, phases)
    b.close()


def test_drift_in_a_batch_whose_scenes_change(E):
    """A scene added to a batch that has run: its drift is told to the host,
    and the calls after it go over."""
    b = E.Batch(1 << 18, 1 << 15, 2)
    b.add_block_scene(scene(E, 40, 30))
    b.step("dfsph_p", 2)
    sc = mixing(E, 440)
    sid = b.add_block_scene(sc)
    b.step("dfsph_p", 40)
    b.synchronize()
    got = launches(b, lambda: b.step("dfsph_p", 20))
    p = E.Simulation.from_block_scene(sc)
    p.set_tuning(PINNED)
    p.advance("dfsph_p", 40)
    want = launches(p, lambda: p.advance("dfsph_p", 20))
    assert 2 * got > want
    for name, x, y in zip("xv", b.state(sid), p.state()):
        assert_bitwise(x, y, name)
    b.close()


def test_drift_within_one_long_call(E):
    """A mixing flow advanced by one call that the host does not wait in: the
    sub-steps past the thirty-second choose on the device."""
    sc = mixing(E, 440)
    a = E.Simulation.from_block_scene(sc)
    p = E.Simulation.from_block_scene(sc)
    p.set_tuning(PINNED)
    got = launches(a, lambda: a.advance("dfsph_p", 150, stats=False))
    p.advance("dfsph_p", 60, stats=False)
    want = launches(p, lambda: p.advance("dfsph_p", 90, stats=False))
    assert 2 * got > want
    for name, x, y in zip("xv", a.state(), p.state()):
        assert_bitwise(x, y, name)
