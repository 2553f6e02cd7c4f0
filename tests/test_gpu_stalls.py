"""Waits inside kernels that give up (made to wait for what nobody sends, or
with a poll limit of none): the calls that return results say so, the
context stays usable, and a scene goes on from a new state with the bits it
would have had."""
import numpy as np
import pytest

from conftest import assert_bitwise
from test_gpu_resident import METHODS, scene

pytestmark = pytest.mark.gpu

POLLS = 1 << 22
GIVE_UP = {"barrier": 1, "values": 2}


@pytest.fixture(scope="module")
def E():
    import emerald_b200
    return emerald_b200


@pytest.mark.parametrize("method", METHODS)
@pytest.mark.parametrize("which", sorted(GIVE_UP))
def test_solve_that_gives_up(E, method, which):
    sc = scene(E, 97, 61)
    sim = E.Simulation.from_block_scene(sc)
    sim.advance(method, 2)
    snap = sim.snapshot()
    sim.inject(E.INJECT_STALL, GIVE_UP[which])
    sim.advance(method, 1, stats=False)
    for call in (sim.state, sim.time, sim.snapshot, sim.neighbors, lambda: sim.array("densities"),
                 lambda: sim.advance(method, 1), lambda: sim.frame(method), sim.state):
        with pytest.raises(E.EmeraldError):
            call()
    sim.inject(E.INJECT_STALL, 0)
    with pytest.raises(E.EmeraldError):
        sim.advance(method, 1)
    sim.restore(snap)
    sim.advance(method, 2)
    want = E.Simulation.from_block_scene(sc)
    want.advance(method, 4)
    for name, x, y in zip("xv", sim.state(), want.state()):
        assert_bitwise(x, y, "%s %s" % (method, name))
    # positions and velocities are a new state too
    sim.inject(E.INJECT_STALL, GIVE_UP[which])
    with pytest.raises(E.EmeraldError):
        sim.advance(method, 1)
    sim.inject(E.INJECT_STALL, 0)
    sim.set_state(sc.fluid, np.zeros_like(sc.fluid))
    assert sim.advance(method, 1)["error_flags"] == 0


@pytest.mark.parametrize("method", ("dfsph_p", "iisph_ap"))
@pytest.mark.parametrize("which", sorted(GIVE_UP))
def test_batch_that_gives_up(E, method, which):
    """More shares than blocks: a scene whose blocks gave up, or that found no
    blocks any more, reports it; one that was solved has its results."""
    scenes = [scene(E, 40 + 13 * (k % 9), 30 + 17 * (k % 5)) for k in range(24)]
    scenes += [scene(E, 330, 301), scene(E, 5, 4)]
    sizes = [sum(-(-len(p) // 128) * 128 for p in ps)
             for ps in ([s.fluid for s in scenes], [s.solid for s in scenes])]
    b = E.Batch(sizes[0], sizes[1], len(scenes))
    ids = [b.add_block_scene(s) for s in scenes]
    b.step(method, 1)
    b.synchronize()
    b.inject(E.INJECT_STALL, GIVE_UP[which])
    b.step(method, 1)
    with pytest.raises(E.EmeraldError):
        b.synchronize()
    with pytest.raises(E.EmeraldError):
        b.step(method, 1)
    b.inject(E.INJECT_STALL, 0)
    failed = []
    for k, sc in enumerate(scenes):
        want = E.Simulation.from_block_scene(sc)
        want.advance(method, 2)
        try:
            got = b.state(ids[k])
        except E.EmeraldError:
            failed.append(k)
            with pytest.raises(E.EmeraldError):
                b.stats(ids[k])
        else:
            for name, x, y in zip("xv", got, want.state()):
                assert_bitwise(x, y, "scene %d %s" % (k, name))
        want.close()
    assert 24 in failed
    for k in failed:
        b.remove_scene(ids[k])
    if len(failed) < len(scenes):
        b.step(method, 1)
        b.synchronize()
    b.close()


@pytest.mark.parametrize("n", [2, 2048, 2049, 30000])
def test_pair_sort_that_gives_up_is_sorted_all_the_same(E, n):
    import ctypes

    import torch
    rng = np.random.Generator(np.random.PCG64(n))
    z = rng.integers(0, max(n // 3, 1), n).astype(np.uint64)
    index = rng.integers(0, max(n // 2, 1), n).astype(np.uint64)   # some pairs twice
    pairs = np.stack([z, index], 1)
    size = ctypes.c_size_t()
    assert E.lib.emerald_index_pairs_workspace(n, ctypes.byref(size)) == 0
    work = torch.full((size.value,), 0xA5, dtype=torch.uint8, device="cuda")
    none = ctypes.c_uint32(0)
    for polls in (ctypes.byref(none), None):
        d = torch.from_numpy(pairs.view(np.int64).copy()).cuda()
        assert E.lib.emerald_sort_index_pairs_inject(
            n, d.data_ptr(), work.data_ptr(), work.numel(),
            torch.cuda.current_stream().cuda_stream, polls) == 0
        assert np.array_equal(d.cpu().numpy().view(np.uint64), pairs[np.lexsort((index, z))])


def test_storage_sort_that_gives_up_is_left_out(E):
    """The order of the storage changes no result; the sort products fail."""
    sc = scene(E, 97, 61)
    a = E.Simulation.from_block_scene(sc)
    b = E.Simulation.from_block_scene(sc)
    b.inject(E.INJECT_SORT_POLLS, 0)
    for sim in (a, b):
        sim.advance("dfsph_p", 20)
    for name, x, y in zip("xv", a.state(), b.state()):
        assert_bitwise(x, y, name)
    with pytest.raises(E.EmeraldError):
        b.sort()
    b.inject(E.INJECT_SORT_POLLS, POLLS)
    for x, y in zip(a.sort(), b.sort()):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("method", METHODS)
@pytest.mark.parametrize("graphs", (True, False))
def test_refused_launch_takes_the_kernels_per_phase(E, method, graphs):
    """A device that refuses the cooperative launch steps a scene all the
    same, from the first call on or from a later one."""
    sc = scene(E, 97, 61)
    want = E.Simulation.from_block_scene(sc)
    want.frame(method)
    want.advance(method, 3)
    for early in (True, False):
        sim = E.Simulation.from_block_scene(sc)
        sim.set_graphs(graphs)
        if early:
            sim.inject(E.INJECT_REFUSE, 1)
        assert sim.frame(method)["error_flags"] == 0
        sim.inject(E.INJECT_REFUSE, 1)
        assert sim.advance(method, 3)["error_flags"] == 0
        for name, x, y in zip("xv", sim.state(), want.state()):
            assert_bitwise(x, y, "%s %s" % (method, name))
        sim.close()
