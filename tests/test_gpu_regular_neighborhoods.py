"""The search of emerald_create_regular_neighborhoods at the edges of its short
lists: 15 to 17 neighbours (the short list holds 16) and 63 to 79 (the cap is
64), equal distances, coincident and nearly coincident points, negative cells
and cell (-1, -1), in one set and between two, with a last warp that is not
full. Counts, indices, distances and vectors equal the oracle's exactly."""
import ctypes

import numpy as np
import pytest

from conftest import assert_bitwise
from scenes import F
from test_gpu_neighbors import points

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cut", [0, 1, 19])
@pytest.mark.parametrize("same", [True, False])
def test_search_equals_the_oracle(oracle, same, cut):
    import torch

    import emerald_b200 as E
    L = E.lib
    h = F(0.0123)
    cell = F(2) * h
    other = points(h, 11)
    xy = other[cut:] if not same else other
    if same:
        xy = other = np.ascontiguousarray(other[cut:])
    other = np.concatenate([other, np.float32([[-h, -h]])]) if not same else other

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a)).cuda()

    def sort(p):
        n = len(p)
        x = dev(p)
        gc = torch.zeros((n, 2), dtype=torch.int32, device="cuda")
        z = torch.zeros(n, dtype=torch.int64, device="cuda")
        pairs = torch.zeros((n, 2), dtype=torch.int64, device="cuda")
        size = ctypes.c_size_t()
        assert L.emerald_index_pairs_workspace(n, ctypes.byref(size)) == 0
        work = torch.zeros(size.value, dtype=torch.uint8, device="cuda")
        bi = torch.zeros(n, dtype=torch.int32, device="cuda")
        assert L.emerald_compute_grid_coords(n, cell, 0.0, 0.0, gc.data_ptr(), x.data_ptr(), None) == 0
        assert L.emerald_compute_z_indices(n, z.data_ptr(), gc.data_ptr(), None) == 0
        assert L.emerald_compute_index_pairs(n, pairs.data_ptr(), z.data_ptr(), None) == 0
        assert L.emerald_sort_index_pairs(n, pairs.data_ptr(), work.data_ptr(), size.value, None) == 0
        assert L.emerald_compute_block_indices(n, bi.data_ptr(), pairs.data_ptr(), work.data_ptr(),
                                               size.value, None) == 0
        nb = int(bi[-1].item()) + 1
        blocks = torch.zeros((nb, 2), dtype=torch.int64, device="cuda")
        assert L.emerald_fill_blocks(n, blocks.data_ptr(), bi.data_ptr(), None) == 0
        return x, gc, pairs, blocks, nb

    torch.cuda.synchronize()
    ox, ogc, pairs, blocks, nb = sort(other)
    x, gc = (ox, ogc) if same else sort(xy)[:2]
    n = len(xy)
    bmap = ctypes.c_void_p()
    assert L.emerald_block_map_create(ctypes.byref(bmap)) == 0
    assert L.emerald_create_block_map(nb, bmap, blocks.data_ptr(), pairs.data_ptr(), None) == 0
    counts = torch.full((n,), 255, dtype=torch.uint8, device="cuda")
    idx = torch.zeros((n, 64), dtype=torch.int64, device="cuda")
    dist = torch.zeros((n, 64), dtype=torch.float32, device="cuda")
    vec = torch.zeros((n, 64, 2), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    assert L.emerald_create_regular_neighborhoods(
        n, cell, counts.data_ptr(), idx.data_ptr(), dist.data_ptr(), vec.data_ptr(), x.data_ptr(),
        gc.data_ptr(), ox.data_ptr(), pairs.data_ptr(), bmap, None) == 0
    torch.cuda.synchronize()
    assert L.emerald_block_map_destroy(bmap) == 0
    oc, oi, od, ov = oracle.neighborhoods(xy, other, same, cell)
    assert_bitwise(counts.cpu().numpy(), oc, "counts")
    live = np.arange(64)[None, :] < oc[:, None]
    # what is past a particle's count stays as it was
    assert_bitwise(idx.cpu().numpy(), np.where(live, oi, 0).astype(np.int64), "indices")
    assert_bitwise(dist.cpu().numpy(), np.where(live, od, 0).astype(np.float32), "distances")
    assert_bitwise(vec.cpu().numpy(), np.where(live[..., None], ov, 0).astype(np.float32), "vectors")
