"""The pair sort at the edges of its tiles (2048 keys), of one tile per block,
and of the sizes sorted in one launch (2^22), with keys that differ in no
digit, in one, in some and in all of them: the lexicographic order of the
pairs, exactly."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def keys(kind, n, rng):
    if kind == "equal":
        return np.full(n, 0x0123456789ABCDEF, np.uint64)
    if kind == "one digit":
        return np.uint64(0x11) + (rng.integers(0, 3, n).astype(np.uint64) << np.uint64(40))
    if kind == "cells":
        return rng.integers(0, max(n // 4, 1), n).astype(np.uint64)
    z = rng.integers(0, 1 << 64, n, dtype=np.uint64)
    z[::7] = np.uint64(0xFFFFFFFFFFFFFFFF)
    return z


@pytest.mark.parametrize("kind", ["equal", "one digit", "cells", "all"])
@pytest.mark.parametrize("n", [2, 2047, 2049, 148 * 2048 + 1, 1 << 19, (1 << 22) + 1])
def test_pairs_are_in_lexicographic_order(kind, n):
    import torch

    import emerald_b200 as E
    rng = np.random.Generator(np.random.PCG64(n))
    z = keys(kind, n, rng)
    index = rng.permutation(n).astype(np.uint64)
    pairs = np.stack([z, index], 1)
    size = ctypes.c_size_t()
    assert E.lib.emerald_index_pairs_workspace(n, ctypes.byref(size)) == 0
    work = torch.full((size.value,), 0xA5, dtype=torch.uint8, device="cuda")
    d = torch.from_numpy(pairs.view(np.int64).copy()).cuda()
    for _ in range(2):  # the second call finds the first one's workspace
        d.copy_(torch.from_numpy(pairs.view(np.int64)))
        assert E.lib.emerald_sort_index_pairs(n, d.data_ptr(), work.data_ptr(), work.numel(),
                                              torch.cuda.current_stream().cuda_stream) == 0
        out = d.cpu().numpy().view(np.uint64)
        assert np.array_equal(out, pairs[np.lexsort((index, z))])
