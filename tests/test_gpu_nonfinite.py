"""A particle whose position has become a NaN (a flow that has blown up) falls
into cell (0, 0) with a NaN distance to everything near it. Its entries in the
others' lists carry W = 0 and GradW = 0, as for any distance outside the
support, so the others' sums do not change."""
import numpy as np
import pytest

from conftest import assert_bitwise
from scenes import F
from test_zz_no_alloc import static_lists

pytestmark = pytest.mark.gpu


# lists in the short form (the first two) and of 17 to 64 entries
@pytest.mark.parametrize("spacing", [1.0, 0.9, 0.5])
@pytest.mark.parametrize("h", [2.0 ** -17, 0.0123, 1.5])
def test_nan_position_adds_nothing(h, spacing):
    import torch

    import emerald_b200 as E
    h = F(h)
    side = 12
    g = (np.arange(side, dtype=np.float64) + 0.25) * float(h) * spacing
    rng = np.random.Generator(np.random.PCG64(3))
    xy = np.stack(np.meshgrid(g, g), -1).reshape(-1, 2)
    xy = (xy + rng.uniform(-0.1, 0.1, xy.shape) * float(h) * spacing).astype(np.float32)
    n = len(xy)
    c0, i0, w0, g0 = static_lists(E, torch, xy, h)
    c1, i1, w1, g1 = static_lists(E, torch, np.concatenate([xy, [[F(np.nan), F(np.nan)]]]).astype(
        np.float32), h)
    # cells (-1..1)^2 look into cell (0, 0)
    near = (np.floor(xy / (F(2) * h)) <= 1).all(axis=1)
    assert near.any() and not near.all() and c0.max() < 64
    assert_bitwise(c1[:n], c0 + near.astype(np.uint8), "counts")
    k = np.arange(64)[None, :]
    last = near[:, None] & (k == c0[:, None])      # a NaN sorts behind every distance
    assert_bitwise(i1[:n], np.where(last, n, i0).astype(np.uint32), "indices")
    assert_bitwise(w1[:n], w0, "W")
    assert_bitwise(g1[:n], g0, "GradW")
    assert c1[n] == near.sum() if near.sum() <= 64 else c1[n] == 64
    assert not w1[n].any() and not g1[n].any()


@pytest.mark.parametrize("where", [(1e12, 1e12), (-1e12, 3e11), (0.3, -1e30), (3e38, 0.2)])
@pytest.mark.parametrize("m", [2, 17, 18, 65, 80])
def test_coincident_points_too_far_out_for_a_cell(where, m):
    """Cells are int32; positions past them share the outermost one. Points at
    the same place there are each other's neighbours like anywhere else: the
    first 64 by index, at distance 0, W(0) and no gradient."""
    import torch

    import emerald_b200 as E
    h = F(0.0123)
    rng = np.random.Generator(np.random.PCG64(m))
    far = np.full((m, 2), 0, np.float32) + np.float32(where)
    near = rng.uniform(0.0, 1.0, (40, 2)).astype(np.float32)
    xy = np.concatenate([far, near])
    counts, idx, w, gw = static_lists(E, torch, xy, h)
    c0, i0, w0, g0 = static_lists(E, torch, near, h)
    assert_bitwise(counts[m:], c0, "counts of the others")
    assert_bitwise(w[m:], w0, "W of the others")
    k = min(m - 1, 64)
    assert (counts[:m] == k).all()
    for i in range(m):
        want = [j for j in range(m) if j != i][:64]
        assert idx[i, :k].tolist() == want
    at_zero = F(1) / (h * h * h * F(3.14159274101257324218750))
    assert (w[:m, :k] == at_zero).all()
    assert not gw[:m].any()
