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
