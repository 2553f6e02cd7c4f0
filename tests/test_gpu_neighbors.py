"""The neighbour search at the edges of its short lists and of its kernel
values: particles with 15 to 17 neighbours (the short list holds 16) and 63 to
79 (the lists keep the first 64 in scan order), equal distances, coincident and
nearly coincident points, and supports on both sides of the range in which W
and GradW divide by multiply-adds ([2^-16, 2^10]). Counts, indices, W and GradW
equal the oracle's bit for bit: both round every operation the same way."""
import numpy as np
import pytest

from conftest import assert_bitwise
from scenes import F
from test_zz_no_alloc import static_lists

pytestmark = pytest.mark.gpu


def points(h, seed):
    """Groups 64 h apart, in random index order."""
    rng = np.random.Generator(np.random.PCG64(seed))
    g = np.arange(9, dtype=np.float64)
    groups = [
        np.stack(np.meshgrid(g, g), -1).reshape(-1, 2),      # spacing h: ties at every shell
        np.stack(np.meshgrid(g, g), -1).reshape(-1, 2) * 0.75,
        rng.uniform(0.0, 12.0, (150, 2)),
        np.zeros((3, 2)),                                    # coincident
        np.array([[0.0, 0.0], [1e-22, 0.0], [0.5, 0.5]]),
    ]
    for m in (16, 17, 18, 64, 65, 66, 80):                   # m - 1 neighbours each
        r = 0.95 * np.sqrt(rng.uniform(0.0, 1.0, m))
        t = rng.uniform(0.0, 2.0 * np.pi, m)
        groups.append(np.stack([r * np.cos(t), r * np.sin(t)], -1))
    xy = np.concatenate([p + np.array([64.0 * (k % 4), 64.0 * (k // 4)])
                         for k, p in enumerate(groups)])
    xy = (xy - np.array([0.0, 64.0])) * float(h)             # the fifth group at the origin
    return xy[rng.permutation(len(xy))].astype(np.float32)


@pytest.mark.parametrize("h", [2.0 ** -16 * (1 - 2.0 ** -24), 2.0 ** -16, 0.0123, 1.5, 2.0 ** 10,
                               2.0 ** 10 * (1 + 2.0 ** -23)])
def test_lists_equal_the_oracle(oracle, h):
    import torch

    import emerald_b200 as E
    h = F(h)
    xy = points(h, 5)
    counts, idx, w, gw = static_lists(E, torch, xy, h)
    oc, oi, od, ov = oracle.neighborhoods(xy, xy, True, F(2) * h)
    assert {2, 15, 16, 17, 63, 64} <= set(oc.tolist())
    assert_bitwise(counts, oc, "counts")
    live = np.arange(64)[None, :] < oc[:, None]
    assert_bitwise(idx, np.where(live, oi, 0), "indices")
    ow = np.zeros_like(w)
    og = np.zeros_like(gw)
    for i, k in zip(*np.nonzero(live)):
        ow[i, k] = oracle.kernel_w(od[i, k], h)
        og[i, k] = oracle.kernel_grad_w(-ov[i, k, 0], -ov[i, k, 1], h)
    assert_bitwise(w, ow, "W")
    assert_bitwise(gw, og, "GradW")
