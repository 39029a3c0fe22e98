"""phx_schedule_morton against a sort by Z-order keys (CPU): the order of the quadtree walk, at sizes around its 8 x 8 tiles
and squares."""
from __future__ import annotations

import numpy as np
import pytest

import phoenix_b200 as P


def by_key(W, H):
    i, j = (a.ravel().astype(np.uint64) for a in np.meshgrid(np.arange(W), np.arange(H), indexing="ij"))
    key = np.zeros(W * H, np.uint64)
    for b in range(16):
        key |= ((i >> np.uint64(b)) & np.uint64(1)) << np.uint64(2 * b)
        key |= ((j >> np.uint64(b)) & np.uint64(1)) << np.uint64(2 * b + 1)
    return np.argsort(key, kind="stable")


@pytest.mark.parametrize("W,H", [(1, 1), (7, 9), (8, 8), (9, 8), (64, 64), (65, 1), (1, 513), (200, 150), (333, 217),
                                 (17, 4097), (65536, 2), (2, 65536), (65537, 2), (1, 70000)])
def test_morton_order(built, W, H):
    assert np.array_equal(P.schedule_morton(W, H), by_key(W, H))
