"""PLOC where its tiles and phases meet: sizes at the edges of the tiles of 224 and 992 clusters and
of the last 256, more tiles than blocks, equal boxes (ties only) and boxes whose areas overflow (the
search without the hardware's minimum and maximum), bit for bit against the restated builder."""
import numpy as np
import pytest

import little_renderer_b200 as L
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def own():
    return L.Context(0)


def same(ctx, boxes, bits=30):
    n = boxes.shape[0]
    lo, hi = np.zeros(3, np.float32), np.ones(3, np.float32)
    p = ctx.params(n, lo, hi, bits, 1)
    want_n, want_a = O.ploc(boxes, *O.params(lo, hi), bits)
    got_n, got_a = ctx.build(p, boxes)
    assert np.array_equal(got_a, want_a)
    bad = np.nonzero((got_n != want_n).any(axis=1))[0]
    assert bad.size == 0, (n, bad.size, bad[:5])


def boxes_of(n, seed, size=0.01):
    rng = np.random.default_rng(seed)
    c, h = rng.random((n, 3), dtype=np.float32), rng.random((n, 3), dtype=np.float32) * np.float32(size)
    out = np.zeros((n, 8), np.float32)
    out[:, 0:3], out[:, 4:7] = c - h, c + h
    return out


@pytest.mark.parametrize("n", [3, 4, 31, 32, 33, 223, 224, 225, 255, 256, 257, 448, 449, 991, 992, 993, 1985, 66_303,
                               66_304, 99_456, 99_457, 150_001])
def test_sizes(own, n):
    same(own, boxes_of(n, n))


@pytest.mark.parametrize("n", [200, 1500, 120_000])
def test_ties(own, n):
    b = boxes_of(n, 5)
    b[:, 0:3] = np.round(b[:, 0:3] * 8) / 8              # few distinct boxes: the lower pair wins
    b[:, 4:7] = b[:, 0:3] + np.float32(0.125)
    same(own, b)


@pytest.mark.parametrize("n", [100, 1500, 130_000])
@pytest.mark.parametrize("big", [1e30, np.inf])
def test_areas_that_overflow(own, n, big):
    b = boxes_of(n, 6)
    at = np.random.default_rng(7).integers(0, n, max(1, n // 200))
    b[at, 4:7] = np.float32(big)
    same(own, b)
