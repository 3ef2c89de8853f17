"""The one-block sort (up to 8192 items) and the hierarchy joined in a block first (512 leaves) at the
edges of their tiles, with codes that tie, run across blocks or differ in one bit, bit for bit against the
restated builder."""
import numpy as np
import pytest

import little_renderer_b200 as L
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def own():
    return L.Context(0)


def boxes_of(n, kind):
    rng = np.random.default_rng(n)
    c = rng.random((n, 3), dtype=np.float32)
    if kind == "ties":
        c = np.round(c * 4) / 4                      # a few codes, long runs of each
    if kind == "line":
        c[:, 1:] = 0.5
        c[:, 0] = np.linspace(0.99, 0.0, n)          # (falling: the sort turns it round)
    if kind == "one":
        c[:] = 0.25
    out = np.zeros((n, 8), np.float32)
    out[:, 0:3], out[:, 4:7] = c - np.float32(1e-3), c + np.float32(1e-3)
    return out


@pytest.mark.parametrize("kind", ["random", "ties", "line", "one"])
@pytest.mark.parametrize("bits", [30, 63])
@pytest.mark.parametrize("n", [1, 2, 3, 32, 33, 511, 512, 513, 1023, 1024, 1025, 2048, 2049, 5120, 5121, 8191, 8192, 8193,
                               70_001])
def test_lbvh(own, n, bits, kind):
    b = boxes_of(n, kind)
    lo, hi = np.zeros(3, np.float32), np.ones(3, np.float32)
    p = own.params(n, lo, hi, bits, 0)
    want_n, want_a = O.lbvh(b, *O.params(lo, hi), bits)
    got_n, got_a = own.build(p, b)
    assert np.array_equal(got_a, want_a)
    assert np.array_equal(got_n, want_n)
