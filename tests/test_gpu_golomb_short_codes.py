"""Golomb decoding of short codes: b = 1, whose counts come from the zeros of
a chunk, and b = 3 and 5, counted while they are read; unary parts over a word,
a chunk and a tile, blocks that end with and without padding, blocks of a few
values next to long ones."""
import numpy as np
import pytest

from test_gpu_golomb import roundtrip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b", [1, 3, 5])
@pytest.mark.parametrize("long", [0, 63, 64, 1023, 1024, 3000, 270000])
def test_runs(dsss, orc, ctx, b, long):
    rng = np.random.default_rng(long + b)
    gaps = rng.integers(0, 4 * b, 9000).astype(np.uint64)
    gaps[rng.integers(0, 9000, 4)] += np.uint64(b * long)
    gaps[-1] = np.uint64(b * long)
    v = np.cumsum(gaps, dtype=np.uint64)
    roundtrip(dsss, orc, ctx, v, [len(v)], [b])
    roundtrip(dsss, orc, ctx, v, [2, 1, 0, 700, len(v) - 703], [b] * 5)


@pytest.mark.parametrize("n", [2, 3, 63, 64, 65, 66, 128, 129, 1024, 1025, 1026])
def test_ends(dsss, orc, ctx, n):
    """b = 1 with gaps of 0: n - 1 zero bits, so that 65, 129 and 1025 values
    fill their last word."""
    v = np.full(n, 5, np.uint64)
    roundtrip(dsss, orc, ctx, v, [n], [1])
    roundtrip(dsss, orc, ctx, np.concatenate([v, v + np.uint64(1), v]), [n, n, n], [1, 1, 7])
