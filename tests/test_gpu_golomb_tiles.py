"""Golomb decoding over several tiles (256 chunks of 1024 bits each): streams
whose readers fall into step late (40-bit remainders), parameters that are
not powers of two, unary parts longer than a chunk and than a tile, and many
short or single-value blocks inside one tile.  Round trips; the words
themselves are compared with the oracle's coder in test_gpu_golomb.py."""
import numpy as np
import pytest

from test_gpu_golomb import dev, host

pytestmark = pytest.mark.gpu


def trip(dsss, ctx, values, counts, bs):
    words, _ = dsss.golomb_encode(ctx, dev(values), counts, bs)
    got, bc = dsss.golomb_decode(ctx, words)
    assert np.array_equal(host(got), np.asarray(values, np.uint64))
    assert bc.tolist() == [c for c in counts if c]


@pytest.mark.parametrize("b", [1 << 40, (1 << 40) + 1, 3 << 39, 1 << 63, 1 << 12, 4095, 1])
def test_several_tiles(dsss, ctx, b):
    rng = np.random.default_rng(b % 1009)
    n = 40000 if b > 1 else 300000  # 5 to 7 tiles and a remainder
    gaps = (rng.exponential(min(b, 1 << 44) * 0.7, n)).astype(np.uint64) if b < 1 << 60 else \
        rng.integers(0, 1 << 45, n, dtype=np.uint64)
    v = np.cumsum(gaps, dtype=np.uint64)
    trip(dsss, ctx, v, [n], [b])
    cut = [n // 3, 1, 0, n // 7, n - n // 3 - 1 - n // 7]
    trip(dsss, ctx, v, cut, [b, b + 1, 7, b, b])


@pytest.mark.parametrize("run", [1000, 1024 * 3 + 5, 256 * 1024 + 77])
def test_unary_parts_over_chunks_and_tiles(dsss, ctx, run):
    rng = np.random.default_rng(run)
    gaps = rng.integers(0, 30, 60000).astype(np.uint64)
    gaps[rng.integers(0, 60000, 5)] += np.uint64(8 * run)
    v = np.cumsum(gaps, dtype=np.uint64)
    trip(dsss, ctx, v, [len(v)], [8])


def test_many_short_blocks(dsss, ctx):
    rng = np.random.default_rng(2)
    counts = [int(x) for x in rng.choice([0, 1, 1, 1, 2, 3, 40, 700], 3000)]
    bs = [int(x) for x in rng.choice([1 << 20, 1 << 44, 12345678901], 3000)]
    v = np.concatenate([np.cumsum(rng.integers(0, 3 * b, c, dtype=np.uint64)) for c, b in zip(counts, bs)])
    trip(dsss, ctx, v, counts, bs)


@pytest.mark.parametrize("n,nr", [(2048, 1), (2048, 5000), (4096, 2), (6145, 3), (6145, 4), (30000, 20000)])
def test_many_ranges(dsss, ctx, n, nr):
    """More ranges than the encoder's tiles of 2048 values, and fewer; range
    starts at the tiles' edges, empty ranges at the end."""
    rng = np.random.default_rng(n + nr)
    cuts = np.sort(np.concatenate([rng.integers(0, n + 1, nr), np.arange(0, n, 2048)]))
    counts = np.diff(np.concatenate([[0], cuts, [n, n, n]])).tolist()
    v = np.cumsum(rng.integers(0, 900, n, dtype=np.uint64))
    trip(dsss, ctx, v, counts, [256] * len(counts))
