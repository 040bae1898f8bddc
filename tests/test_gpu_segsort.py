"""The segment sorter on its own (inputs of at most 4096 strings never reach
an MSD pass): sizes at the edges of its variants, groups of equal strings
around every hand-over (8 / 32 strings), chains that leave a pivot at many
depths, LCPs over thousands of bytes (more pivot codes than buckets), and
common parts longer than one pivot pass compares (16382 bytes).  Order and
LCPs equal the oracle's; equal strings keep ascending ids."""
import numpy as np
import pytest

from inputs import prefixes_of_each_other, random_strings, shared_head, with_duplicates
from test_gpu_parity import u64

pytestmark = pytest.mark.gpu


def check(dsss, orc, ctx, strs, p=1):
    hs = dsss.from_bytes_list(strs)
    order, lcp = dsss.local_sort_lcp(ctx, dsss.DeviceStrings(hs), p)
    ro, rl = orc.local_sort(orc.Strings.from_host(hs), dsss.equal_parts(hs.n, p))
    assert np.array_equal(u64(order, hs.n), ro)
    assert np.array_equal(u64(lcp, hs.n), rl)


@pytest.mark.parametrize("alphabet", [b"ACGT", bytes(range(1, 256)), b"AB"], ids=["dna", "bytes", "ab"])
@pytest.mark.parametrize("n", [2, 3, 8, 9, 31, 32, 33, 255, 256, 257, 1023, 1024, 1025, 4095, 4096])
def test_sizes(dsss, orc, ctx, n, alphabet):
    check(dsss, orc, ctx, random_strings(n, 0, 40, alphabet, seed=n))


@pytest.mark.parametrize("c", [2, 7, 8, 9, 31, 32, 33, 40, 300, 1500])
def test_equal_strings(dsss, orc, ctx, c):
    """Groups of c equal strings (short ones, that end inside a key, and long
    ones) between distinct ones, in random order."""
    rng = np.random.default_rng(c)
    strs = []
    for _ in range(max(1, 2600 // (4 * c))):
        for L in (0, 5, 8, 300):
            strs += [bytes(rng.integers(65, 91, L).astype(np.uint8))] * c
    strs += random_strings(700, 0, 20, b"ABCDEF", seed=c)
    rng.shuffle(strs)
    check(dsss, orc, ctx, strs[:4096])


@pytest.mark.parametrize("head", [40, 250, 3000, 40000])
@pytest.mark.parametrize("n", [12, 32, 200, 900, 3000])
def test_chains(dsss, orc, ctx, n, head):
    """Strings that copy a random length of one head: every LCP up to `head`
    (beyond 4096 bytes no variant has a bucket per code; beyond 16382 a pass
    does not reach the end)."""
    if n * head > 40_000_000:
        n = 40_000_000 // head
    check(dsss, orc, ctx, with_duplicates(shared_head(n, head, 9, seed=head + n), 0.2, seed=3))


def test_long_common_parts(dsss, orc, ctx):
    """Common parts around the most bytes a pass compares, with equal strings."""
    rng = np.random.default_rng(8)
    base = bytes(rng.integers(65, 91, 33000).astype(np.uint8))
    strs = []
    for cut in (16373, 16381, 16382, 16383, 16390, 16391, 32760, 32764, 32772, 33000):
        strs += [base[:cut], base[:cut] + b"A", base[:cut] + b"zz", base[:cut] + b"zz", base]
    rng.shuffle(strs)
    for k in (len(strs), 32, 7):
        check(dsss, orc, ctx, strs[:k])


def test_prefixes_and_many_segments(dsss, orc, ctx):
    check(dsss, orc, ctx, prefixes_of_each_other(4096, seed=2))
    check(dsss, orc, ctx, with_duplicates(random_strings(20000, 0, 30, b"ab", seed=5), 0.5, seed=6), p=23)


@pytest.mark.parametrize("sizes", [(2, 3, 4, 5), (31, 32, 33), (63, 64, 65), (2, 60, 3, 62, 64, 33, 7)],
                         ids=["small", "lanes", "elements", "mixed"])
@pytest.mark.parametrize("reach", [20, 200, 700, 17000])
def test_groups_of_one_warp(dsss, orc, ctx, sizes, reach):
    """Groups with one 8-byte key, of sizes at the hand-over between warp and
    CTA and in mixtures that share a warp: copies of up to `reach` bytes of a
    common text, equal strings among them, a few that agree for much longer
    than the others."""
    rng = np.random.default_rng(reach + len(sizes))
    strs, g = [], 0
    while len(strs) < min(1500, 12_000_000 // reach):
        c = sizes[g % len(sizes)]
        head = bytes(rng.integers(65, 91, reach).astype(np.uint8))
        for _ in range(c):
            cut = reach if rng.random() < 0.1 else 8 + int(rng.integers(0, reach - 7))
            strs.append(head[:cut] + bytes(rng.integers(65, 68, int(rng.integers(0, 3))).astype(np.uint8)))
        g += 1
    rng.shuffle(strs)
    check(dsss, orc, ctx, strs)
