"""The MSD passes over the arena (segments above the 4096-string cutoff):
groups of equal strings larger than the cutoff, which go on by id, strings
that end inside a digit, digits that span bytes, wide gaps between differing
bits, and segments at the edges of tiles.  Order and LCPs equal the oracle's;
equal strings keep ascending ids."""
import numpy as np
import pytest

from inputs import random_strings, with_duplicates
from test_gpu_parity import u64

pytestmark = pytest.mark.gpu


def pool(n, strs, seed):
    rng = np.random.default_rng(seed)
    return [strs[int(i)] for i in rng.integers(0, len(strs), n)]


def sparse(n, seed):
    """Keys whose differing bits lie far apart (first, middle and last bytes)."""
    rng = np.random.default_rng(seed)
    out = []
    for a, b, c in zip(rng.integers(0, 2, n), rng.integers(0, 4, n), rng.integers(0, 3, n)):
        out.append(bytes([65 + int(a), 80, 80, 80 + 5 * int(b), 80, 80, 80, 90 + int(c)]) + bytes(rng.integers(65, 70, 3).astype(np.uint8)))
    return out


FAMILIES = {
    "all_equal": lambda: [b"equal strings"] * 20000,
    "all_empty": lambda: [b""] * 9000,
    "three": lambda: pool(40000, [b"", b"a", b"a long string that many share"], 1),
    "ends": lambda: pool(60000, [b"A" * k for k in range(6)], 2),
    "ends_in_digit": lambda: pool(50000, [b"K", b"KA", b"KAB", b"KABCDEFGH", b"L", b"M" * 9], 3) +
    random_strings(20000, 0, 12, b"KLM", seed=4),
    "skew": lambda: with_duplicates(random_strings(60000, 0, 30, b"AB", seed=5), 0.7, seed=6),
    "sparse": lambda: sparse(50000, 7),
    "bytes": lambda: random_strings(60000, 1, 10, bytes(range(1, 256)), seed=8),
    "tile_edges": lambda: random_strings(3 * 4096 + 1, 5, 9, b"ABCDEFGHIJ", seed=9),
}


@pytest.mark.parametrize("p", [1, 3])
@pytest.mark.parametrize("small_max", [0, 700])
@pytest.mark.parametrize("fam", FAMILIES)
def test_passes(dsss, orc, ctx, fam, small_max, p):
    strs = FAMILIES[fam]()
    hs = dsss.from_bytes_list(strs)
    with dsss.tuned(sort_pivot=1 if p == 1 else 0):
        order, lcp = dsss.local_sort_lcp(ctx, dsss.DeviceStrings(hs), p, small_sort_max=small_max)
    ro, rl = orc.local_sort(orc.Strings.from_host(hs), dsss.equal_parts(hs.n, p))
    assert np.array_equal(u64(order, hs.n), ro)
    assert np.array_equal(u64(lcp, hs.n), rl)
