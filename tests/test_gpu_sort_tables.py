"""The string sort's tables: their size follows from the strings and the
cutoff, whatever the number of parts, so that sorts of very many parts fit a
context's budget; count rows are zeroed as passes come to use them (digits of
8 and 10 bits, one segment up to thousands, a workspace that another call left
dirty)."""
import numpy as np
import pytest

from inputs import random_strings, shared_head, with_duplicates
from test_gpu_parity import u64

pytestmark = pytest.mark.gpu


def check(dsss, orc, ctx, hs, pb, small_max):
    order, lcp = dsss.local_sort_lcp(ctx, dsss.DeviceStrings(hs), len(pb) - 1, part_begin=pb, small_sort_max=small_max)
    ro, rl = orc.local_sort(orc.Strings.from_host(hs), pb)
    assert np.array_equal(u64(order, hs.n), ro)
    assert np.array_equal(u64(lcp, hs.n), rl)


@pytest.mark.parametrize("small_max", [0, 2])
def test_many_parts_fit(dsss, orc, small_max):
    """200000 parts of two strings in 100 bytes of scratch per string (the
    handles, ids, keys and lists take 49), more at a cutoff of 2, where
    every third string may start a large segment."""
    n, p = 400000, 200000
    hs = dsss.from_bytes_list(random_strings(n, 0, 12, b"AB", seed=1))
    ctx = dsss.Context(0, hbm_budget=n * (100 if small_max == 0 else 1400))
    check(dsss, orc, ctx, hs, np.arange(p + 1, dtype=np.uint64) * 2, small_max)
    ctx.close()


@pytest.mark.parametrize("small_max", [2, 40, 255, 256, 700, 1023, 1024, 1500])
@pytest.mark.parametrize("p", [1, 5, 700])
def test_rows_as_passes_use_them(dsss, orc, ctx, p, small_max):
    n = 300000
    hs = dsss.from_bytes_list(random_strings(n, 0, 9, b"ABCDE", seed=p))
    ds = dsss.DeviceStrings(hs)
    dsss.pd_sort(ctx, ds, 3)  # leaves its own data where the rows will be
    check(dsss, orc, ctx, hs, dsss.equal_parts(n, p), small_max)


@pytest.mark.parametrize("pivot", [0, 1])
@pytest.mark.parametrize("small_max", [64, 255, 256, 4096])
@pytest.mark.parametrize("fam", ["dups", "head", "distinct"])
def test_digits_and_pivots(dsss, orc, ctx, fam, small_max, pivot):
    """Digits of 8 and of 10 bits with and without pivot passes; distinct
    strings need no handles, the others go back to theirs."""
    n = 40000
    strs = {"dups": lambda: with_duplicates(random_strings(n, 0, 40, b"ACGT", seed=3), 0.5, seed=4),
            "head": lambda: shared_head(n, 200, 8, seed=5),
            "distinct": lambda: random_strings(n, 8, 9, bytes(range(33, 127)), seed=6)}[fam]()
    hs = dsss.from_bytes_list(strs)
    with dsss.tuned(sort_pivot=pivot):
        check(dsss, orc, ctx, hs, dsss.equal_parts(n, 3), small_max)
