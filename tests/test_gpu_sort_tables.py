"""The string sort's tables: their size follows from the strings and the
cutoff, whatever the number of parts, so that sorts of very many parts fit a
context's budget; count rows are zeroed as passes come to use them (digits of
8 and 10 bits, one segment up to thousands, a workspace that another call left
dirty)."""
import numpy as np
import pytest

from inputs import random_strings
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
