"""The min tree behind prefix decompression at the edges of its blocks (2048
values, 11 levels per launch) and scans whose arrays start off a 16-byte word:
the staged pipeline against the oracle at those sizes."""
import numpy as np
import pytest

from inputs import random_strings
from test_gpu_parity import u64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [2, 3])
@pytest.mark.parametrize("n", [2, 3, 127, 1024, 2047, 2048, 2049, 4095, 4096, 4097, 20481, 70001])
def test_staged_sizes(dsss, orc, ctx, n, p):
    strs = random_strings(n, 4, 60, b"AB", seed=n)
    hs = dsss.from_bytes_list(strs)
    ds = dsss.DeviceStrings(hs)
    order, lcp = dsss.local_sort_lcp(ctx, ds, p)
    dp, _ = dsss.dp_prefixes(ctx, ds, order, lcp, p)
    iv = dsss.partition(ctx, ds, order, dp, p)
    g = dsss.bucket_scatter(ctx, ds, p, order, lcp, dp, iv)
    out = dsss.lcp_merge(ctx, g["chars"], g["char_total"], g["lcp"], g["counts"], g["offsets"],
                         char_start=g["char_start"])
    pb = dsss.equal_parts(n, p)
    r = orc.pd_sort(orc.Strings.from_host(hs), pb)
    assert np.array_equal(iv, r["intervals"])
    assert np.array_equal(u64(out["merged_lcp"], n), r["merged_lcp"])
    local = u64(order, n)

    def merged(index, pe):
        return [strs[int(local[int(pb[int(q)]) + int(i)])] for i, q in zip(index, pe)]

    assert merged(u64(out["perm_index"], n), u64(out["perm_pe"], n)) == merged(r["perm_index"], r["perm_pe"])
