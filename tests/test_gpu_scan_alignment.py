"""Scans into output arrays that start off a 16-byte word: the offsets that
dsss_ms_sort and dsss_hq_sort write, at a pointer 8 bytes into an allocation,
with fewer strings than one launch scans (32768) and more."""
import ctypes

import numpy as np
import pytest
import torch

from inputs import random_strings
from test_gpu_hq import check_hq
from test_gpu_ms import check_ms

pytestmark = pytest.mark.gpu


def arrays(n, cap):
    """Outputs of n strings; every array starts one element into its allocation."""
    a = {k: torch.empty(n + 1, dtype=torch.int32, device="cuda")[1:] for k in ("local_order", "lengths", "lcp", "source")}
    a["offsets"] = torch.full((n + 2,), -1, dtype=torch.int64, device="cuda")[1:]
    a["chars"] = torch.empty(cap + 64, dtype=torch.uint8, device="cuda")
    assert a["offsets"].data_ptr() % 16 == 8
    return a


@pytest.mark.parametrize("n", [7, 16384, 32768, 32769, 70001])
@pytest.mark.parametrize("path", ["ms", "hq"])
def test_offsets_off_a_word(dsss, orc, ctx, path, n):
    p = 3
    hs = dsss.from_bytes_list(random_strings(n, 0, 30, b"ABCD", seed=n))
    ds = dsss.DeviceStrings(hs)
    pb = dsss.equal_parts(n, p)
    cap = int(hs.lengths.astype(np.uint64).sum()) + n
    out = arrays(n, cap)
    ptr = {k: v.data_ptr() for k, v in out.items()}
    arena = ds.arena()
    if path == "ms":
        out.update(intervals=np.zeros(p * p, np.uint64), recv_counts=np.zeros(p, np.uint64))
        opts = dsss._opts(0, 2, 0, 0)
        res = dsss.MsResult(ptr["local_order"], out["intervals"].ctypes.data, ptr["chars"], cap, ptr["offsets"],
                            ptr["lengths"], ptr["lcp"], ptr["source"], out["recv_counts"].ctypes.data, 0)
        dsss.check(dsss.lib().dsss_ms_sort(ctx.h, ctypes.byref(arena), p, pb.ctypes.data, ctypes.byref(opts),
                                           ctypes.byref(res), None))
        out["avg_lcp"] = int(res.avg_lcp)
        check_ms(dsss, orc, hs, out, pb)
    else:
        out["counts"] = np.zeros(p, np.uint64)
        res = dsss.HqResult(out["counts"].ctypes.data, ptr["chars"], cap, ptr["offsets"], ptr["lengths"],
                            ptr["source"], 0)
        dsss.check(dsss.lib().dsss_hq_sort(ctx.h, ctypes.byref(arena), p, pb.ctypes.data, dsss.HQ_SEED,
                                           ctypes.byref(res), None))
        out["levels"] = int(res.levels)
        check_hq(dsss, orc, hs, out, pb)
    assert int(out["offsets"][n]) == -1  # nothing is written behind the last
