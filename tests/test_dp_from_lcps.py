"""Distinguishing prefixes from the LCPs of one global order.  Over the order
of all strings, a string's prefix length is the first depth of the schedule
8, 24, 40, 72, ... above the larger LCP with its two neighbours, or its
length if that is smaller: checked against the oracle's hash rounds on the
CPU, and the kernel against the oracle on the GPU at the schedule's edges.
The hash rounds stay behind dsss_dp_prefixes (orders sorted per PE); their
forms are checked there under the knobs that pick them."""
import numpy as np
import pytest

from dist_oracle import pack_list
from inputs import cases, long_prefix, random_strings, shared_head, with_duplicates


def schedule_edges(seed=5):
    """Pairs and triples of strings whose LCPs and lengths lie at, one below
    and one above every depth of the schedule up to 264."""
    rng = np.random.default_rng(seed)
    strs = []
    for d in (8, 24, 40, 72, 136, 264):
        for l in (d - 1, d, d + 1):
            for extra in (0, 1, 2, 9):
                head = bytes(rng.integers(65, 91, l).astype(np.uint8))
                strs += [head + b"a" * extra, head + b"b" * extra, head]
    return strs


def families():
    return [(name, s) for name, s in cases() if len(s) >= 2] + [
        ("schedule_edges", schedule_edges()),
        ("edges_dups", with_duplicates(schedule_edges(6), 0.4)),
        ("long_prefix_dups", with_duplicates(long_prefix(3000, 100, 8), 0.2)),
        ("shared_head", shared_head(2000)),
        ("ab", random_strings(3000, 0, 60, b"AB", seed=5))]


def depth_above(m):
    d = 8
    step = 16
    while d <= m:
        d, step = 8 + step, 2 * step
    return d


@pytest.mark.parametrize("name,strs", families(), ids=[f[0] for f in families()])
def test_rule_equals_the_rounds(orc, name, strs):
    chars, offs, lens, _ = pack_list(strs)
    s = orc.Strings(chars, offs.astype(np.uint64), lens.astype(np.uint32))
    n = s.n
    pb = np.array([0, n], np.uint64)
    order, lcp = orc.local_sort(s, pb)
    dp, _ = orc.dp_rounds(s, pb, order, lcp)
    lcp = [int(x) for x in lcp] + [0]
    for i in range(n):
        m = max(lcp[i] if i else 0, lcp[i + 1])
        assert int(dp[i]) == min(depth_above(m), len(strs[int(order[i])])), (name, i)


@pytest.mark.gpu
@pytest.mark.parametrize("p", [2, 5])
@pytest.mark.parametrize("fam", [0, 1], ids=["edges", "edges_dups"])
def test_kernel_at_the_schedule_edges(dsss, orc, ctx, fam, p):
    from test_gpu_parity import check_pd
    strs = schedule_edges() if fam == 0 else with_duplicates(schedule_edges(6), 0.4)
    hs = dsss.from_bytes_list(strs)
    check_pd(dsss, orc, hs, dsss.pd_sort(ctx, dsss.DeviceStrings(hs), p), p)


@pytest.mark.gpu
@pytest.mark.parametrize("knobs", [dict(dp_filter_min=0), dict(dp_filter_min=0, dp_filter_bits=4), dict(dp_split=1),
                                   dict(dp_digest=64), dict(dp_digest=0), dict(dp_table=8)], ids=str)
@pytest.mark.parametrize("p", [1, 6])
def test_hash_rounds_under_knobs(dsss, orc, ctx, knobs, p):
    import torch
    strs = with_duplicates(long_prefix(3000, 90, 12, 71) + random_strings(3000, 0, 40, b"AB", 72), 0.3, 73)
    hs = dsss.from_bytes_list(strs)
    s = orc.Strings.from_host(hs)
    pb = dsss.equal_parts(hs.n, p)
    ro, rl = orc.local_sort(s, pb)
    rdp, rcounts = orc.dp_rounds(s, pb, ro, rl)
    order = torch.from_numpy(ro.astype(np.int32)).cuda()
    lcp = torch.from_numpy(rl.astype(np.int32)).cuda()
    with dsss.tuned(**knobs):
        dp, counts = dsss.dp_prefixes(ctx, dsss.DeviceStrings(hs), order, lcp, p)
    assert np.array_equal(dp.cpu().numpy().astype(np.uint64), rdp)
    assert counts.tolist() == rcounts.tolist()
