"""The hash rounds behind dsss_dp_prefixes under each of their knobs
(fingerprint filter, split hashing, table size, arena order): the full path
takes its distinguishing prefixes from the global order and runs no hash
round, so the knobs are tested where they act.  Prefix lengths and the
candidates left after every round equal the oracle's."""
import numpy as np
import pytest

from inputs import cases
from test_gpu_parity import host_of, u64

pytestmark = pytest.mark.gpu

CASES = [c for c in cases() if len(c[1]) >= 8]
KNOBS = [dict(dp_filter_min=0), dict(dp_filter_min=0, dp_filter_bits=4), dict(dp_filter_min=0, dp_filter_bits=64),
         dict(dp_filter_min=500), dict(dp_split=1), dict(dp_split=1, dp_digest=0), dict(dp_table=8, dp_digest=0),
         dict(dp_digest=0), dict(dp_digest=1), dict(dp_digest=64)]


def check(dsss, orc, ctx, hs, p, knobs):
    import torch
    s = orc.Strings.from_host(hs)
    pb = dsss.equal_parts(hs.n, p)
    ro, rl = orc.local_sort(s, pb)
    rdp, rcounts = orc.dp_rounds(s, pb, ro, rl)
    order = torch.from_numpy(ro.astype(np.uint32).view(np.int32)).cuda()
    lcp = torch.from_numpy(rl.astype(np.uint32).view(np.int32)).cuda()
    ds = dsss.DeviceStrings(hs)
    for kn in knobs:
        with dsss.tuned(**kn):
            dp, counts = dsss.dp_prefixes(ctx, ds, order, lcp, p)
        assert np.array_equal(u64(dp, hs.n), rdp), kn
        assert counts.tolist() == rcounts.tolist(), kn


@pytest.mark.parametrize("p", [2, 5])
@pytest.mark.parametrize("name,strs", CASES, ids=[c[0] for c in CASES])
def test_cases(dsss, orc, ctx, name, strs, p):
    check(dsss, orc, ctx, host_of(dsss, strs), p, KNOBS)


@pytest.mark.parametrize("gen", ["dn", "suffix"])
def test_larger(dsss, orc, ctx, gen):
    hs = dsss.gen_dn(60000, 100, 50, seed=31) if gen == "dn" else dsss.gen_suffix_strings(60000, 256, seed=3)
    check(dsss, orc, ctx, hs, 4, KNOBS)
