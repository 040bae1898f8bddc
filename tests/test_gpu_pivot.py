"""The sampled pivot of the MSD passes' pivot passes: chains of nested
prefixes (shared head, one string's prefixes, equal strings among them,
chains longer than the 127 bytes a pass resolves) in segments of a few to
thousands of strings; order and LCPs equal the oracle's."""
import numpy as np
import pytest

from inputs import prefixes_of_each_other, run_suffixes, shared_head, with_duplicates
from test_gpu_parity import u64

pytestmark = pytest.mark.gpu

FAMILIES = {
    "shared_head": lambda: shared_head(6000, 90, 12, seed=1),
    "long_head": lambda: shared_head(5000, 400, 3, seed=2),
    "prefixes": lambda: prefixes_of_each_other(5000, seed=3),
    "dups": lambda: with_duplicates(shared_head(6000, 200, 2, seed=4), 0.6, seed=5),
    "runs": lambda: run_suffixes(seed=6),
}


@pytest.mark.parametrize("small_max", [2, 63, 300, 4096])
@pytest.mark.parametrize("p", [1, 3])
@pytest.mark.parametrize("fam", FAMILIES)
def test_chains(dsss, orc, ctx, fam, p, small_max):
    hs = dsss.from_bytes_list(FAMILIES[fam]())
    order, lcp = dsss.local_sort_lcp(ctx, dsss.DeviceStrings(hs), p, small_sort_max=small_max)
    ro, rl = orc.local_sort(orc.Strings.from_host(hs), dsss.equal_parts(hs.n, p))
    assert np.array_equal(u64(order, hs.n), ro)
    assert np.array_equal(u64(lcp, hs.n), rl)
