"""bench.py counts the sort's first pass and the multisplits as they run: the
words up to the key behind the part that all strings share, and 24 bytes per
string for every multisplit launch."""
import os
import sys
import types

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402


@pytest.mark.parametrize("shared,per", [(0, [8, 8]), (1, [16, 11]), (44, [56, 11]), (48, [56, 11]), (49, [64, 11]),
                                        (55, [64, 11])])
def test_first_pass_words(shared, per):
    """rel + 15 over 8 words of 8 bytes, or the string and its NUL."""
    algo, _ = bench.first_pass_bytes(np.array([200, 10], np.uint32), shared)
    assert algo == sum(per) + 2 * 20


def test_long_shared_part_writes_no_keys():
    algo, _ = bench.first_pass_bytes(np.array([200, 10], np.uint32), 56)
    assert algo == 57 + 12 + 11 + 12


def test_rooflines_as_they_run():
    torch = pytest.importorskip("torch")
    n, L = 1000, 200
    out = {"dp": torch.full((n,), 72, dtype=torch.int32), "merged_lcp": torch.full((n,), 50, dtype=torch.int32)}
    kt = {"k_prefix": (2, 0.02), "k_ms_scatter_pay": (4, 0.01), "stage:sort": (2, 0.06)}
    r = bench.sort_rooflines(out, np.full(n, L, np.uint32), n, kt, 2, 1000.0, "measured", 44)
    for k in (r["roofline"], r["rooflines"]["k_prefix"]):
        assert k["algo_bytes"] == 76 * n
        assert k["achieved"] == pytest.approx(76 * n / 1e-5 / 1e9) and k["frac"] == pytest.approx(k["achieved"] / 1000)
    assert r["rooflines"]["k_ms_scatter_pay"]["algo_bytes"] == 48 * n


@pytest.mark.parametrize("p", [1, 2])
def test_shared_prefix(p):
    torch = pytest.importorskip("torch")
    strs = [b"headCC", b"headA", b"headB", b"heaZ"]
    offs = np.cumsum([0] + [len(s) + 1 for s in strs])[:-1]
    ds = types.SimpleNamespace(chars=torch.tensor(list(b"\0".join(strs) + b"\0"), dtype=torch.uint8),
                               offsets=torch.from_numpy(offs), lengths=torch.tensor([len(s) for s in strs]))
    order = sorted(range(4), key=lambda i: strs[i])  # 3, 1, 2, 0
    if p == 1:
        out = {"part_begin": [0, 4], "local_order": torch.tensor(order)}
    else:  # PE 0 holds strings 0 and 1, PE 1 the others
        out = {"part_begin": [0, 2, 4], "local_order": torch.tensor([1, 0, 3, 2]),
               "perm_pe": torch.tensor([1, 0, 1, 0]), "perm_index": torch.tensor([0, 0, 1, 1])}
    assert bench.shared_prefix(out, ds, 4) == 3
