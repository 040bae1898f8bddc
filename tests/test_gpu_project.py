"""Local orders, splitters, bounds and merged sequences read off the global
order: against the oracle where the selection of samples and the ranks inside
a splitter's run of equal strings can go wrong (tile edges of 2048 positions,
more samples than strings, PEs without strings, runs of equal strings across
PEs and tiles, empty strings, both samplers, uneven batches, samples cut
inside a run of the merge-sort path)."""
import numpy as np
import pytest

from inputs import long_prefix, random_strings, with_duplicates
from test_gpu_ms import check_ms
from test_gpu_parity import check_pd, u64

pytestmark = pytest.mark.gpu


def runs(n, kinds, seed):
    """n strings out of `kinds` distinct ones (runs of equal strings over many tiles)."""
    rng = np.random.default_rng(seed)
    pool = [bytes(rng.integers(97, 123, int(k)).astype(np.uint8)) for k in rng.integers(0, 30, kinds)]
    return [pool[int(i)] for i in rng.integers(0, kinds, n)]


FAMILIES = {
    "tile-1": lambda: random_strings(2047, 0, 12, b"ABC", seed=1),
    "tile": lambda: random_strings(2048, 3, 12, b"ABC", seed=2),
    "tile+1": lambda: random_strings(2049, 0, 12, b"ABC", seed=3),
    "few": lambda: random_strings(9, 0, 3, b"AB", seed=4),
    "equal": lambda: [b"same"] * 7000,
    "empty": lambda: [b""] * 5000 + [b"a", b"b"],
    "two": lambda: runs(9000, 2, 5),
    "ten": lambda: runs(9000, 10, 6),
    "dups": lambda: with_duplicates(long_prefix(9000, 60, 4, seed=7), 0.5, seed=8),
    "long_run": lambda: with_duplicates([b"x" * 700 + bytes([65 + i % 20]) for i in range(6000)], 0.5, seed=9),
}


@pytest.mark.parametrize("sampler", [0, 2])
@pytest.mark.parametrize("p", [2, 5, 33])
@pytest.mark.parametrize("fam", FAMILIES)
def test_partition_from_ranks(dsss, orc, ctx, fam, p, sampler):
    hs = dsss.from_bytes_list(FAMILIES[fam]())
    out = dsss.pd_sort(ctx, dsss.DeviceStrings(hs), p, sampler=sampler)
    check_pd(dsss, orc, hs, out, p, indexed=sampler == 2)


@pytest.mark.parametrize("fam", ["tile+1", "ten", "dups"])
def test_uneven_pes(dsss, orc, ctx, fam):
    hs = dsss.from_bytes_list(FAMILIES[fam]())
    n = hs.n
    pb = np.array([0, 0, 1, n // 2, n // 2, n // 2 + 3, n, n], np.uint64)
    out = dsss.pd_sort(ctx, dsss.DeviceStrings(hs), 7, part_begin=pb)
    check_pd(dsss, orc, hs, out, 7)


@pytest.mark.parametrize("sampler", [0, 2])
def test_batch_equals_single_calls(dsss, ctx, sampler):
    sets = [dsss.from_bytes_list(FAMILIES[f]()) for f in ("ten", "few", "tile", "equal", "dups")]
    sets.insert(2, dsss.from_bytes_list([]))
    hs, sb = dsss.concat_sets(sets)
    p = 6
    out = dsss.pd_sort_batched(ctx, dsss.DeviceStrings(hs), len(sets), p, dsss.batched_parts(sb, p), sampler=sampler)
    iv = np.asarray(out["intervals"]).reshape(len(sets), p * p)
    for s, h in enumerate(sets):
        b, e = int(sb[s]), int(sb[s + 1])
        if b == e:
            assert not iv[s].any()
            continue
        ref = dsss.pd_sort(ctx, dsss.DeviceStrings(h), p, sampler=sampler)
        assert np.array_equal(iv[s], np.asarray(ref["intervals"])), s
        for k in ("dp", "perm_index", "perm_pe", "merged_lcp"):
            assert np.array_equal(u64(out[k], hs.n)[b:e], u64(ref[k], h.n)), (s, k)
        assert np.array_equal(u64(out["local_order"], hs.n)[b:e] - b, u64(ref["local_order"], h.n)), s


@pytest.mark.parametrize("p", [3, 7])
@pytest.mark.parametrize("seed", range(4))
def test_samples_cut_inside_a_run(dsss, orc, ctx, p, seed):
    """The merge-sort path cuts samples to 200 (avg + 5) bytes.  Two PEs hold
    only prefixes, around that length, of one long string, the others short
    strings: a splitter then is a cut prefix that equals none, one or several
    strings, with longer ones behind them."""
    rng = np.random.default_rng(seed)
    head = b"M" + bytes(rng.integers(65, 91, 3000).astype(np.uint8))
    short = [bytes(rng.integers(65, 91, 6).astype(np.uint8)) for _ in range(30000)]
    probe = dsss.from_bytes_list([head[:1700]] * 20 + short)
    pb = np.concatenate([[0, 10, 20], 20 + np.arange(1, p - 1) * 30000 // (p - 2)]).astype(np.uint64)
    avg = orc.ms_sort(orc.Strings.from_host(probe), pb)["avg_lcp"]
    cut = 200 * (avg + 5)
    long = [head[:cut + int(d)] for d in rng.choice([-40, -1, 0, 0, 1, 1, 30, 200], 20)]
    hs = dsss.from_bytes_list(long + short)
    out = dsss.ms_sort(ctx, dsss.DeviceStrings(hs), p, part_begin=pb)
    assert out["avg_lcp"] == avg
    check_ms(dsss, orc, hs, out, pb)


@pytest.mark.parametrize("n,parts", [
    (1, [0, 1]), (2, [0, 1, 2]), (31, [0, 31]), (2048, [0, 1024, 2048]), (2049, [0, 2, 4, 2049]),
    (4500, [0, 2, 2, 5, 4500]), (6200, [0, 1, 3, 40, 3000, 6200]), (6200, None),
], ids=str)
def test_sum_of_local_lcps(dsss, orc, ctx, n, parts):
    """The average local LCP comes from the global LCPs, tile by tile: PEs
    with two strings many tiles apart, with none in most tiles and with all of
    them.  LCPs are longer than n, so that one wrong pair changes the average."""
    rng = np.random.default_rng(n)
    head = b"h" * (n + 50)
    strs = [head + bytes(rng.integers(65, 91, 12).astype(np.uint8)) for _ in range(n)]
    rng.shuffle(strs)
    pb = dsss.equal_parts(n, 37) if parts is None else np.array(parts, np.uint64)
    hs = dsss.from_bytes_list(strs)
    out = dsss.ms_sort(ctx, dsss.DeviceStrings(hs), len(pb) - 1, part_begin=pb)
    assert out["avg_lcp"] == orc.ms_sort(orc.Strings.from_host(hs), pb)["avg_lcp"]
