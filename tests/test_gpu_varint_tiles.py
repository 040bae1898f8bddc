"""Varint coding in tiles of 4096 values or bytes: sizes at the tiles' edges,
values whose bytes lie on both sides of an edge, buffers that start at any
byte, range boundaries anywhere in a tile, and malformed values at an edge."""
import numpy as np
import pytest
import torch

from test_gpu_varint import values

pytestmark = pytest.mark.gpu


def dev(v):
    return torch.from_numpy(v.astype(np.uint32).view(np.int32)).cuda()


@pytest.mark.parametrize("shift", [0, 1, 7, 15])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 1365, 4095, 4096, 4097, 8192, 50021])
@pytest.mark.parametrize("kind", ["mixed", "one", "five"])
def test_round_trip(dsss, orc, ctx, kind, n, shift):
    v = {"mixed": values(n, n), "one": np.arange(n) % 128, "five": np.arange(n) + 2**32 - n}[kind].astype(np.uint64)
    rng = np.random.default_rng(n)
    cuts = np.sort(rng.integers(0, n + 1, 40))
    ranges = np.diff(np.concatenate([[0], cuts, [n]])).tolist()
    got, per = dsss.varint_encode(ctx, dev(v), ranges)
    want, wper = orc.varint_encode(v, ranges)
    assert np.array_equal(got.cpu().numpy(), want)
    assert np.array_equal(per, wper)
    moved = torch.empty(len(want) + shift + 64, dtype=torch.uint8, device="cuda").fill_(0x85)
    moved[shift:shift + len(want)] = got  # bytes around the stream look like open values
    back = dsss.varint_decode(ctx, moved[shift:shift + len(want)], n)
    assert np.array_equal(back.cpu().numpy().view(np.uint32).astype(np.uint64), v)


@pytest.mark.parametrize("at", [0, 5, 4085, 4090, 4091, 4092, 4095, 4096, 8187, 9000])
def test_malformed_values(dsss, ctx, at):
    ok = np.full(9100, 0x01, np.uint8)
    for bad in ([0x80] * 5 + [0x01], [0xFF] * 4 + [0x1F]):  # six bytes; above 2^32 - 1
        b = ok.copy()
        b[at:at + len(bad)] = bad
        n = int((b < 0x80).sum())
        with pytest.raises(dsss.DsssError):
            dsss.varint_decode(ctx, torch.from_numpy(b).cuda(), n)
        with pytest.raises(dsss.DsssError):
            dsss.varint_decode(ctx, torch.from_numpy(b).cuda(), n + 1)
    b = ok[:at + 1].copy()
    b[at] = 0x81  # cut off
    with pytest.raises(dsss.DsssError):
        dsss.varint_decode(ctx, torch.from_numpy(b).cuda(), at)


@pytest.mark.parametrize("n,nr", [(4096, 1), (4096, 2), (4096, 9000), (12288, 3), (12289, 4), (50021, 20000), (1, 7)])
def test_many_ranges(dsss, orc, ctx, n, nr):
    """More boundaries than tiles (counted per tile) and fewer (one by one),
    boundaries at the tiles' edges and at n among them."""
    v = values(n + nr, n)
    rng = np.random.default_rng(nr)
    cuts = np.sort(np.concatenate([rng.integers(0, n + 1, nr), np.minimum(np.arange(0, n, 4096), n)]))
    ranges = np.diff(np.concatenate([[0], cuts, [n, n]])).tolist()
    got, per = dsss.varint_encode(ctx, dev(v), ranges)
    want, wper = orc.varint_encode(v, ranges)
    assert np.array_equal(got.cpu().numpy(), want)
    assert np.array_equal(per, wper)
