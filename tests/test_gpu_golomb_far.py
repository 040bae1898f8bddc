"""Golomb decoding of a tile whose chunks lie more than 2^32 bits apart: a
block of one value has no chunk, so the headers of millions of such blocks
(512 MB of them here) can lie between two chunks of the same tile.  The block
behind them starts 2^32 bits and a little behind the tile's first staged word:
a place kept in 32 bits would fall back into the staged words."""
import ctypes

import numpy as np
import pytest

from test_gpu_golomb import host

pytestmark = pytest.mark.gpu


def test_chunks_2_32_bits_apart(dsss, orc):
    import torch
    ctx = dsss.Context(0)  # its own: the block table takes gigabytes of scratch and pinned memory
    b = 1 << 20
    rng = np.random.default_rng(11)
    v0 = np.cumsum(rng.integers(0, 2 * b, 4, dtype=np.uint64))
    v1 = np.cumsum(rng.integers(0, 2 * b, 700, dtype=np.uint64))  # a dozen chunks of 1024 bits
    w0, _ = orc.golomb_encode(v0, [4], [b])
    w1, _ = orc.golomb_encode(v1, [700], [b])
    singles = (2**26 - len(w0)) // 3 + 200
    one = torch.tensor([2, 1, 7], dtype=torch.int64, device="cuda")
    words = torch.cat([torch.from_numpy(w0.view(np.int64)).cuda(), one.repeat(singles),
                       torch.from_numpy(w1.view(np.int64)).cuda()])
    # the second block's code bits behind the first one's, both after 3 header words
    assert 0 < (len(w0) + 3 * singles) * 64 - 2**32 < 300 * 1024
    blocks, total = singles + 2, singles + 704
    values = torch.empty(total, dtype=torch.int64, device="cuda")
    counts = np.zeros(blocks, np.uint64)
    n, nb = ctypes.c_uint64(0), ctypes.c_uint32(0)
    dsss.check(dsss.lib().dsss_golomb_decode(ctx.h, words.data_ptr(), words.numel(), values.data_ptr(), total,
                                             ctypes.byref(n), counts.ctypes.data, blocks, ctypes.byref(nb), None))
    assert (n.value, nb.value) == (total, blocks)
    assert counts[0] == 4 and counts[-1] == 700 and (counts[1:-1] == 1).all()
    assert np.array_equal(host(values[:4]), v0)
    assert bool((values[4:-700] == 7).all())
    assert np.array_equal(host(values[-700:]), v1)
    ctx.close()
