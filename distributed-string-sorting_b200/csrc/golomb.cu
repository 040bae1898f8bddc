// Golomb/delta coding of sorted 64-bit values: the wire format of the
// reference's hash exchange with sequentialGolombEncoding
// (AllToAllHashesGolomb, src/sorter/distributed/bloomfilter.hpp:164-313, over
// getDeltaEncoding / getDeltaDecoding, src/encoding/golomb_encoding.hpp:50-110,
// and thrill's Golomb bit streams, src/encoding/golomb_bit_stream.hpp,
// bit_stream.hpp, delta_stream.hpp).  A destination with c > 0 values gets
// the block [S, b, v_0, bit words], S the number of words after S; the bit
// words hold, most significant bit first, the code of every gap
// v_i - v_{i-1}: q = gap / b ones, a zero, and r = gap mod b in truncated
// binary (k = ceil(log2 b) bits holding r + 2^k - b when r >= 2^k - b, else
// k - 1 bits holding r); the last word's unused bits are ones.  A destination
// without values gets no words.
//
// Encoding is data-parallel: code lengths summed per tile of values, a scan of
// the tiles, then each thread puts the codes of its consecutive values together
// word by word; the words it shares with its neighbours are ORed in.  A
// variable-length code is read sequentially; the decoder cuts each block's bits
// into chunks of GB_CHUNK_BITS, reads every chunk from a guessed code start and
// again from where its predecessor's last code ended, until no start changes.
// The first chunk of a block starts right, so the starts are exact once they
// agree.  A reader that starts inside a code falls into step with the codes
// after some of them (a few for short remainders, some hundred for 40-bit
// ones), so the repetitions run inside a block of threads, over 256 chunks in
// shared memory, and the blocks of threads then agree among themselves in two
// rounds (in the worst case, as many as the stream has such tiles).
#include <algorithm>
#include <cmath>
#include <vector>

#include "internal.cuh"

namespace dsss {

constexpr uint64_t GB_CHUNK_BITS = 1024;
constexpr uint64_t GB_MAX_Q = 1ull << 31;  // longest unary part coded (a gap of 2^31 b)

static uint32_t gb_ceil_log2(uint64_t b) {  // tlx::integer_log2_ceil
    uint32_t k = 0;
    while (k < 64 && (1ull << k) < b) ++k;
    return k;
}

// Range of value i: the last r with rbeg[r] <= i (empty ranges share their
// start with the next range, which is the one that holds i).
__device__ __forceinline__ uint32_t gb_range_of(const uint64_t* rbeg, uint32_t nranges, uint64_t i) {
    uint32_t lo = 0, hi = nranges;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (rbeg[mid] <= i) lo = mid;
        else hi = mid;
    }
    return lo;
}

struct GbParams {
    const uint64_t* rbeg;  // nranges + 1 value indices
    const uint64_t* b;
    const uint64_t* little;  // 2^k - b
    const uint32_t* k;
    uint32_t nranges;
};

__device__ __forceinline__ void gb_code(const GbParams& P, uint32_t r, uint64_t gap, uint64_t& q, uint64_t& val,
                                        uint32_t& kk) {
    const uint64_t b = P.b[r], little = P.little[r];
    const uint32_t k = P.k[r];
    if (little == 0) {  // b = 2^k
        q = gap >> k;   // k <= 63
        val = gap & (b - 1);
        kk = k;
        return;
    }
    q = gap / b;
    const uint64_t rem = gap - q * b;
    if (rem >= little) {
        val = rem + little;
        kk = k;
    } else {
        val = rem;
        kk = k - 1;
    }
}

constexpr uint32_t GE_NT = 256, GE_IPT = 8, GE_TILE = GE_NT * GE_IPT;  // values of an encoder's tile

// Length of value i's code in range r; the first value of a range is not
// coded.  err bit 1: not ascending, bit 2: too long.
__device__ __forceinline__ uint32_t gb_code_len(const uint64_t* v, uint64_t i, const GbParams& P, uint32_t r, uint32_t* err) {
    if (i == P.rbeg[r]) return 0;
    const uint64_t x = v[i], y = v[i - 1];
    if (x < y && err) atomicOr(err, 1u);
    uint64_t q, val;
    uint32_t kk;
    gb_code(P, r, x - y, q, val, kk);
    if (q > GB_MAX_Q) {
        if (err) atomicOr(err, 2u);
        return 0;
    }
    return (uint32_t)(q + 1 + kk);
}

// Sum over the block; every thread gets it.
__device__ __forceinline__ uint64_t gb_block_sum(uint64_t x) {
    __shared__ uint64_t ws[GE_NT / 32];
#pragma unroll
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = x;
    __syncthreads();
    uint64_t t = 0;
#pragma unroll
    for (uint32_t q = 0; q < GE_NT / 32; ++q) t += ws[q];
    return t;
}

// Code bits of each tile of values.  Most tiles lie in one range, whose search
// then is the tile's.  (Lengths and their positions of every value, 64-bit
// divisions where b is a power of two and an OR per code: 4e6 hashes to 23 MB
// 0.22 ms with the size query, now 0.13.)
__global__ void __launch_bounds__(GE_NT) k_gb_len(const uint64_t* v, uint64_t n, GbParams P, uint64_t* bits, uint32_t* err) {
    const uint64_t tb = (uint64_t)blockIdx.x * GE_TILE;
    const uint32_t r0 = gb_range_of(P.rbeg, P.nranges, tb), r1 = gb_range_of(P.rbeg, P.nranges, min(n, tb + GE_TILE) - 1);
    uint64_t s = 0;
#pragma unroll
    for (uint32_t j = 0; j < GE_IPT; ++j) {
        const uint64_t i = tb + j * GE_NT + threadIdx.x;
        if (i < n) s += gb_code_len(v, i, P, r0 == r1 ? r0 : gb_range_of(P.rbeg, P.nranges, i), err);
    }
    s = gb_block_sum(s);
    if (threadIdx.x == 0) bits[blockIdx.x] = s;
}

// One block: exclusive sums of the tiles' bits in place; the total behind them.
__global__ void __launch_bounds__(1024) k_gb_scan(uint64_t* bits, uint64_t tiles) {
    __shared__ uint64_t ws[32];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint64_t carry = 0;
    for (uint64_t b = 0; b < tiles; b += 1024) {
        const uint64_t i = b + threadIdx.x, x = i < tiles ? bits[i] : 0ull;
        uint64_t y = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t z = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= (uint32_t)o) y += z;
        }
        if (lane == 31) ws[w] = y;
        __syncthreads();
        uint64_t before = carry;
        for (uint32_t q = 0; q < 32; ++q) {
            if (q < w) before += ws[q];
            carry += ws[q];
        }
        if (i < tiles) bits[i] = before + y - x;
        __syncthreads();
    }
    if (threadIdx.x == 0) bits[tiles] = carry;
}

// Bits before each range (and behind the last): its tile's and those of the
// values in the tile before it.  A block per range.
__global__ void __launch_bounds__(GE_NT) k_gb_range_bits(const uint64_t* v, uint64_t n, GbParams P, const uint64_t* bits,
                                                       uint64_t tiles, uint64_t* rpos) {
    const uint32_t r = blockIdx.x;
    const uint64_t e = P.rbeg[r];
    uint64_t s = 0;
    if (e < n)
        for (uint64_t i = e / GE_TILE * GE_TILE + threadIdx.x; i < e; i += GE_NT)
            s += gb_code_len(v, i, P, gb_range_of(P.rbeg, P.nranges, i), nullptr);
    s = gb_block_sum(s);
    if (threadIdx.x == 0) rpos[r] = e < n ? bits[e / GE_TILE] + s : bits[tiles];
}

// The same with more ranges than tiles: a block per tile scans its values once
// and serves every range that starts there (the last tile also those at n).
__global__ void __launch_bounds__(GE_NT) k_gb_range_bits_tiled(const uint64_t* v, uint64_t n, GbParams P,
                                                               const uint64_t* bits, uint64_t tiles, uint64_t* rpos) {
    __shared__ uint64_t pre[GE_TILE], ws[GE_NT / 32];
    const uint64_t tb = (uint64_t)blockIdx.x * GE_TILE, i0 = tb + threadIdx.x * GE_IPT;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t len[GE_IPT];
    uint64_t sum = 0;
#pragma unroll
    for (uint32_t j = 0; j < GE_IPT; ++j) {
        len[j] = i0 + j < n ? gb_code_len(v, i0 + j, P, gb_range_of(P.rbeg, P.nranges, i0 + j), nullptr) : 0u;
        sum += len[j];
    }
    uint64_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    uint64_t t = bits[blockIdx.x] + x - sum;
    for (uint32_t q = 0; q < w; ++q) t += ws[q];
#pragma unroll
    for (uint32_t j = 0; j < GE_IPT; ++j) {
        pre[threadIdx.x * GE_IPT + j] = t;
        t += len[j];
    }
    __syncthreads();
    const uint32_t lo = first_at_least(P.rbeg, P.nranges + 1, tb);
    const uint32_t hi = blockIdx.x + 1 == tiles ? P.nranges + 1 : first_at_least(P.rbeg, P.nranges + 1, tb + GE_TILE);
    for (uint32_t r = lo + threadIdx.x; r < hi; r += GE_NT) {
        const uint64_t e = P.rbeg[r];
        rpos[r] = e < n ? pre[e - tb] : bits[tiles];
    }
}

// Appends bits to a zeroed stream, most significant first: a word that the
// writer fills from its first bit is stored, the others are ORed in.
struct GbWriter {
    unsigned long long* w;
    uint64_t acc;
    uint32_t a;   // bits of the current word before the next one
    bool shared;  // the current word's first bits are another's
    __device__ __forceinline__ void open(unsigned long long* words, uint64_t t) {
        w = words + (t >> 6);
        a = (uint32_t)(t & 63);
        acc = 0;
        shared = a != 0;
    }
    __device__ __forceinline__ void next() {
        if (shared) atomicOr(w, (unsigned long long)acc);
        else *w = acc;
        ++w;
        acc = 0;
        a = 0;
        shared = false;
    }
    // the nb (1..64) low bits of x, which has no others
    __device__ __forceinline__ void put(uint64_t x, uint32_t nb) {
        if (a + nb < 64) {
            acc |= x << (64 - a - nb);
            a += nb;
            return;
        }
        const uint32_t rest = a + nb - 64;  // 0..63
        acc |= x >> rest;
        next();
        if (rest) acc = x << (64 - rest);
        a = rest;
    }
    __device__ __forceinline__ void close() {
        if (acc) atomicOr(w, (unsigned long long)acc);
    }
};

__global__ void __launch_bounds__(GE_NT) k_gb_write(const uint64_t* v, uint64_t n, GbParams P, const uint64_t* bits,
                                                    const uint64_t* rpos, const uint64_t* woff, unsigned long long* out) {
    __shared__ uint64_t ws[GE_NT / 32];
    const uint64_t i0 = (uint64_t)blockIdx.x * GE_TILE + threadIdx.x * GE_IPT;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t r = i0 < n ? gb_range_of(P.rbeg, P.nranges, i0) : 0u;
    const uint32_t r0 = r;
    uint64_t sum = 0;
    for (uint32_t j = 0; j < GE_IPT && i0 + j < n; ++j) {
        while (i0 + j >= P.rbeg[r + 1]) ++r;  // (ranges without values too)
        sum += gb_code_len(v, i0 + j, P, r, nullptr);
    }
    uint64_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    uint64_t t = bits[blockIdx.x] + x - sum;
    for (uint32_t q = 0; q < w; ++q) t += ws[q];
    if (i0 >= n) return;
    r = r0;
    GbWriter W;
    W.open(out + woff[r] + 3, t - rpos[r]);
    for (uint32_t j = 0; j < GE_IPT && i0 + j < n; ++j) {
        const uint64_t i = i0 + j;
        if (i >= P.rbeg[r + 1]) {
            W.close();
            while (i >= P.rbeg[r + 1]) ++r;
            W.open(out + woff[r] + 3, 0);
        }
        if (i == P.rbeg[r]) continue;
        uint64_t q, val;
        uint32_t kk;
        gb_code(P, r, v[i] - v[i - 1], q, val, kk);
        if (q > GB_MAX_Q) continue;  // (an error by now)
        for (; q >= 64; q -= 64) W.put(~0ull, 64);
        W.put((2ull << q) - 2, (uint32_t)q + 1);  // q ones, a zero
        if (kk) W.put(val, kk);
    }
    W.close();
}

// Header words and the ones after the last code (after k_gb_write).
__global__ void k_gb_head(const uint64_t* v, GbParams P, const uint64_t* rbits, const uint64_t* rwords,
                          const uint64_t* woff, unsigned long long* out) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= P.nranges || rwords[r] == 0) return;
    unsigned long long* w = out + woff[r];
    w[0] = rwords[r] - 1;
    w[1] = P.b[r];
    w[2] = v[P.rbeg[r]];
    const uint64_t bits = rbits[r];
    if (bits & 63) w[3 + bits / 64] |= ~0ull >> (bits & 63);
}

// ---------------------------------------------------------------- decode ----
// Block table: one thread follows the S words.  blk[4j..4j+3] = (position,
// S, b, first value) of block j; *nb the blocks; err bit 1: a block runs past the
// buffer, is too short or has b = 0; bit 2: more than max_blocks blocks.
__global__ void k_gb_blocks(const unsigned long long* w, uint64_t nwords, uint32_t max_blocks, uint64_t* blk,
                            uint32_t* nb, uint32_t* err) {
    uint64_t pos = 0;
    uint32_t j = 0;
    while (pos < nwords) {
        if (j >= max_blocks) {
            atomicOr(err, 2u);
            break;
        }
        const uint64_t S = w[pos];
        if (S < 2 || S > nwords - pos - 1 || w[pos + 1] == 0) {
            atomicOr(err, 1u);
            break;
        }
        blk[4 * j] = pos;
        blk[4 * j + 1] = S;
        blk[4 * j + 2] = w[pos + 1];
        blk[4 * j + 3] = w[pos + 2];
        ++j;
        pos += 1 + S;
    }
    *nb = j;
}

// One block of the stream, as the chunk kernels use it.
struct GbBlock {
    uint64_t bit0, bit1;  // its code bits
    uint64_t b, little;
    uint64_t first;       // its uncoded first value
    uint32_t chunk0;      // its first chunk (chunk0 of entry nb: all chunks)
    uint32_t k;
};

// A tile is GB_TILE consecutive chunks, one thread each; its words (and the
// headers of the blocks that end inside it) are staged in shared memory as
// 32-bit halves in stream order, one half of padding per 32 so that threads at
// the same place of their chunks read different banks.
constexpr uint32_t GB_TILE = 256;
constexpr uint32_t GB_CUT = 1u << 31;  // in a chunk's count: its last code is cut off by the block's end
constexpr uint32_t GB_WARM = 32;  // chunks before the tile that its first reading runs in over
constexpr uint32_t GB_STAGE = (GB_TILE + GB_WARM) * (GB_CHUNK_BITS / 64 + 3) + 2;
__device__ __forceinline__ uint32_t gb_skew(uint32_t i) { return i + (i >> 5); }
constexpr size_t GB_SMEM = (size_t)(2 * GB_STAGE + GB_STAGE / 16 + 2) * 4;

struct GbReader {
    const unsigned long long* w;   // the stream
    const uint32_t* sw;            // words [w0, w1) of it, staged
    uint64_t w0, w1, nwords, bit1;
    uint64_t b, little;
    uint32_t k;
    __device__ __forceinline__ uint64_t word(uint64_t x) const {
        if (x >= w0 && x < w1) {
            const uint32_t i = 2 * (uint32_t)(x - w0);
            return (uint64_t)sw[gb_skew(i)] << 32 | sw[gb_skew(i + 1)];
        }
        return x < nwords ? w[x] : 0ull;
    }
    // The 64 bits from bit t on, 0 past the block's end.
    __device__ __forceinline__ uint64_t peek(uint64_t t) const {
        if (t >= bit1) return 0;
        const uint32_t a = (uint32_t)(t & 63);
        const uint64_t x = t >> 6;
        uint64_t v = word(x) << a;
        if (a) v |= word(x + 1) >> (64 - a);
        const uint64_t left = bit1 - t;
        if (left < 64) v &= ~0ull << (64 - left);
        return v;
    }
    // Reads the code at t (t < bit1).  Returns false at the stream's end (only
    // ones up to bit1: the padding); else sets the gap and moves t past the
    // code (t > bit1: the code is cut off).
    __device__ __forceinline__ bool read(uint64_t& t, uint64_t& gap) const {
        uint64_t v = peek(t);
        uint32_t ones = (uint32_t)__clzll(~v);
        if (ones + 1 + k <= 64) {  // the whole code, or the stream's end, in one word
            if (t + ones >= bit1) return false;
            t += ones + 1;
            uint64_t r = 0;
            if (k) {
                const uint32_t lo = k - 1;
                v <<= ones + 1;
                if (lo) r = v >> (64 - lo);
                t += lo;
                if (r >= little) {
                    r = ((r << 1) | ((v << lo) >> 63)) - little;
                    ++t;
                }
            }
            gap = ones * b + r;
            return true;
        }
        uint64_t q = 0;
        for (bool zero = ones < 64;;) {
            t += ones;
            q += ones;
            if (t >= bit1) return false;
            if (zero) break;
            const uint32_t left = 64 - (uint32_t)(t & 63);  // to the word's end; a block ends with a word
            ones = min((uint32_t)__clzll(~(word(t >> 6) << (64 - left))), left);
            zero = ones < left;
        }
        ++t;  // the zero
        uint64_t r = 0;
        if (k) {
            const uint32_t lo = k - 1;
            v = peek(t);
            if (lo) r = v >> (64 - lo);
            t += lo;
            if (r >= little) {
                r = ((r << 1) | ((v << lo) >> 63)) - little;
                ++t;
            }
        }
        gap = q * b + r;
        return true;
    }
};

// Chunk c: its block (the last j with chunk0 <= c) and its bits [cs, ce).
__device__ __forceinline__ uint32_t gb_chunk(const GbBlock* blk, uint32_t nb, uint32_t c, uint64_t& cs, uint64_t& ce) {
    uint32_t lo = 0, hi = nb;
    while (hi - lo > 1) {
        const uint32_t m = (lo + hi) >> 1;
        if (blk[m].chunk0 <= c) lo = m;
        else hi = m;
    }
    cs = blk[lo].bit0 + (uint64_t)(c - blk[lo].chunk0) * GB_CHUNK_BITS;
    ce = min(cs + GB_CHUNK_BITS, blk[lo].bit1);
    return lo;
}

// Stages the tile's words (the block's threads together) and sets up each
// thread's reader for its chunk c (none from nch on); cs, ce: the chunk's bits.
// The chunks staged are [first, nch or the tile's end).  Returns its block's
// number.
__device__ __forceinline__ uint32_t gb_stage(const unsigned long long* w, uint64_t nwords, const GbBlock* blk,
                                             uint32_t nb, uint32_t nch, uint32_t* sw, GbReader& R, uint32_t c,
                                             uint32_t first, uint64_t& cs, uint64_t& ce) {
    __shared__ unsigned long long s_range[2];
    const uint32_t cl = min(nch, blockIdx.x * GB_TILE + GB_TILE) - 1;
    uint32_t j = 0xFFFFFFFFu;
    cs = ce = 0;
    R.w = w;
    R.sw = sw;
    R.nwords = nwords;
    R.bit1 = 0;
    R.b = 1;
    R.little = 0;
    R.k = 0;
    if (c < nch) {
        j = gb_chunk(blk, nb, c, cs, ce);
        R.bit1 = blk[j].bit1;
        R.b = blk[j].b;
        R.little = blk[j].little;
        R.k = blk[j].k;
        if (c == first) s_range[0] = cs >> 6;
        if (c == cl) s_range[1] = min((ce + 63) / 64 + 2, nwords);
    }
    __syncthreads();
    R.w0 = s_range[0];
    R.w1 = min((uint64_t)s_range[1], R.w0 + GB_STAGE);
    for (uint32_t i = threadIdx.x; i < (uint32_t)(R.w1 - R.w0); i += blockDim.x) {
        const uint64_t v = w[R.w0 + i];
        sw[gb_skew(2 * i)] = (uint32_t)(v >> 32);
        sw[gb_skew(2 * i + 1)] = (uint32_t)v;
    }
    __syncthreads();
    return j;
}

// One reading of the tiles: every chunk is read from g[c] (round 0: its own
// first bit) and then again from where its predecessor in the block stopped,
// until no start of the tile changes.  A tile's first chunk starts where the
// previous tile stopped in the previous round (end_in); a tile whose start
// holds is left as it is.  cnt, sum: the codes that start in each chunk and
// the sum of their gaps; end_out: where each tile stopped; *changed: some
// tile now stops elsewhere.  A wrong start falls into step after some hundred
// codes (20 chunks of 40-bit codes), so in round 0 another warp reads the
// GB_WARM chunks before the tile in step with it and the tile's own start is
// right already: round 1 then finds nothing to do, and if that ever is not so
// the rounds go on.  (Without that warp every tile was read again in round 1:
// 0.31 ms for the four launches, now 0.25.  Rounds over the whole stream, each
// re-reading every chunk, took 21 launches of 0.5 ms for 4e6 hashes, 20.5 of the
// 29 ms of a there-and-back.)  Bound by the instructions per code and round:
// where b is a power of two a code's length is its unary part plus a constant,
// so the repetitions read one funnel-shifted word per code and no remainder
// (1.08 -> 0.31 ms), and counts and gap sums are taken once, at the end.  Other
// codes are counted as they are read (b = 3, 2000 values there and back: 1.34 ->
// 0.76 ms with one read of 64 bits per code).
__global__ void __launch_bounds__(GB_TILE + GB_WARM) k_gb_walk(const unsigned long long* w, uint64_t nwords, const GbBlock* blk,
                                                     uint32_t nb, uint32_t nch, int round, const uint64_t* end_in,
                                                     uint64_t* end_out, uint64_t* g, uint32_t* cnt,
                                                     unsigned long long* sum, uint32_t* changed) {
    extern __shared__ __align__(16) uint32_t gb_sm[];
    __shared__ unsigned long long e[GB_TILE + GB_WARM];
    // threads GB_TILE on (round 0): the chunks before the tile
    const bool warm = threadIdx.x >= GB_TILE;
    const uint32_t c0 = blockIdx.x * GB_TILE;
    const uint32_t first = round == 0 && c0 ? c0 - GB_WARM : c0;
    const uint32_t c = !warm ? c0 + threadIdx.x : c0 ? c0 - GB_WARM + (threadIdx.x - GB_TILE) : nch;
    if (round) {  // the tile's start: unchanged, or settled since the stream's (or the block's) first bit
        uint64_t cs, ce;
        const uint32_t j = gb_chunk(blk, nb, c0, cs, ce);
        const bool keep = blockIdx.x == 0 || blk[j].chunk0 == c0 || g[c0] == end_in[blockIdx.x - 1];
        if (keep) {  // the same for the whole block
            if (threadIdx.x == 0) end_out[blockIdx.x] = end_in[blockIdx.x];
            return;
        }
    }
    GbReader R;
    uint64_t cs, ce;
    const uint32_t j = gb_stage(w, nwords, blk, nb, nch, gb_sm, R, c, first, cs, ce);
    const bool valid = c < nch;
    const bool chained = valid && c != first && blk[j].chunk0 != c;  // starts where the thread with the chunk before stopped
    const uint32_t before = threadIdx.x ? threadIdx.x - 1 : GB_TILE + GB_WARM - 1;
    uint64_t start = valid ? (round ? g[c] : cs) : 0;
    if (round && threadIdx.x == 0) start = end_in[blockIdx.x - 1];
    // the codes a repetition can step over by their unary part alone: b a
    // power of two, the word read and the code's end inside the block.  Places
    // are 32 bits from the first staged word; blocks of one value have no
    // chunk, and enough of them put a chunk of the tile further off.
    const uint64_t o = R.w0 * 64;
    uint32_t lim = 0;
    if (valid && R.little == 0 && (ce - o) >> 32 == 0) {
        const uint64_t staged = (R.w1 - R.w0) * 64, left = R.bit1 - o;
        const uint64_t room = min(staged, left);
        if (room > 64ull + R.k + 33) lim = (uint32_t)(room - 64 - R.k - 33);
    }
    // without such codes a reading counts as it goes; else the counts and gap
    // sums are taken once, at the end
    const bool counted = lim == 0;
    bool redo = valid;
    uint64_t t = start;
    uint32_t m = 0;
    unsigned long long s = 0;
    for (;;) {
        if (redo) {
            t = start;
            m = 0;
            s = 0;
            while (t < ce) {
                const uint32_t u = (uint32_t)(t - o);  // o <= cs <= t < ce: exact wherever lim is not 0
                if (u < lim) {
                    const uint32_t i = u >> 5;
                    const uint32_t x = __funnelshift_l(gb_sm[gb_skew(i + 1)], gb_sm[gb_skew(i)], u & 31);
                    const uint32_t ones = (uint32_t)__clz(~x);
                    if (ones < 32) {
                        t += ones + 1 + R.k;
                        continue;
                    }
                }
                uint64_t gap;
                if (!R.read(t, gap)) {
                    t = R.bit1;
                    break;
                }
                ++m;
                s += gap;
            }
            e[threadIdx.x] = t;
        }
        __syncthreads();
        redo = chained && e[before] != start;
        if (redo) start = e[before];
        if (!__syncthreads_or(redo)) break;
    }
    if (!valid || warm) return;
    if (!counted && R.k == 0) {  // b = 1: a zero per code, its gap the ones before it
        m = 0;
        uint64_t last = start;  // behind the last zero
        for (uint64_t p = start; p < t; p += 64) {
            uint64_t zeros = ~R.peek(p);
            if (t - p < 64) zeros &= ~0ull << (64 - (t - p));
            m += (uint32_t)__popcll(zeros);
            if (zeros) last = p + 65 - (uint32_t)__ffsll((long long)zeros);
        }
        s = last - start - m;
    } else if (!counted) {
        m = 0;
        s = 0;
        t = start;
        while (t < ce) {
            uint64_t gap;
            if (!R.read(t, gap)) {
                t = R.bit1;
                break;
            }
            ++m;
            s += gap;
        }
    }
    g[c] = start;
    cnt[c] = m | (t > R.bit1 ? GB_CUT : 0u);
    sum[c] = s;
    if (threadIdx.x == GB_TILE - 1 || c + 1 == nch) {
        if (round && t != end_in[blockIdx.x]) *changed = 1;
        end_out[blockIdx.x] = t;
    }
}

// Exclusive scan of (m, s) over the block's threads, and the totals.
__device__ __forceinline__ void gb_block_scan(uint32_t m, unsigned long long s, uint32_t& pm, unsigned long long& ps,
                                              uint32_t& tm, unsigned long long& ts) {
    __shared__ uint32_t wm[GB_TILE / 32];
    __shared__ unsigned long long wsum[GB_TILE / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = m;
    unsigned long long y = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t xx = __shfl_up_sync(0xffffffffu, x, o);
        const unsigned long long yy = __shfl_up_sync(0xffffffffu, y, o);
        if (lane >= o) {
            x += xx;
            y += yy;
        }
    }
    if (lane == 31) {
        wm[w] = x;
        wsum[w] = y;
    }
    __syncthreads();
    pm = x - m;
    ps = y - s;
    tm = 0;
    ts = 0;
    for (int k = 0; k < (int)(GB_TILE / 32); ++k) {
        if (k < w) {
            pm += wm[k];
            ps += wsum[k];
        }
        tm += wm[k];
        ts += wsum[k];
    }
    __syncthreads();
}

// Codes and gap sums before every chunk inside its tile, and the tiles' totals.
__global__ void __launch_bounds__(GB_TILE) k_gb_prefix(uint32_t nch, const uint32_t* cnt, const unsigned long long* sum,
                                                       uint32_t* pcnt, unsigned long long* psum, uint32_t* tcnt,
                                                       unsigned long long* tsum, uint32_t* cut) {
    const uint32_t c = blockIdx.x * GB_TILE + threadIdx.x;
    const uint32_t v = c < nch ? cnt[c] : 0u;
    if (v & GB_CUT) *cut = 1;
    uint32_t pm, tm;
    unsigned long long ps, ts;
    gb_block_scan(v & ~GB_CUT, c < nch ? sum[c] : 0ull, pm, ps, tm, ts);
    if (c < nch) {
        pcnt[c] = pm;
        psum[c] = ps;
    }
    if (threadIdx.x == 0) {
        tcnt[blockIdx.x] = tm;
        tsum[blockIdx.x] = ts;
    }
}

// One block: codes and gap sums before every tile (entry `tiles`: all).
__global__ void __launch_bounds__(GB_TILE) k_gb_tiles(uint32_t tiles, const uint32_t* tcnt,
                                                      const unsigned long long* tsum, uint64_t* bcnt,
                                                      unsigned long long* bsum) {
    uint64_t cm = 0;
    unsigned long long cs = 0;
    for (uint32_t b = 0; b < tiles; b += GB_TILE) {
        const uint32_t i = b + threadIdx.x;
        uint32_t pm, tm;
        unsigned long long ps, ts;
        gb_block_scan(i < tiles ? tcnt[i] : 0u, i < tiles ? tsum[i] : 0ull, pm, ps, tm, ts);
        if (i < tiles) {
            bcnt[i] = cm + pm;
            bsum[i] = cs + ps;
        }
        cm += tm;
        cs += ts;
    }
    if (threadIdx.x == 0) {
        bcnt[tiles] = cm;
        bsum[tiles] = cs;
    }
}

// Codes and gap sums before every block (entry nb: all).
__global__ void k_gb_starts(const GbBlock* blk, uint32_t nb, uint32_t nch, uint32_t tiles, const uint64_t* bcnt,
                            const unsigned long long* bsum, const uint32_t* pcnt, const unsigned long long* psum,
                            uint64_t* ocnt, unsigned long long* osum) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j > nb) return;
    const uint32_t c = j < nb ? blk[j].chunk0 : nch;
    ocnt[j] = c < nch ? bcnt[c / GB_TILE] + pcnt[c] : bcnt[tiles];
    osum[j] = c < nch ? bsum[c / GB_TILE] + psum[c] : bsum[tiles];
}

// The values: block j's uncoded first value goes to ocnt[j] + j, its chunks'
// codes behind it, each the first value plus the gaps up to it.
__global__ void k_gb_firsts(const GbBlock* blk, uint32_t nb, const uint64_t* ocnt, unsigned long long* out) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < nb) out[ocnt[j] + j] = blk[j].first;
}

__global__ void __launch_bounds__(GB_TILE) k_gb_emit(const unsigned long long* w, uint64_t nwords, const GbBlock* blk,
                                                     uint32_t nb, uint32_t nch, const uint64_t* g, const uint64_t* bcnt,
                                                     const unsigned long long* bsum, const uint32_t* pcnt,
                                                     const unsigned long long* psum, const unsigned long long* osum,
                                                     unsigned long long* out) {
    extern __shared__ __align__(16) uint32_t gb_sm[];
    GbReader R;
    uint64_t cs, ce;
    const uint32_t c = blockIdx.x * GB_TILE + threadIdx.x;
    const uint32_t j = gb_stage(w, nwords, blk, nb, nch, gb_sm, R, c, blockIdx.x * GB_TILE, cs, ce);
    if (c >= nch) return;
    uint64_t t = g[c];
    uint64_t o = bcnt[blockIdx.x] + pcnt[c] + j + 1;
    uint64_t run = blk[j].first + (bsum[blockIdx.x] + psum[c] - osum[j]);
    while (t < ce) {
        uint64_t gap;
        if (!R.read(t, gap)) break;
        run += gap;
        out[o++] = run;
    }
}

}  // namespace dsss

using namespace dsss;

extern "C" {

uint64_t dsss_golomb_param(uint64_t max_value, uint64_t count) {
    if (count == 0) return 1;
    const uint64_t avg = max_value / count;
    if (avg < 1) return 1;
    const uint64_t k = (uint64_t)std::floor(std::log2((double)avg));
    return 1ull << k;
}

uint64_t dsss_golomb_param_hashes(uint64_t count, uint32_t p) {
    if (p == 0) return 0;
    const uint64_t b = dsss_golomb_param(~0ull / p, count);
    return b == 1 ? 20000000000ull : b;
}

int dsss_golomb_encode(dsss_ctx* ctx, const uint64_t* values, const uint64_t* range_counts, uint32_t nranges,
                       const uint64_t* b, uint64_t* out, uint64_t out_cap, uint64_t* out_words, uint64_t* range_words,
                       dsss_stream_t stream) {
    if (!ctx) return fail(DSSS_EINVAL, "ctx is NULL");
    ActiveCtx active(ctx);
    if (!out_words || (nranges && (!range_counts || !b || !range_words)))
        return fail(DSSS_EINVAL, "output pointers missing");
    std::vector<uint64_t> rbeg(nranges + 1, 0), little(nranges), bb(nranges);
    std::vector<uint32_t> kk(nranges);
    for (uint32_t r = 0; r < nranges; ++r) {
        if (b[r] == 0) return fail(DSSS_EINVAL, "range %u: the Golomb parameter b must be >= 1", r);
        rbeg[r + 1] = rbeg[r] + range_counts[r];
        bb[r] = b[r];
        kk[r] = gb_ceil_log2(b[r]);
        little[r] = (kk[r] >= 64 ? 0ull : (1ull << kk[r])) - b[r];
    }
    const uint64_t n = rbeg[nranges];
    if (n && !values) return fail(DSSS_EINVAL, "values is NULL");
    DSSS_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t st = (cudaStream_t)stream;
    const uint64_t R = nranges ? nranges : 1, tiles = (n + GE_TILE - 1) / GE_TILE;
    const uint64_t prm_bytes = (3 * R + 1) * 8 + R * 4;  // rbeg, b, 2^k - b, k
    uint64_t *prm, *bits, *rpos, *place;
    uint32_t* err;
    auto plan = [&](Carve& c) {
        prm = (uint64_t*)c.take<unsigned char>(prm_bytes);
        bits = c.take<uint64_t>(tiles + 1);
        rpos = c.take<uint64_t>(R + 2);  // the error flags behind it
        place = c.take<uint64_t>(3 * R);  // the blocks' bits, words and offsets
    };
    Carve s0(nullptr);
    plan(s0);
    DSSS_TRY(ensure_ws(ctx, s0.used));
    const uint64_t prm_words = (prm_bytes + 7) / 8;
    DSSS_TRY(ensure_pin(ctx, (prm_words + 3 * R) * 8 + 64));
    Carve c(ctx->ws);
    plan(c);
    err = (uint32_t*)(rpos + R + 1);
    uint64_t* pin = (uint64_t*)ctx->pin;  // the parameters, then rpos
    uint64_t* at = pin + prm_words;       // place
    *out_words = 0;
    if (nranges == 0) return DSSS_OK;
    std::copy(rbeg.begin(), rbeg.end(), pin);
    std::copy(bb.begin(), bb.end(), pin + R + 1);
    std::copy(little.begin(), little.end(), pin + 2 * R + 1);
    std::copy(kk.begin(), kk.end(), (uint32_t*)(pin + 3 * R + 1));
    DSSS_CUDA(cudaMemcpyAsync(prm, pin, prm_bytes, cudaMemcpyHostToDevice, st));
    DSSS_CUDA(cudaMemsetAsync(rpos, 0, (R + 2) * 8, st));
    GbParams P{prm, prm + R + 1, prm + 2 * R + 1, (const uint32_t*)(prm + 3 * R + 1), nranges};
    if (n) {
        DSSS_LAUNCH("k_gb_len", st, k_gb_len<<<(unsigned)tiles, GE_NT, 0, st>>>(values, n, P, bits, err));
        DSSS_LAUNCH("k_gb_scan", st, k_gb_scan<<<1, 1024, 0, st>>>(bits, tiles));
        if (R + 1 > tiles)
            DSSS_LAUNCH("k_gb_range_bits", st,
                        k_gb_range_bits_tiled<<<(unsigned)tiles, GE_NT, 0, st>>>(values, n, P, bits, tiles, rpos));
        else
            DSSS_LAUNCH("k_gb_range_bits", st,
                        k_gb_range_bits<<<(unsigned)R + 1, GE_NT, 0, st>>>(values, n, P, bits, tiles, rpos));
    }
    DSSS_CUDA(cudaMemcpyAsync(pin, rpos, (R + 2) * 8, cudaMemcpyDeviceToHost, st));
    DSSS_CUDA(cudaStreamSynchronize(st));
    const uint32_t e = (uint32_t)(pin[R + 1] & 0xFFFFFFFFu);
    if (e & 1u) return fail(DSSS_EINVAL, "the values of a range must be ascending");
    if (e & 2u) return fail(DSSS_EINVAL, "a gap needs more than 2^31 unary bits (b too small for the values)");
    // a block's bits, words (0 for an empty range) and offset
    uint64_t total = 0;
    for (uint32_t r = 0; r < nranges; ++r) {
        at[r] = pin[r + 1] - pin[r];
        at[R + r] = range_words[r] = rbeg[r + 1] == rbeg[r] ? 0 : 3 + (at[r] + 63) / 64;
        at[2 * R + r] = total;
        total += range_words[r];
    }
    *out_words = total;
    if (!out) return DSSS_OK;  // size query
    if (total > out_cap) return fail(DSSS_EINVAL, "out_cap %llu below the %llu coded words",
                                     (unsigned long long)out_cap, (unsigned long long)total);
    if (total == 0) return DSSS_OK;
    DSSS_CUDA(cudaMemcpyAsync(place, at, 3 * R * 8, cudaMemcpyHostToDevice, st));
    DSSS_CUDA(cudaMemsetAsync(out, 0, total * 8, st));
    unsigned long long* o = (unsigned long long*)out;
    DSSS_LAUNCH("k_gb_write", st, k_gb_write<<<(unsigned)tiles, GE_NT, 0, st>>>(values, n, P, bits, rpos, place + 2 * R, o));
    DSSS_LAUNCH("k_gb_head", st,
                k_gb_head<<<grid_for(nranges, 128), 128, 0, st>>>(values, P, place, place + R, place + 2 * R, o));
    DSSS_CUDA(cudaGetLastError());
    DSSS_CUDA(cudaStreamSynchronize(st));
    return DSSS_OK;
}

int dsss_golomb_decode(dsss_ctx* ctx, const uint64_t* words, uint64_t nwords, uint64_t* values, uint64_t cap_values,
                       uint64_t* n_values, uint64_t* block_counts, uint32_t max_blocks, uint32_t* nblocks,
                       dsss_stream_t stream) {
    if (!ctx) return fail(DSSS_EINVAL, "ctx is NULL");
    ActiveCtx active(ctx);
    if (!n_values || !nblocks || (max_blocks && !block_counts)) return fail(DSSS_EINVAL, "output pointers missing");
    if (nwords && !words) return fail(DSSS_EINVAL, "words is NULL");
    *n_values = 0;
    *nblocks = 0;
    if (nwords == 0) return DSSS_OK;
    if (max_blocks == 0) return fail(DSSS_EINVAL, "max_blocks is 0 for a non-empty buffer");
    DSSS_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t st = (cudaStream_t)stream;
    const unsigned long long* w = (const unsigned long long*)words;
    // 1. the block table
    {
        Carve s0(nullptr);
        s0.take<uint64_t>(4ull * max_blocks);
        s0.take<uint32_t>(2);
        DSSS_TRY(ensure_ws(ctx, s0.used));
    }
    DSSS_TRY(ensure_pin(ctx, 32ull * max_blocks + 64));
    std::vector<uint64_t> blk;
    uint32_t nb = 0;
    {
        Carve c(ctx->ws);
        uint64_t* dblk = c.take<uint64_t>(4ull * max_blocks);
        uint32_t* dnb = c.take<uint32_t>(2);
        DSSS_CUDA(cudaMemsetAsync(dnb, 0, 8, st));
        DSSS_LAUNCH("k_gb_blocks", st, k_gb_blocks<<<1, 1, 0, st>>>(w, nwords, max_blocks, dblk, dnb, dnb + 1));
        uint64_t* pin64 = (uint64_t*)ctx->pin;
        uint32_t* pin = (uint32_t*)(pin64 + 4ull * max_blocks);
        const uint32_t early = max_blocks <= 1024 ? max_blocks : 0;  // a table that small comes along at once
        if (early) DSSS_CUDA(cudaMemcpyAsync(pin64, dblk, 32ull * early, cudaMemcpyDeviceToHost, st));
        DSSS_CUDA(cudaMemcpyAsync(pin, dnb, 8, cudaMemcpyDeviceToHost, st));
        DSSS_CUDA(cudaStreamSynchronize(st));
        nb = pin[0];
        if (pin[1] & 1u) return fail(DSSS_EINVAL, "a Golomb block runs past the buffer, is too short or has b = 0");
        if (pin[1] & 2u) return fail(DSSS_EINVAL, "more than max_blocks = %u blocks", max_blocks);
        if (!early) {
            DSSS_CUDA(cudaMemcpyAsync(pin64, dblk, 32ull * nb, cudaMemcpyDeviceToHost, st));
            DSSS_CUDA(cudaStreamSynchronize(st));
        }
        blk.assign(pin64, pin64 + 4ull * nb);
    }
    // 2. the blocks with their chunks
    std::vector<GbBlock> hb(nb + 1);
    uint64_t chunks = 0;
    for (uint32_t j = 0; j < nb; ++j) {
        const uint64_t pos = blk[4 * j], S = blk[4 * j + 1], b = blk[4 * j + 2];
        const uint32_t k = gb_ceil_log2(b);
        const uint64_t bit0 = (pos + 3) * 64, bit1 = (pos + 1 + S) * 64;
        hb[j] = GbBlock{bit0, bit1, b, (k >= 64 ? 0ull : (1ull << k)) - b, blk[4 * j + 3], (uint32_t)chunks, k};
        chunks += (bit1 - bit0 + GB_CHUNK_BITS - 1) / GB_CHUNK_BITS;
    }
    hb[nb] = GbBlock{};
    hb[nb].chunk0 = (uint32_t)chunks;
    if (chunks >= (1ull << 32) - GB_TILE) return fail(DSSS_ENOTSUP, "Golomb stream of 2^42 bits or more");
    const uint32_t nch = (uint32_t)chunks, tiles = (nch + GB_TILE - 1) / GB_TILE;
    const uint64_t NC = nch ? nch : 1, NT = (uint64_t)tiles + 1;
    GbBlock* dblk;
    uint64_t *g, *end[2], *bcnt, *ocnt;
    uint32_t *cnt, *pcnt, *tcnt, *flags;
    unsigned long long *sum, *psum, *tsum, *bsum, *osum;
    auto plan = [&](Carve& c) {
        dblk = c.take<GbBlock>(nb + 1);
        g = c.take<uint64_t>(NC);
        cnt = c.take<uint32_t>(NC);
        sum = c.take<unsigned long long>(NC);
        pcnt = c.take<uint32_t>(NC);
        psum = c.take<unsigned long long>(NC);
        end[0] = c.take<uint64_t>(NT);
        end[1] = c.take<uint64_t>(NT);
        tcnt = c.take<uint32_t>(NT);
        tsum = c.take<unsigned long long>(NT);
        bcnt = c.take<uint64_t>(NT);
        bsum = c.take<unsigned long long>(NT);
        ocnt = c.take<uint64_t>(nb + 1);
        osum = c.take<unsigned long long>(nb + 1);
        flags = c.take<uint32_t>(2);  // [0] a tile stopped elsewhere, [1] a code is cut off
    };
    Carve s1(nullptr);
    plan(s1);
    DSSS_TRY(ensure_ws(ctx, s1.used));
    Carve c(ctx->ws);
    plan(c);
    uint64_t* pin64 = (uint64_t*)ctx->pin;  // 32 max_blocks + 64 bytes, nb <= max_blocks
    uint32_t* pin = (uint32_t*)(pin64 + nb + 1);
    DSSS_CUDA(cudaMemcpyAsync(dblk, hb.data(), (nb + 1) * sizeof(GbBlock), cudaMemcpyHostToDevice, st));
    DSSS_CUDA(cudaMemsetAsync(flags, 0, 8, st));
    static std::atomic<uint64_t> walk_configured{0}, emit_configured{0};
    DSSS_TRY(set_smem_once(walk_configured, k_gb_walk, (int)GB_SMEM));
    DSSS_TRY(set_smem_once(emit_configured, k_gb_emit, (int)GB_SMEM));
    // 3. read the tiles until no tile stops elsewhere (each round settles at
    // least one more tile of every block); the output places follow every
    // round from the second on, since that one nearly always is the last:
    // each block's first value, then its chunks' codes
    bool settled = false;
    for (uint32_t round = 0; round <= tiles + 1 && !settled; ++round) {
        if (nch) {
            if (round > 1) DSSS_CUDA(cudaMemsetAsync(flags, 0, 8, st));
            DSSS_LAUNCH("k_gb_walk", st,
                        k_gb_walk<<<tiles, GB_TILE + (round ? 0 : GB_WARM), GB_SMEM, st>>>(w, nwords, dblk, nb, nch, (int)round,
                                                                  end[(round & 1) ^ 1], end[round & 1], g, cnt, sum,
                                                                  flags));
            if (round == 0) continue;
            DSSS_LAUNCH("k_gb_prefix", st,
                        k_gb_prefix<<<tiles, GB_TILE, 0, st>>>(nch, cnt, sum, pcnt, psum, tcnt, tsum, flags + 1));
        }
        DSSS_LAUNCH("k_gb_tiles", st, k_gb_tiles<<<1, GB_TILE, 0, st>>>(tiles, tcnt, tsum, bcnt, bsum));
        DSSS_LAUNCH("k_gb_starts", st,
                    k_gb_starts<<<grid_for(nb + 1, 128), 128, 0, st>>>(dblk, nb, nch, tiles, bcnt, bsum, pcnt, psum,
                                                                      ocnt, osum));
        DSSS_CUDA(cudaGetLastError());
        DSSS_CUDA(cudaMemcpyAsync(pin64, ocnt, (nb + 1) * 8, cudaMemcpyDeviceToHost, st));
        DSSS_CUDA(cudaMemcpyAsync(pin, flags, 8, cudaMemcpyDeviceToHost, st));
        DSSS_CUDA(cudaStreamSynchronize(st));
        settled = nch == 0 || pin[0] == 0;
    }
    if (!settled) return fail(DSSS_EDEVICE, "Golomb chunk starts did not settle");
    if (pin[1]) return fail(DSSS_EINVAL, "a Golomb code is cut off by its block's end");
    const uint64_t total = pin64[nb] + nb;
    for (uint32_t j = 0; j < nb; ++j) block_counts[j] = pin64[j + 1] - pin64[j] + 1;
    *n_values = total;
    *nblocks = nb;
    if (!values) return DSSS_OK;  // size query
    if (total > cap_values) return fail(DSSS_EINVAL, "cap_values %llu below the %llu coded values",
                                        (unsigned long long)cap_values, (unsigned long long)total);
    unsigned long long* out = (unsigned long long*)values;
    DSSS_LAUNCH("k_gb_firsts", st, k_gb_firsts<<<grid_for(nb, 128), 128, 0, st>>>(dblk, nb, ocnt, out));
    if (nch)
        DSSS_LAUNCH("k_gb_emit", st,
                    k_gb_emit<<<tiles, GB_TILE, GB_SMEM, st>>>(w, nwords, dblk, nb, nch, g, bcnt, bsum, pcnt, psum,
                                                              osum, out));
    DSSS_CUDA(cudaGetLastError());
    DSSS_CUDA(cudaStreamSynchronize(st));
    return DSSS_OK;
}

}  // extern "C"
