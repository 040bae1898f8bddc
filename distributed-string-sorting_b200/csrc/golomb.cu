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
// Encoding is data-parallel: code lengths, a scan, then every code ORed into
// its words.  A variable-length code is read sequentially; the decoder cuts
// each block's bits into chunks of GB_CHUNK_BITS, reads every chunk from a
// guessed code start and again from where its predecessor's last code ended,
// until no start changes.  The first chunk of a block starts right, so the
// starts are exact once they agree.  A reader that starts inside a code falls
// into step with the codes after some of them (a few for short remainders,
// some hundred for 40-bit ones), so the repetitions run inside a block of
// threads, over 256 chunks in shared memory, and the blocks of threads then
// agree among themselves in two rounds (in the worst case, as many as the
// stream has such tiles).
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

__global__ void k_gb_len(const uint64_t* v, uint64_t n, GbParams P, uint32_t* len, uint32_t* err) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t r = gb_range_of(P.rbeg, P.nranges, i);
    if (i == P.rbeg[r]) {  // the first value of a range is not coded
        len[i] = 0;
        return;
    }
    if (v[i] < v[i - 1]) atomicOr(err, 1u);  // not ascending
    uint64_t q, val;
    uint32_t kk;
    gb_code(P, r, v[i] - v[i - 1], q, val, kk);
    if (q > GB_MAX_Q) {
        atomicOr(err, 2u);
        len[i] = 0;
        return;
    }
    len[i] = (uint32_t)(q + 1 + kk);
}

// Bits and words of every range's block (0 words for an empty range).
__global__ void k_gb_range_words(const uint64_t* pos, uint64_t n, const uint64_t* total, GbParams P, uint64_t* rbits,
                                 uint64_t* rwords) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= P.nranges) return;
    const uint64_t b0 = P.rbeg[r], b1 = P.rbeg[r + 1];
    if (b1 == b0) {
        rbits[r] = 0;
        rwords[r] = 0;
        return;
    }
    const uint64_t bits = (b1 < n ? pos[b1] : *total) - pos[b0];
    rbits[r] = bits;
    rwords[r] = 3 + (bits + 63) / 64;
}

// Ones over bits [t, t + q) of w (bit 0 = the first word's most significant).
__device__ __forceinline__ void gb_ones(unsigned long long* w, uint64_t t, uint64_t q) {
    if (q == 0) return;
    const uint64_t e = t + q - 1;
    const uint64_t w0 = t >> 6, w1 = e >> 6;
    const uint32_t a = (uint32_t)(t & 63), z = (uint32_t)(e & 63);
    if (w0 == w1) {
        atomicOr(&w[w0], (~0ull >> a) & (~0ull << (63 - z)));
        return;
    }
    atomicOr(&w[w0], ~0ull >> a);
    for (uint64_t x = w0 + 1; x < w1; ++x) w[x] = ~0ull;  // words wholly inside one code
    atomicOr(&w[w1], ~0ull << (63 - z));
}

// The nb (1..64) low bits of val at bits [t, t + nb), most significant first.
__device__ __forceinline__ void gb_bits(unsigned long long* w, uint64_t t, uint64_t val, uint32_t nb) {
    const uint32_t a = (uint32_t)(t & 63);
    const uint64_t x = t >> 6;
    if (a + nb <= 64) {
        atomicOr(&w[x], (unsigned long long)(val << (64 - a - nb)));
    } else {
        const uint32_t second = a + nb - 64;
        atomicOr(&w[x], (unsigned long long)(val >> second));
        atomicOr(&w[x + 1], (unsigned long long)(val << (64 - second)));
    }
}

__global__ void k_gb_write(const uint64_t* v, uint64_t n, GbParams P, const uint64_t* pos, const uint64_t* woff,
                           unsigned long long* out) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t r = gb_range_of(P.rbeg, P.nranges, i);
    const uint64_t b0 = P.rbeg[r];
    if (i == b0) return;
    unsigned long long* w = out + woff[r] + 3;
    uint64_t t = pos[i] - pos[b0];
    uint64_t q, val;
    uint32_t kk;
    gb_code(P, r, v[i] - v[i - 1], q, val, kk);
    if (q > GB_MAX_Q) return;
    gb_ones(w, t, q);
    t += q + 1;  // the zero is already there
    if (kk) gb_bits(w, t, val, kk);
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
constexpr uint32_t GB_STAGE = GB_TILE * (GB_CHUNK_BITS / 64) + 3 * GB_TILE + 2;
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
        uint64_t q = 0;
        for (;;) {
            const uint32_t ones = (uint32_t)__clzll(~peek(t));
            t += ones;
            q += ones;
            if (t >= bit1) return false;
            if (ones < 64) break;
        }
        ++t;  // the zero
        uint64_t r = 0;
        if (k) {
            const uint32_t lo = k - 1;
            const uint64_t v = peek(t);
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
// thread's reader; cs, ce: the thread's chunk (cs = ce: none).  Returns its
// block's number.
__device__ __forceinline__ uint32_t gb_stage(const unsigned long long* w, uint64_t nwords, const GbBlock* blk,
                                             uint32_t nb, uint32_t nch, uint32_t* sw, GbReader& R,
                                             uint64_t& cs, uint64_t& ce) {
    __shared__ unsigned long long s_range[2];
    const uint32_t c0 = blockIdx.x * GB_TILE, c = c0 + threadIdx.x, cl = min(nch, c0 + GB_TILE) - 1;
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
        if (c == c0) s_range[0] = cs >> 6;
        if (c == cl) s_range[1] = min((ce + 63) / 64 + 2, nwords);
    }
    __syncthreads();
    R.w0 = s_range[0];
    R.w1 = min((uint64_t)s_range[1], R.w0 + GB_STAGE);
    for (uint32_t i = threadIdx.x; i < (uint32_t)(R.w1 - R.w0); i += GB_TILE) {
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
// codes (20 chunks of 40-bit codes), far less than a tile, so two rounds
// settle the stream.  (Rounds over the whole stream, each re-reading every
// chunk, took 21 launches of 0.5 ms for 4e6 hashes, 20.5 of the 29 ms of a
// there-and-back.)  Bound by the instructions per code and round: where b is a
// power of two a code's length is its unary part plus a constant, so the
// repetitions read one funnel-shifted word per code and no remainder (1.08 ->
// 0.31 ms for the four launches); counts and gap sums are taken once, at the
// end.
__global__ void __launch_bounds__(GB_TILE) k_gb_walk(const unsigned long long* w, uint64_t nwords, const GbBlock* blk,
                                                     uint32_t nb, uint32_t nch, int round, const uint64_t* end_in,
                                                     uint64_t* end_out, uint64_t* g, uint32_t* cnt,
                                                     unsigned long long* sum, uint32_t* changed) {
    extern __shared__ __align__(16) uint32_t gb_sm[];
    __shared__ unsigned long long e[GB_TILE];
    const uint32_t c0 = blockIdx.x * GB_TILE, c = c0 + threadIdx.x;
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
    const uint32_t j = gb_stage(w, nwords, blk, nb, nch, gb_sm, R, cs, ce);
    const bool valid = c < nch;
    const bool chained = valid && threadIdx.x > 0 && blk[j].chunk0 != c;  // starts where the thread before stopped
    uint64_t start = valid ? (round ? g[c] : cs) : 0;
    if (round && threadIdx.x == 0) start = end_in[blockIdx.x - 1];
    // the codes a repetition can step over by their unary part alone: b a
    // power of two, the word read and the code's end inside the block
    const uint64_t o = R.w0 * 64;
    uint32_t lim = 0;
    if (valid && R.little == 0) {
        const uint64_t staged = (R.w1 - R.w0) * 64, left = R.bit1 - o;
        const uint64_t room = min(staged, left);
        if (room > 64ull + R.k + 33) lim = (uint32_t)(room - 64 - R.k - 33);
    }
    bool redo = valid;
    uint64_t t = start;
    for (;;) {
        if (redo) {
            t = start;
            while (t < ce) {
                const uint32_t u = (uint32_t)(t - o);  // t >= cs >= o: a chunk's codes start inside it
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
            }
            e[threadIdx.x] = t;
        }
        __syncthreads();
        redo = chained && e[threadIdx.x - 1] != start;
        if (redo) start = e[threadIdx.x - 1];
        if (!__syncthreads_or(redo)) break;
    }
    uint32_t m = 0;
    unsigned long long s = 0;
    if (valid) {
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
    if (!valid) return;
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
    const uint32_t j = gb_stage(w, nwords, blk, nb, nch, gb_sm, R, cs, ce);
    const uint32_t c = blockIdx.x * GB_TILE + threadIdx.x;
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
    const uint64_t N = n ? n : 1, R = nranges ? nranges : 1;
    auto plan = [&](Carve& c, uint32_t*& len, uint64_t*& pos, uint64_t*& tot, void*& scan, uint64_t*& prm,
                    uint32_t*& pk, uint64_t*& rbits, uint64_t*& rw, uint64_t*& woff, uint32_t*& err) {
        len = c.take<uint32_t>(N);
        pos = c.take<uint64_t>(N);
        tot = c.take<uint64_t>(1);
        scan = c.take<unsigned char>(scan_scratch_bytes(N));
        prm = c.take<uint64_t>(3 * R + 1);  // rbeg, b, little
        pk = c.take<uint32_t>(R);
        rbits = c.take<uint64_t>(R);
        rw = c.take<uint64_t>(R);
        woff = c.take<uint64_t>(R);
        err = c.take<uint32_t>(1);
    };
    uint32_t *len, *pk, *err;
    uint64_t *pos, *tot, *prm, *rbits, *rw, *woff;
    void* scan;
    Carve s0(nullptr);
    plan(s0, len, pos, tot, scan, prm, pk, rbits, rw, woff, err);
    DSSS_TRY(ensure_ws(ctx, s0.used));
    DSSS_TRY(ensure_pin(ctx, 8 * (R + 4)));
    Carve c(ctx->ws);
    plan(c, len, pos, tot, scan, prm, pk, rbits, rw, woff, err);
    uint64_t* pin = (uint64_t*)ctx->pin;
    *out_words = 0;
    if (nranges == 0) return DSSS_OK;
    DSSS_CUDA(cudaMemcpyAsync(prm, rbeg.data(), (nranges + 1) * 8, cudaMemcpyHostToDevice, st));
    DSSS_CUDA(cudaMemcpyAsync(prm + nranges + 1, bb.data(), nranges * 8, cudaMemcpyHostToDevice, st));
    DSSS_CUDA(cudaMemcpyAsync(prm + 2 * nranges + 1, little.data(), nranges * 8, cudaMemcpyHostToDevice, st));
    DSSS_CUDA(cudaMemcpyAsync(pk, kk.data(), nranges * 4, cudaMemcpyHostToDevice, st));
    DSSS_CUDA(cudaMemsetAsync(err, 0, 4, st));
    GbParams P{prm, prm + nranges + 1, prm + 2 * nranges + 1, pk, nranges};
    if (n) {
        DSSS_LAUNCH("k_gb_len", st, k_gb_len<<<grid_for(n, 256), 256, 0, st>>>(values, n, P, len, err));
        DSSS_TRY(exclusive_scan_u32_to_u64(len, pos, n, tot, scan, st));
    } else {
        DSSS_CUDA(cudaMemsetAsync(tot, 0, 8, st));
    }
    DSSS_LAUNCH("k_gb_range_words", st,
                k_gb_range_words<<<grid_for(nranges, 128), 128, 0, st>>>(pos, n, tot, P, rbits, rw));
    DSSS_CUDA(cudaMemcpyAsync(pin, rw, nranges * 8, cudaMemcpyDeviceToHost, st));
    DSSS_CUDA(cudaMemcpyAsync(pin + nranges, err, 4, cudaMemcpyDeviceToHost, st));
    DSSS_CUDA(cudaStreamSynchronize(st));
    const uint32_t e = (uint32_t)(pin[nranges] & 0xFFFFFFFFu);
    if (e & 1u) return fail(DSSS_EINVAL, "the values of a range must be ascending");
    if (e & 2u) return fail(DSSS_EINVAL, "a gap needs more than 2^31 unary bits (b too small for the values)");
    std::vector<uint64_t> wo(nranges);
    uint64_t total = 0;
    for (uint32_t r = 0; r < nranges; ++r) {
        range_words[r] = pin[r];
        wo[r] = total;
        total += pin[r];
    }
    *out_words = total;
    if (!out) return DSSS_OK;  // size query
    if (total > out_cap) return fail(DSSS_EINVAL, "out_cap %llu below the %llu coded words",
                                     (unsigned long long)out_cap, (unsigned long long)total);
    if (total == 0) return DSSS_OK;
    DSSS_CUDA(cudaMemcpyAsync(woff, wo.data(), nranges * 8, cudaMemcpyHostToDevice, st));
    DSSS_CUDA(cudaMemsetAsync(out, 0, total * 8, st));
    unsigned long long* o = (unsigned long long*)out;
    if (n) DSSS_LAUNCH("k_gb_write", st, k_gb_write<<<grid_for(n, 256), 256, 0, st>>>(values, n, P, pos, woff, o));
    DSSS_LAUNCH("k_gb_head", st, k_gb_head<<<grid_for(nranges, 128), 128, 0, st>>>(values, P, rbits, rw, woff, o));
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
        uint32_t* pin = (uint32_t*)ctx->pin;
        DSSS_CUDA(cudaMemcpyAsync(pin, dnb, 8, cudaMemcpyDeviceToHost, st));
        DSSS_CUDA(cudaStreamSynchronize(st));
        nb = pin[0];
        if (pin[1] & 1u) return fail(DSSS_EINVAL, "a Golomb block runs past the buffer, is too short or has b = 0");
        if (pin[1] & 2u) return fail(DSSS_EINVAL, "more than max_blocks = %u blocks", max_blocks);
        blk.resize(4ull * nb);
        uint64_t* pin64 = (uint64_t*)ctx->pin;
        DSSS_CUDA(cudaMemcpyAsync(pin64, dblk, 32ull * nb, cudaMemcpyDeviceToHost, st));
        DSSS_CUDA(cudaStreamSynchronize(st));
        std::copy(pin64, pin64 + 4ull * nb, blk.begin());
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
    if (nch) {
        // 3. read the tiles until no tile stops elsewhere (each round settles
        // at least one more tile of every block)
        bool settled = false;
        for (uint32_t round = 0; round <= tiles + 1 && !settled; ++round) {
            if (round > 1) DSSS_CUDA(cudaMemsetAsync(flags, 0, 4, st));
            DSSS_LAUNCH("k_gb_walk", st,
                        k_gb_walk<<<tiles, GB_TILE, GB_SMEM, st>>>(w, nwords, dblk, nb, nch, (int)round,
                                                                  end[(round & 1) ^ 1], end[round & 1], g, cnt, sum,
                                                                  flags));
            if (round == 0) continue;
            DSSS_CUDA(cudaGetLastError());
            DSSS_CUDA(cudaMemcpyAsync(pin, flags, 4, cudaMemcpyDeviceToHost, st));
            DSSS_CUDA(cudaStreamSynchronize(st));
            settled = pin[0] == 0;
        }
        if (!settled) return fail(DSSS_EDEVICE, "Golomb chunk starts did not settle");
    }
    // 4. output places: each block's first value, then its chunks' codes
    if (nch)
        DSSS_LAUNCH("k_gb_prefix", st,
                    k_gb_prefix<<<tiles, GB_TILE, 0, st>>>(nch, cnt, sum, pcnt, psum, tcnt, tsum, flags + 1));
    DSSS_LAUNCH("k_gb_tiles", st, k_gb_tiles<<<1, GB_TILE, 0, st>>>(tiles, tcnt, tsum, bcnt, bsum));
    DSSS_LAUNCH("k_gb_starts", st,
                k_gb_starts<<<grid_for(nb + 1, 128), 128, 0, st>>>(dblk, nb, nch, tiles, bcnt, bsum, pcnt, psum, ocnt,
                                                                  osum));
    DSSS_CUDA(cudaGetLastError());
    DSSS_CUDA(cudaMemcpyAsync(pin64, ocnt, (nb + 1) * 8, cudaMemcpyDeviceToHost, st));
    DSSS_CUDA(cudaMemcpyAsync(pin, flags, 8, cudaMemcpyDeviceToHost, st));
    DSSS_CUDA(cudaStreamSynchronize(st));
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
