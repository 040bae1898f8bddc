// K3 — segmented MSD string sort with LCP output, the role radixsort_CI3
// plays per PE in the reference (tlx/sort/strings/radix_sort.hpp:861-884,
// called at src/sorter/distributed/prefix_doubling.hpp:228).
//
// Elements are string ids; every segment is sorted independently (a PE's
// strings, or the whole set).  Large segments (> small_max) are refined by
// MSD passes over 8-byte big-endian key chunks:
//   prefix   : common prefix of the segment (compare each string with the
//              first one), so a segment's key starts at its first differing byte;
//   keys/diff: gather the 8-byte key at that depth, OR of (key ^ key0) tells
//              which key byte is the first to differ;
//   hist     : per segment, counts of a digit of up to 8 bits: the most
//              significant bits in which its keys may differ;
//   scan     : per segment, bucket starts, bucket-start LCPs, the children;
//   scatter  : ids and keys to their buckets, places reserved per tile by one
//              atomic per digit (the order inside a bucket does not matter:
//              equal strings are ordered by id at the end).
// A child that keeps more than half of its parent (a chain of long shared
// prefixes, e.g. suffixes inside repeats or strings that share a long common
// head) would lose one byte per pass; it is flagged for a pivot pass instead:
// every string's LCP with one of the segment's strings (up to 127 bytes) and
// the byte after it become a two-byte pseudo key whose order is the strings'
// order, so one pass resolves up to 127 bytes of the chain.
// Children of size <= small_max finish in one CTA (k_seg_sort): bucket passes
// on the keys' differing bits in shared memory, ties re-keyed against a pivot
// until every group is a single string or byte-identical strings.
// LCPs are written where they become known: depth + first differing byte at
// every bucket / group boundary, the length for byte-identical neighbours.
// Ties between byte-identical strings keep ascending id order.
#include <algorithm>

#include "internal.cuh"
#include "strsort.cuh"

namespace dsss {

constexpr int LT_NT = 256, LT_IPT = 16, LT_TILE = LT_NT * LT_IPT;
constexpr uint32_t PREFIX_CAP = 256;
// F_KEYS: the key array holds the segment's keys at Seg.depth; F_PIVOT: the
// next pass is a pivot pass; F_PSEUDO: the keys are pivot pseudo keys; F_ID:
// the strings are equal (Seg.depth their length) and are sorted by id.
constexpr uint32_t F_PARITY = 1u, F_KEYS = 2u, F_PIVOT = 4u, F_PSEUDO = 8u, F_ID = 16u;
constexpr uint32_t PIVOT_CAP = 127;  // pseudo key byte 0 holds codes 0 .. 2 * PIVOT_CAP
constexpr uint32_t NO_PIVOT = 0xFFFFFFFFu;

// The bits that pick a key's bucket: up to `want` of the most significant
// bits of diff, in at most 8 runs of neighbouring bits.  A key's bucket is the
// OR over the runs of ((key >> lo) >> sh) & mask; every bit above lo that is
// not chosen is the same in all keys, so buckets order as keys do.  In a
// pseudo group of the segment sorter whose code bits are all chosen, a bucket
// holds one code; otherwise (LCPs over thousands of bytes) `mixed` is set.
struct BucketBits {
    uint32_t lo, nruns, wide, all;  // wide: the bits span more than 32; all: every differing bit is chosen
    uint32_t mixed;
    uint32_t sh[8], mask[8];
};

struct Seg {
    uint32_t start, size, depth, flags;
    uint32_t newdepth;
    // speculated common-prefix depth + 1 (0: none) and the OR of key ^ key0
    // over the keys k_prefix wrote at that depth (segments without keys)
    uint32_t spec;
    unsigned long long spec_diff;
    // bits in which the keys may differ: exact for keys made in this pass, the
    // parent's bits below its digit for keys carried over
    unsigned long long diff;
    uint32_t piv;    // pivot pass: the pivot's string id (NO_PIVOT: the first string)
    uint32_t ended;  // bucket 0 holds the strings that end at the first differing byte
    unsigned long long exact;  // the bits in which the keys do differ (k_hist)
    uint32_t stay, pad;        // the pass does not move the segment
    BucketBits bits;  // this pass's digit
};

struct SmallSeg {
    uint32_t start, size, depth, flags;
};

constexpr int NBINS = 4;
__host__ __device__ constexpr int bin_cap(int b) { return b == 0 ? 32 : b == 1 ? 256 : b == 2 ? 1024 : 4096; }
__host__ __device__ __forceinline__ int bin_of(uint32_t size) {
    return size <= 32 ? 0 : size <= 256 ? 1 : size <= 1024 ? 2 : 3;
}

// Counters block (device): [0] n_large_next, [1..4] n_small per bin, [8] total
// tiles, [10] error flag (a guard tripped), [11] large segments of the next
// pass without keys or with a pivot pass.
struct SortState {
    ArenaDev a;
    uint32_t* ord[2];
    unsigned long long* key[2];
    uint32_t* ord_out;
    uint32_t* lcp_out;
    Seg* large[2];
    SmallSeg* small[NBINS];
    uint32_t* tile0;
    uint32_t* hist;    // D per large segment, zero between passes
    uint32_t* bucket;  // D + 1 per large segment: where the buckets start
    uint32_t* cursor;  // D per large segment: where their next tile goes
    uint32_t dbits;    // digits of up to dbits bits, D = 1 << dbits
    uint32_t* counters;
    uint32_t small_max;
    uint32_t pivot;  // pivot passes enabled
    uint32_t iota;   // first pass over the whole arena: position i holds id i
    uint64_t n;
    uint64_t cap_large, cap_small[NBINS], cap_tiles;
    const uint32_t* seg_depth;  // optional: each segment's shared prefix length
};

__device__ __forceinline__ uint32_t ord_of(const SortState& S, uint32_t par, uint32_t i) {
    return S.iota ? i : S.ord[par][i];
}

// The last s with first[s] <= t, by all lanes of a warp together (32 probes
// per step: three dependent reads for 32768 segments).
__device__ __forceinline__ uint32_t find_seg(const uint32_t* first, uint32_t nseg, uint32_t t) {
    uint32_t lo = 0, hi = nseg;
    while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t x = lo + (threadIdx.x & 31) * step;
        const uint32_t below = __popc(__ballot_sync(0xffffffffu, x < hi && first[x] <= t));
        lo += (below - 1) * step;
        hi = min(hi, lo + step);
    }
    return lo;
}

__device__ __forceinline__ void push_small(const SortState& S, uint32_t start, uint32_t size, uint32_t depth,
                                           uint32_t flags) {
    const int b = bin_of(size);
    const uint32_t slot = atomicAdd(&S.counters[1 + b], 1u);
    if (slot >= S.cap_small[b]) {
        atomicExch(&S.counters[10], 1u);
        return;
    }
    S.small[b][slot] = SmallSeg{start, size, depth, flags};
}

__device__ __forceinline__ void push_large(const SortState& S, Seg* dst, uint32_t start, uint32_t size, uint32_t depth,
                                           uint32_t flags, uint64_t diff = 0) {
    const uint32_t slot = atomicAdd(&S.counters[0], 1u);
    if (slot >= S.cap_large) {
        atomicExch(&S.counters[10], 1u);
        return;
    }
    if (!(flags & F_KEYS)) atomicAdd(&S.counters[11], 1u);
    Seg& s = dst[slot];
    s.start = start;
    s.size = size;
    s.depth = depth;
    s.flags = flags;
    s.newdepth = 0xFFFFFFFFu;
    s.spec = 0;
    s.spec_diff = 0;
    s.diff = diff;
    s.piv = NO_PIVOT;
    s.ended = 0;
    s.exact = 0;
    s.stay = 0;
    s.pad = 0;
}

// ------------------------------------------------------------------ init ----
__global__ void k_init_ids(uint32_t* ord, const uint32_t* in, uint64_t n) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) ord[i] = in ? in[i] : (uint32_t)i;
}

// pb: p + 1 segment bounds (NULL: one segment of n strings).
__global__ void k_init_segs(SortState S, const uint64_t* pb, uint32_t p) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= p) return;
    const uint32_t start = pb ? (uint32_t)pb[q] : 0u, size = pb ? (uint32_t)(pb[q + 1] - pb[q]) : (uint32_t)S.n;
    if (size == 0) return;
    S.lcp_out[start] = 0;
    if (size == 1) {
        S.ord_out[start] = ord_of(S, 0, start);
        return;
    }
    // a segment whose strings are known to share their first bytes starts there
    const uint32_t d = S.seg_depth ? S.seg_depth[q] : 0u;
    if (size > S.small_max) push_large(S, S.large[0], start, size, d, 0);
    else push_small(S, start, size, d, 0);
}

// ---------------------------------------------------------------- prefix ----
// Big-endian key words [d, d + 8 W) of a string (0 past its end) from at most
// W + 1 aligned 8-byte loads, all issued before any is used.  Words wholly
// past the end are not loaded, so at most 15 bytes past a string are read
// (the arena contract pads 32).
template <int W>
__device__ __forceinline__ void key_words(const uint8_t* chars, uint64_t off, uint32_t len, uint32_t d,
                                          uint32_t want, uint64_t (&x)[W]) {
    const uint32_t avail = d < len ? (len - d + 7) >> 3 : 0;
    const uint32_t words = want < avail ? want : avail;
    const uintptr_t p = (uintptr_t)(chars + off + d);
    const unsigned long long* q = (const unsigned long long*)(p & ~(uintptr_t)7);
    const unsigned sh = (unsigned)(p & 7) * 8;
    uint64_t raw[W + 1];
    const uint32_t loads = words ? words + (sh != 0) : 0;
#pragma unroll
    for (int w = 0; w <= W; ++w) raw[w] = (uint32_t)w < loads ? __ldg(q + w) : 0ull;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        uint64_t v = sh ? (raw[w] >> sh) | (raw[w + 1] << (64 - sh)) : raw[w];
        const uint32_t at = d + 8 * w;
        if ((uint32_t)w >= words || at >= len) {
            v = 0;
        } else if (len - at < 8) {
            v &= (1ull << ((len - at) * 8)) - 1;
        }
        x[w] = bswap64(v);
    }
}

constexpr int PF_W = 8;  // prefix words compared per batch (64 bytes)
constexpr uint32_t SPEC_MAX = 56;  // speculated depths stay below d0 + 56 (key inside 64 bytes)

// The pivot of a pivot pass: of PIVOT_SAMPLE evenly spaced members, the one
// with the largest sum of LCPs (from the segment's depth, PIVOT_CAP bytes at
// most) with the others.  In a chain of nested prefixes that is a string of the
// longest shared part, so one pass peels nearly the whole chain; with the
// segment's first string as pivot, every pass left the half of the chain that
// shares more than it does.  Measured on 4e6 strings whose shared prefix has a
// random length: 18 passes -> 4, 2.51 -> 1.69 ms per call.
constexpr uint32_t PIVOT_SAMPLE = 64, PIVOT_WORDS = (PIVOT_CAP + 7) / 8;
__device__ void choose_pivot(const SortState& S, Seg& sg, unsigned long long (*pw)[PIVOT_SAMPLE], uint32_t* psum,
                             uint32_t* pid) {
    const uint32_t* ord = S.ord[sg.flags & F_PARITY];
    const uint32_t m = min(sg.size, PIVOT_SAMPLE), d0 = sg.depth;
    for (uint32_t x = threadIdx.x; x < m * (PIVOT_WORDS / 4); x += blockDim.x) {
        const uint32_t k = x % m, w0 = 4 * (x / m);
        const uint32_t id = ord[sg.start + (uint32_t)((uint64_t)k * sg.size / m)];
        uint64_t off, v[4];
        uint32_t len;
        str_of(S.a, id, off, len);
        key_words<4>(S.a.chars, off, len, d0 + 8 * w0, 4, v);
#pragma unroll
        for (int q = 0; q < 4; ++q) pw[w0 + q][k] = v[q];
        if (w0 == 0) {
            pid[k] = id;
            psum[k] = 0;
        }
    }
    __syncthreads();
    for (uint32_t x = threadIdx.x; x < m * m; x += blockDim.x) {
        const uint32_t i = x % m, j = x / m;
        if (i >= j) continue;
        uint32_t l = 8 * PIVOT_WORDS;
        for (uint32_t w = 0; w < PIVOT_WORDS; ++w) {
            const uint64_t a = pw[w][i], b = pw[w][j];
            if (a != b) {
                l = 8 * w + key_lcp(a, b);
                break;
            }
            if (zero_byte(a) < 8) break;  // equal strings: the longest of LCPs
        }
        l = min(l, PIVOT_CAP);
        atomicAdd(&psum[i], l);
        atomicAdd(&psum[j], l);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        uint32_t best = 0;  // the sum (at most 63 * 127) above, the sample below
        for (uint32_t k = threadIdx.x; k < m; k += 32) best = max(best, psum[k] << 8 | k);
        best = __reduce_max_sync(0xffffffffu, best);
        if (threadIdx.x == 0) sg.piv = pid[best & 0xFFu];
    }
    __syncthreads();  // the sample buffers are reused by the next segment
}

// Speculated common prefix of each segment without keys: the smallest LCP with
// the segment's first string over up to 256 evenly spaced members, when it is
// below d0 + SPEC_MAX.  k_prefix then reads each string once for both the
// check (the segment's common prefix is exactly that depth iff no member
// leaves the first string earlier) and the key at that depth; a wrong guess
// only costs the usual key gather of k_keys_diff.  Segments whose samples all
// share SPEC_MAX bytes keep the plain prefix search (long common prefixes).
__global__ void __launch_bounds__(256) k_spec(SortState S, Seg* segs, uint32_t nseg) {
    __shared__ uint32_t wmin[8];
    __shared__ unsigned long long pw[PIVOT_WORDS][PIVOT_SAMPLE];
    __shared__ uint32_t psum[PIVOT_SAMPLE], pid[PIVOT_SAMPLE];
    for (uint32_t si = blockIdx.x; si < nseg; si += gridDim.x) {
        Seg& sg = segs[si];
        if (sg.flags & F_PIVOT) {  // the same for the whole block
            choose_pivot(S, sg, pw, psum, pid);
            continue;
        }
        if (sg.flags & (F_KEYS | F_ID)) continue;
        const uint32_t par = sg.flags & F_PARITY;
        const uint32_t d0 = sg.depth;
        uint32_t l = 0xFFFFFFFFu;
        const uint32_t m = sg.size < 256u ? sg.size : 256u;
        if (threadIdx.x < m) {
            uint64_t off0, off;
            uint32_t len0, len;
            str_of(S.a, ord_of(S, par, sg.start), off0, len0);
            const uint32_t i = sg.start + (uint32_t)((uint64_t)threadIdx.x * sg.size / m);
            str_of(S.a, ord_of(S, par, i), off, len);
            uint64_t x[7], y[7];
            key_words<7>(S.a.chars, off, len, d0, 7, x);
            key_words<7>(S.a.chars, off0, len0, d0, 7, y);
            l = d0 + SPEC_MAX;
#pragma unroll
            for (int w = 6; w >= 0; --w) {  // the first word that differs or ends wins
                if (x[w] != y[w]) l = d0 + 8 * w + key_lcp(x[w], y[w]);
                else if (zero_byte(x[w]) < 8) l = d0 + 8 * w + zero_byte(x[w]);
            }
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) l = min(l, __shfl_xor_sync(0xffffffffu, l, o));
        if ((threadIdx.x & 31) == 0) wmin[threadIdx.x >> 5] = l;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t v = wmin[0];
            for (int w = 1; w < 8; ++w) v = min(v, wmin[w]);
            sg.spec = v < d0 + SPEC_MAX ? v + 1 : 0u;
            sg.spec_diff = 0;
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(LT_NT, 6) k_prefix(SortState S, Seg* segs, uint32_t nseg) {
    const uint32_t t = blockIdx.x;
    if (t >= S.counters[8]) return;
    const uint32_t si = find_seg(S.tile0, nseg, t);
    Seg& sg = segs[si];
    if (sg.flags & (F_KEYS | F_PIVOT | F_ID)) return;
    const uint32_t par = sg.flags & F_PARITY;
    const uint32_t tb = sg.start + (t - S.tile0[si]) * LT_TILE;
    const uint32_t te = min(sg.start + sg.size, tb + LT_TILE);
    const uint32_t d0 = sg.depth, cap = d0 + PREFIX_CAP;
    const uint32_t s0 = ord_of(S, par, sg.start);
    uint64_t off0;
    uint32_t len0;
    str_of(S.a, s0, off0, len0);
    // the first string's first 64 bytes from d0, shared by the block
    __shared__ unsigned long long y[PF_W];
    if (threadIdx.x == 0) {
        uint64_t v[PF_W];
        key_words<PF_W>(S.a.chars, off0, len0, d0, PF_W, v);
#pragma unroll
        for (int w = 0; w < PF_W; ++w) y[w] = v[w];
    }
    __syncthreads();
    if (sg.spec) {
        // speculated depth D: LCP with the first string capped at D, and the
        // key at D, from one load of the words covering [d0, D + 8)
        const uint32_t D = sg.spec - 1, rel = D - d0;
        const uint32_t want = (rel + 15) >> 3;
        const uint32_t kw = rel >> 3, kr = (rel & 7) * 8;
        const uint64_t key0 = kr ? (y[kw] << kr) | (y[kw + 1] >> (64 - kr)) : y[kw];
        unsigned long long* key = S.key[par];
        uint32_t mn = 0xFFFFFFFFu;
        uint64_t df = 0;
        for (uint32_t i = tb + threadIdx.x; i < te; i += LT_NT) {
            uint64_t off;
            uint32_t len;
            str_of(S.a, ord_of(S, par, i), off, len);
            uint64_t x[PF_W];
            key_words<PF_W>(S.a.chars, off, len, d0, want, x);
            uint32_t l = D;
#pragma unroll
            for (int w = PF_W - 1; w >= 0; --w) {  // the first word that differs or ends wins
                if ((uint32_t)(8 * w) < rel) {
                    if (x[w] != y[w]) l = min(D, d0 + 8 * w + key_lcp(x[w], y[w]));
                    else if (zero_byte(x[w]) < 8) l = min(D, d0 + 8 * w + zero_byte(x[w]));
                }
            }
            uint64_t lo = 0, hi = 0;  // words kw and kw + 1, selected without indexing x at run time
#pragma unroll
            for (int w = 0; w < PF_W; ++w) {
                if ((uint32_t)w == kw) lo = x[w];
                if ((uint32_t)w == kw + 1) hi = x[w];
            }
            const uint64_t k = kr ? (lo << kr) | (hi >> (64 - kr)) : lo;
            key[i] = k;
            df |= k ^ key0;
            mn = min(mn, l);
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
            df |= __shfl_xor_sync(0xffffffffu, df, o);
        }
        if ((threadIdx.x & 31) == 0) {
            if (mn != 0xFFFFFFFFu) atomicMin(&sg.newdepth, mn);
            if (df) atomicOr(&sg.spec_diff, (unsigned long long)df);
        }
        return;
    }
    uint32_t mn = 0xFFFFFFFFu;
    for (uint32_t i = tb + threadIdx.x; i < te; i += LT_NT) {
        uint64_t off;
        uint32_t len;
        str_of(S.a, ord_of(S, par, i), off, len);
        // no need to compare past this thread's minimum so far
        const uint32_t lim = min(cap, mn);
        uint32_t l = 0;
        bool done = false;
        // first batch: every word up to the limit loaded at once
        {
            const uint32_t want = lim > d0 ? min((lim - d0 + 7) >> 3, (uint32_t)PF_W) : 0u;
            uint64_t x[PF_W];
            key_words<PF_W>(S.a.chars, off, len, d0, want, x);
#pragma unroll
            for (int w = 0; w < PF_W; ++w) {
                if (!done && (uint32_t)w < want) {
                    if (x[w] != y[w]) {
                        l = d0 + 8 * w + key_lcp(x[w], y[w]);
                        done = true;
                    } else {
                        const uint32_t z = zero_byte(x[w]);
                        if (z < 8) {
                            l = d0 + 8 * w + z;
                            done = true;
                        }
                    }
                }
            }
            if (!done && d0 + 8 * want >= lim) {
                l = d0 + 8 * want;
                done = true;
            }
        }
        // longer common prefixes: 16 bytes per step
        for (uint32_t d = d0 + 8 * PF_W; !done;) {
            uint64_t xx[2], yy[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                xx[q] = key8(S.a.chars, off, len, d + 8 * q);
                yy[q] = key8(S.a.chars, off0, len0, d + 8 * q);
            }
            l = d + 16;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if (!done) {
                    if (xx[q] != yy[q]) {
                        l = d + 8 * q + key_lcp(xx[q], yy[q]);
                        done = true;
                    } else {
                        const uint32_t z = zero_byte(xx[q]);
                        if (z < 8) {
                            l = d + 8 * q + z;
                            done = true;
                        }
                    }
                }
            }
            if (done) break;
            d += 16;
            if (d >= lim) {
                l = d;
                break;
            }
        }
        mn = min(mn, l);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    if ((threadIdx.x & 31) == 0 && mn != 0xFFFFFFFFu) atomicMin(&sg.newdepth, mn);
}

// ------------------------------------------------------------- keys/diff ----
constexpr int KD_ILP = 8;
__global__ void __launch_bounds__(LT_NT) k_keys_diff(SortState S, Seg* segs, uint32_t nseg) {
    const uint32_t t = blockIdx.x;
    if (t >= S.counters[8]) return;
    const uint32_t si = find_seg(S.tile0, nseg, t);
    Seg& sg = segs[si];
    if (sg.flags & (F_KEYS | F_PIVOT)) return;  // keys carried over, or made by k_pivot
    const bool by_id = sg.flags & F_ID;
    if (!by_id && sg.spec && sg.newdepth == sg.spec - 1) {
        // the speculated depth was the common prefix: k_prefix wrote the keys
        if (t == S.tile0[si] && threadIdx.x == 0) sg.diff = sg.spec_diff;
        return;
    }
    const uint32_t par = sg.flags & F_PARITY, depth = sg.newdepth;
    unsigned long long* key = S.key[par];
    const uint32_t tb = sg.start + (t - S.tile0[si]) * LT_TILE;
    const uint32_t te = min(sg.start + sg.size, tb + LT_TILE);
    const uint32_t s0 = ord_of(S, par, sg.start);
    const uint64_t k0 = by_id ? (uint64_t)s0 : key8_of(S.a, s0, depth);
    uint64_t df = 0;
    // KD_ILP independent gathers in flight per thread
    for (uint32_t i0 = tb + threadIdx.x; i0 < te; i0 += KD_ILP * LT_NT) {
        uint32_t s[KD_ILP];
        uint64_t off[KD_ILP];
        uint32_t len[KD_ILP];
#pragma unroll
        for (int q = 0; q < KD_ILP; ++q) {
            const uint32_t i = i0 + q * LT_NT;
            s[q] = i < te ? ord_of(S, par, i) : 0u;
        }
        if (by_id) {
#pragma unroll
            for (int q = 0; q < KD_ILP; ++q) {
                const uint32_t i = i0 + q * LT_NT;
                if (i < te) {
                    key[i] = s[q];
                    df |= s[q] ^ k0;
                }
            }
            continue;
        }
#pragma unroll
        for (int q = 0; q < KD_ILP; ++q) {
            const uint32_t i = i0 + q * LT_NT;
            off[q] = 0;
            len[q] = 0;
            if (i < te) str_of(S.a, s[q], off[q], len[q]);
        }
#pragma unroll
        for (int q = 0; q < KD_ILP; ++q) {
            const uint32_t i = i0 + q * LT_NT;
            if (i < te) {
                const uint64_t k = key8(S.a.chars, off[q], len[q], depth);
                key[i] = k;
                df |= k ^ k0;
            }
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) df |= __shfl_xor_sync(0xffffffffu, df, o);
    if ((threadIdx.x & 31) == 0 && df) atomicOr(&sg.diff, (unsigned long long)df);
}

// ----------------------------------------------------------------- pivot ----
// Pivot pass of an F_PIVOT segment at depth d (all its strings share their
// first d bytes) with pivot s0, one of its strings.  For string x, l = LCP(x, s0)
// counted from d and capped at PIVOT_CAP, and x's pseudo key holds
//   byte 0: code = l            if x < s0 (x's byte at l is smaller: x ends
//                               there or differs downwards),
//                = PIVOT_CAP    if x matches s0 for PIVOT_CAP bytes or equals it,
//                = 2*PIVOT_CAP - l  if x > s0;
//   byte 1: x's byte at d + l (0 for the code PIVOT_CAP).
// Ascending pseudo keys are ascending strings: two strings below s0 with
// different l compare at the smaller l, where the one with the smaller l has
// the smaller byte; above s0 the larger l comes first; equal codes compare by
// the byte at d + l.  Strings with the same pseudo key share their first
// d + l + 1 bytes (d + PIVOT_CAP for the middle code), and the LCP of two
// strings with different codes is d + min(l, l').
__device__ __forceinline__ uint32_t pivot_l(uint32_t code) { return code <= PIVOT_CAP ? code : 2 * PIVOT_CAP - code; }

// Pseudo key of string (off, len) against the pivot, whose big-endian words
// from depth d0 (zero past its end) are y[0..PIVOT_WORDS): 32 bytes of the
// string per step, all their loads in flight together.
__device__ __forceinline__ uint64_t pivot_key(const uint8_t* chars, uint64_t off, uint32_t len,
                                              const unsigned long long* y, uint32_t d0) {
    for (uint32_t c = 0; c < PIVOT_WORDS; c += 4) {
        uint64_t x[4];
        key_words<4>(chars, off, len, d0 + 8 * c, 4, x);
        uint32_t l = 0xFFFFFFFFu;
        uint64_t xw = 0, yw = 0;
#pragma unroll
        for (int q = 3; q >= 0; --q) {  // the first word that differs or ends wins
            const uint64_t v = y[c + q];
            if (x[q] != v || zero_byte(v) < 8) {
                l = 8 * (c + q);
                xw = x[q];
                yw = v;
            }
        }
        if (l == 0xFFFFFFFFu) continue;
        if (xw == yw) break;  // equal to the pivot
        const uint32_t j = key_lcp(xw, yw);
        l += j;
        if (l >= PIVOT_CAP) break;
        const uint32_t bx = (uint32_t)(xw >> (56 - 8 * j)) & 0xFFu, by = (uint32_t)(yw >> (56 - 8 * j)) & 0xFFu;
        return (uint64_t)(bx < by ? l : 2 * PIVOT_CAP - l) << 56 | (uint64_t)bx << 48;
    }
    return (uint64_t)PIVOT_CAP << 56;
}

__global__ void __launch_bounds__(LT_NT) k_pivot(SortState S, Seg* segs, uint32_t nseg) {
    const uint32_t t = blockIdx.x;
    if (t >= S.counters[8]) return;
    const uint32_t si = find_seg(S.tile0, nseg, t);
    Seg& sg = segs[si];
    if (!(sg.flags & F_PIVOT)) return;
    const uint32_t par = sg.flags & F_PARITY;
    const uint32_t* ord = S.ord[par];
    unsigned long long* key = S.key[par];
    const uint32_t tb = sg.start + (t - S.tile0[si]) * LT_TILE;
    const uint32_t te = min(sg.start + sg.size, tb + LT_TILE);
    __shared__ unsigned long long y[PIVOT_WORDS];
    if (threadIdx.x < PIVOT_WORDS) {
        uint64_t off0;
        uint32_t len0;
        str_of(S.a, sg.piv == NO_PIVOT ? ord[sg.start] : sg.piv, off0, len0);
        y[threadIdx.x] = key8(S.a.chars, off0, len0, sg.depth + 8 * threadIdx.x);
    }
    __syncthreads();
    const uint64_t k0 = (uint64_t)PIVOT_CAP << 56;
    uint64_t df = 0;
    for (uint32_t i = tb + threadIdx.x; i < te; i += LT_NT) {
        uint64_t off;
        uint32_t len;
        str_of(S.a, ord[i], off, len);
        const uint64_t k = pivot_key(S.a.chars, off, len, y, sg.depth);
        key[i] = k;
        df |= k ^ k0;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) df |= __shfl_xor_sync(0xffffffffu, df, o);
    if ((threadIdx.x & 31) == 0 && df) atomicOr(&sg.diff, (unsigned long long)df);
}

// ------------------------------------------------------------------ hist ----
__device__ __forceinline__ uint32_t bucket_of_key(const BucketBits& B, uint64_t k) {
    uint32_t b = 0;
    for (uint32_t r = 0; r < B.nruns; ++r) b |= (uint32_t)(k >> (B.lo + B.sh[r])) & B.mask[r];
    return b;
}

__device__ __forceinline__ void bucket_bits(BucketBits& B, uint64_t diff, uint32_t want) {
    uint32_t n = 0, left = want, lo = 0;
    uint64_t x = diff;
    const uint32_t hi = 63u - (uint32_t)__clzll(diff);
    // a run's lowest bit and length, for the second loop
    do {
        const uint32_t h = 63u - (uint32_t)__clzll(x);
        const uint32_t take = min((uint32_t)__clzll(~(x << (63u - h))), left);  // set bits from h down
        lo = h - take + 1;
        B.sh[n] = lo;
        B.mask[n] = (1u << take) - 1u;
        left -= take;
        x &= (1ull << lo) - 1;
        ++n;
    } while (x && n < 8 && left);
    B.lo = lo;
    B.nruns = n;
    B.wide = hi - lo >= 32;
    B.all = x == 0;
    B.mixed = (x >> 48) != 0;
    uint32_t place = 0;
    for (uint32_t k = n; k-- > 0;) {
        const uint32_t m = B.mask[k];
        B.sh[k] = B.sh[k] - lo - place;
        B.mask[k] = m << place;
        place += (uint32_t)__popc(m);
    }
}

// This pass's digit of a segment: pivot pseudo keys split on a whole byte (the
// code, then the byte behind the LCP), other keys on their most significant
// differing bits: as many as leave about DIGIT_TARGET strings per bucket, in
// equal parts where one pass of DIGIT_BITS_MAX is too few.  A digit over letters
// (5 differing bits per byte) or DNA (4) covers more than a byte: 1e8 random
// six-letter keys take two passes, four by bytes and three by 8 bits (whose
// last one leaves segments of 100 to 200 strings: counts, scatters and segment
// sorter 4.7 ms, with passes of 9 and 10 bits 3.4 ms); narrower digits for
// segments just above the cutoff keep their children from being a few strings
// each.
constexpr uint32_t DIGIT_TARGET = 1200, DIGIT_BITS_MAX = 10, DIGIT_MAX = 1u << DIGIT_BITS_MAX;
__device__ __forceinline__ void segment_digit(BucketBits& B, uint64_t diff, uint32_t flags, uint32_t size,
                                              uint32_t dbits) {
    if (flags & (F_PIVOT | F_PSEUDO)) {
        B.lo = 56 - 8 * (uint32_t)(__clzll(diff) >> 3);
        B.nruns = 1;
        B.wide = 0;
        B.all = 0;
        B.mixed = 0;
        B.sh[0] = 0;
        B.mask[0] = 0xFFu;
        return;
    }
    const uint32_t need = max(3u, 33u - (uint32_t)__clz((size / DIGIT_TARGET) | 1u));
    const uint32_t passes = (need + dbits - 1) / dbits;
    bucket_bits(B, diff, (need + passes - 1) / passes);
}

// The bits of a key that a digit holds.
__device__ __forceinline__ uint64_t digit_mask(const BucketBits& B) {
    uint64_t m = 0;
    for (uint32_t r = 0; r < B.nruns; ++r) m |= (uint64_t)B.mask[r] << (B.lo + B.sh[r]);
    return m;
}

// Bucket numbers of N keys (the runs outermost: one shared read per run).
template <int N>
__device__ __forceinline__ void digits_of(const BucketBits& B, const uint64_t (&k)[N], uint32_t (&d)[N]) {
    const uint32_t lo = B.lo, nr = B.nruns;
#pragma unroll
    for (int j = 0; j < N; ++j) d[j] = 0;
    if (B.wide) {
        for (uint32_t r = 0; r < nr; ++r) {
            const uint32_t sh = lo + B.sh[r], mask = B.mask[r];
#pragma unroll
            for (int j = 0; j < N; ++j) d[j] |= (uint32_t)(k[j] >> sh) & mask;
        }
        return;
    }
    uint32_t x[N];
#pragma unroll
    for (int j = 0; j < N; ++j) x[j] = (uint32_t)(k[j] >> lo);
    for (uint32_t r = 0; r < nr; ++r) {
        const uint32_t sh = B.sh[r], mask = B.mask[r];
#pragma unroll
        for (int j = 0; j < N; ++j) d[j] |= (x[j] >> sh) & mask;
    }
}

// Counts per segment and digit, and the bits in which the keys do differ: a
// tile's counts in shared memory (a row for every two warps), then one global
// atomic per digit.  Bound by the 8-byte key read.
constexpr int HIST_ROWS = LT_NT / 64;
__global__ void __launch_bounds__(LT_NT, 4) k_hist(SortState S, Seg* segs, uint32_t nseg) {
    __shared__ uint32_t hist[HIST_ROWS][DIGIT_MAX];
    __shared__ unsigned long long s_diff[LT_NT / 32];
    __shared__ BucketBits B;
    const uint32_t t = blockIdx.x, D = 1u << S.dbits;
    if (t >= S.counters[8]) return;
    const uint32_t si = find_seg(S.tile0, nseg, t);
    Seg& sg = segs[si];
    const uint64_t diff = sg.diff;
    if (diff == 0) return;
    const uint32_t start = sg.start, size = sg.size, flags = sg.flags;
    const uint32_t tb = start + (t - S.tile0[si]) * LT_TILE;
    const uint32_t te = min(start + size, tb + LT_TILE);
    const unsigned long long* key = S.key[flags & F_PARITY];
    // the tile's keys loaded before the digit is known (one DRAM wait)
    uint64_t k[LT_IPT];
#pragma unroll
    for (int j = 0; j < LT_IPT; ++j) {
        const uint32_t i = tb + j * LT_NT + threadIdx.x;
        k[j] = i < te ? key[i] : 0;
    }
    const uint64_t k0 = key[start];
    if (threadIdx.x == 0) segment_digit(B, diff, flags, size, S.dbits);
#pragma unroll
    for (int w = 0; w < HIST_ROWS; ++w)
        for (uint32_t x = threadIdx.x; x < D; x += LT_NT) hist[w][x] = 0;
    __syncthreads();
    uint32_t d[LT_IPT];
    digits_of(B, k, d);
    uint32_t* wh = hist[threadIdx.x >> 6];
#pragma unroll
    for (int j = 0; j < LT_IPT; ++j)
        if (tb + j * LT_NT + threadIdx.x < te) atomicAdd(&wh[d[j]], 1u);
    uint64_t df = 0;
#pragma unroll
    for (int j = 0; j < LT_IPT; ++j)
        if (tb + j * LT_NT + threadIdx.x < te) df |= k[j] ^ k0;
    const uint32_t dlo = __reduce_or_sync(0xffffffffu, (uint32_t)df);
    const uint32_t dhi = __reduce_or_sync(0xffffffffu, (uint32_t)(df >> 32));
    if ((threadIdx.x & 31) == 0) s_diff[threadIdx.x >> 5] = (unsigned long long)dhi << 32 | dlo;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long x = 0;
#pragma unroll
        for (int w = 0; w < LT_NT / 32; ++w) x |= s_diff[w];
        if (x) atomicOr(&sg.exact, x);
    }
    for (uint32_t x = threadIdx.x; x < D; x += LT_NT) {
        uint32_t c = 0;
#pragma unroll
        for (int w = 0; w < HIST_ROWS; ++w) c += hist[w][x];
        if (c) atomicAdd(&S.hist[((uint64_t)si << S.dbits) + x], c);
    }
}

// ----------------------------------------------------------- segment scan ----
// One block per segment: bucket starts, the LCPs at bucket starts, and the
// segment's children; DPT consecutive digits per thread.
template <int DPT>
__global__ void __launch_bounds__(256) k_seg_scan(SortState S, Seg* segs, Seg* next) {
    constexpr uint32_t D = 256 * DPT;
    __shared__ uint32_t wsum[8], any[D / 32];  // any: the digits that occur
    __shared__ uint32_t s_small[NBINS], s_base[NBINS];
    __shared__ BucketBits B;
    const uint32_t si = blockIdx.x;
    Seg& sg = segs[si];
    const uint32_t start = sg.start, size = sg.size, flags = sg.flags, par = flags & F_PARITY, np = par ^ 1u;
    const uint64_t diff = sg.exact;
    const bool pseudo = (flags & (F_PIVOT | F_PSEUDO)) != 0, by_id = (flags & F_ID) != 0;
    const uint32_t depth = (flags & (F_KEYS | F_PIVOT | F_ID)) ? sg.depth : sg.newdepth;
    const uint64_t k0 = S.key[par][start];
    if (diff == 0) {
        // Every key equal: byte-identical strings if the key holds their end,
        // else continue deeper without keys.
        // (counted in one bucket when the parent left bits open)
        uint32_t* hist = S.hist + (uint64_t)si * D + threadIdx.x * DPT;
        for (int q = 0; q < DPT; ++q) hist[q] = 0;
        if (threadIdx.x != 0) return;
        sg.stay = 1;
        uint32_t fin = 0xFFFFFFFFu, cont = 0, cflags = par;
        if (pseudo) {
            const uint32_t code = (uint32_t)(k0 >> 56), byte = (uint32_t)(k0 >> 48) & 0xFFu;
            if (code == PIVOT_CAP) {
                uint64_t o0;
                uint32_t l0;
                str_of(S.a, ord_of(S, par, start), o0, l0);
                if (l0 < depth + PIVOT_CAP) fin = l0;  // all equal the pivot
                else cont = depth + PIVOT_CAP;
            } else if (byte == 0) {
                fin = depth + pivot_l(code);  // all end where they leave the pivot
            } else {
                cont = depth + pivot_l(code) + 1;
            }
            cflags |= F_PIVOT;
        } else {
            const uint32_t z = zero_byte(k0);
            if (z < 8) fin = depth + z;
            else cont = depth + 8;
        }
        if (fin != 0xFFFFFFFFu) push_large(S, next, start, size, fin, par | F_ID);
        else push_large(S, next, start, size, cont, cflags);
        return;
    }
    uint32_t tot[DPT], sum = 0, occ = 0;
    uint32_t* hist = S.hist + (uint64_t)si * D + threadIdx.x * DPT;
#pragma unroll
    for (int q = 0; q < DPT; ++q) {
        tot[q] = hist[q];
        hist[q] = 0;
        sum += tot[q];
        occ |= (tot[q] != 0 ? 1u : 0u) << q;
    }
    if (threadIdx.x < D / 32) any[threadIdx.x] = 0;
    if (threadIdx.x < NBINS) s_small[threadIdx.x] = 0;
    if (threadIdx.x == 0) segment_digit(B, sg.diff, flags, size, S.dbits);
    // block exclusive scan over the digits
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    if (occ) atomicOr(&any[threadIdx.x * DPT / 32], occ << (threadIdx.x * DPT % 32));
    uint32_t cs = start + x - sum;
    for (int k = 0; k < w; ++k) cs += wsum[k];
    __syncthreads();
    // byte b is the first that may differ; bucket 0 holds the strings that end
    // there if that byte's differing bits are all in the digit and it has no
    // constant nonzero part
    const uint32_t b = (uint32_t)(__clzll(diff) >> 3), shift = 56 - 8 * b;
    const uint64_t mask = digit_mask(B), rest = diff & ~mask;
    const bool plain = !pseudo && !by_id, code_split = pseudo && b == 0;
    if ((diff & mask) == 0) {  // one bucket: the same keys again, on the bits that do differ
        if (threadIdx.x == 0) {
            sg.stay = 1;
            push_large(S, next, start, size, depth, par | F_KEYS | (flags & F_ID) | (pseudo ? F_PSEUDO : 0u), diff);
        }
        return;
    }
    const bool ended = plain ? (((k0 >> shift) & ~(diff >> shift)) & 0xFFu) == 0 && ((rest >> shift) & 0xFFu) == 0
                             : pseudo && !code_split;
    const uint32_t lcp_here = pseudo ? depth + pivot_l((uint32_t)(k0 >> 56)) : depth + b;
    if (threadIdx.x == 0) {
        sg.bits = B;
        sg.ended = ended;
        S.bucket[(uint64_t)si * (D + 1) + D] = start + size;
    }
    // small children get their places by one global atomic per bin and block
    uint32_t sdepth[DPT], sflags[DPT], sslot[DPT];
#pragma unroll
    for (int q = 0; q < DPT; ++q) sslot[q] = 0xFFFFFFFFu;
    auto small = [&](int q, uint32_t dp, uint32_t fl) {
        sdepth[q] = dp;
        sflags[q] = fl;
        sslot[q] = atomicAdd(&s_small[bin_of(tot[q])], 1u);
    };
    const uint32_t cs0 = cs;
#pragma unroll
    for (int q = 0; q < DPT; ++q) {
        const uint32_t d = threadIdx.x * DPT + q, total = tot[q];
        if (q) cs += tot[q - 1];
        S.bucket[(uint64_t)si * (D + 1) + d] = cs;
        S.cursor[(uint64_t)si * D + d] = cs;
        if (total == 0) continue;
        if (cs != start) {
            // LCP with the bucket before (the last smaller digit that occurs)
            int pw = (int)(d >> 5);
            uint32_t m = any[pw] & ((1u << (d & 31)) - 1u);
            while (m == 0) m = any[--pw];
            const uint32_t pd = (uint32_t)pw * 32 + 31u - (uint32_t)__clz(m);
            uint32_t l = lcp_here;
            if (by_id) {
                l = depth;
            } else if (code_split) {
                l = depth + min(pivot_l(d), pivot_l(pd));
            } else if (plain) {
                // the byte of the highest bit in which the two digits differ
                const uint32_t h = 31u - (uint32_t)__clz(d ^ pd);
                for (uint32_t r = 0; r < B.nruns; ++r)
                    if ((B.mask[r] >> h) & 1u) l = depth + ((63u - (B.lo + B.sh[r] + h)) >> 3);
            }
            S.lcp_out[cs] = l;
        }
        if (total < 2) continue;
        const bool big = total > S.small_max;
        // a chain: most strings stay together, and not because most of the
        // digit's bits, left open by the parent, do not differ here
        const bool chain = S.pivot && 2 * (uint64_t)total > size &&
                           (pseudo || rest == 0 || 2 * __popcll(diff & mask) >= __popcll(mask));
        if (by_id) {
            if (big) push_large(S, next, cs, total, depth, np | F_KEYS | F_ID, rest);
            else small(q, depth, np | F_ID);
        } else if (ended && d == 0) {
            // equal strings: the scatter makes their ids the keys
            const uint32_t fin = lcp_here;
            if (big) push_large(S, next, cs, total, fin, np | F_KEYS | F_ID,
                                (2ull << (63 - __clzll(max(S.n, S.a.n)))) - 1);
            else small(q, fin, np | F_ID);
        } else if (plain) {
            // children keep the parent's keys, whose bits down to the digit's
            // lowest are now common; one that keeps most of the parent gets a
            // pivot pass
            if (!big) small(q, depth, np | F_KEYS);
            else if (chain) push_large(S, next, cs, total, depth + ((64u - B.lo) >> 3), np | F_PIVOT);
            else push_large(S, next, cs, total, depth, np | F_KEYS, rest);
        } else if (code_split) {
            // split by pivot code (only the pivot pass's own segment): large
            // children keep the pseudo keys, small ones restart from the depth
            // their strings share
            if (big) {
                // (the code of the pivot itself has no byte behind it)
                push_large(S, next, cs, total, depth, np | F_KEYS | F_PSEUDO,
                           d == PIVOT_CAP ? 0 : rest & ~(0xFFull << 56));
            } else {
                uint32_t cd = depth + pivot_l(d);
                if (d == PIVOT_CAP) {
                    uint64_t o0;
                    uint32_t l0;
                    str_of(S.a, sg.piv == NO_PIVOT ? ord_of(S, par, start) : sg.piv, o0, l0);
                    cd = min(depth + PIVOT_CAP, l0);
                }
                small(q, cd, np);
            }
        } else {
            // split by the byte after the shared d + l bytes
            const uint32_t cd = lcp_here + 1;
            if (big) push_large(S, next, cs, total, cd, np | (chain ? F_PIVOT : 0u));
            else small(q, cd, np);
        }
    }
    __syncthreads();
    if (threadIdx.x < NBINS) {
        const uint32_t m = s_small[threadIdx.x];
        s_base[threadIdx.x] = m ? atomicAdd(&S.counters[1 + threadIdx.x], m) : 0u;
    }
    __syncthreads();
    cs = cs0;
#pragma unroll
    for (int q = 0; q < DPT; ++q) {
        if (sslot[q] != 0xFFFFFFFFu) {
            const int bin = bin_of(tot[q]);
            const uint32_t at = s_base[bin] + sslot[q];
            if (at < S.cap_small[bin]) S.small[bin][at] = SmallSeg{cs, tot[q], sdepth[q], sflags[q]};
            else atomicExch(&S.counters[10], 1u);
        }
        cs += tot[q];
    }
}

// --------------------------------------------------------------- scatter ----
// The tile is reordered by digit in shared memory, places from shared
// atomics, so that the global writes of each digit's run are contiguous; one
// global atomic per digit reserves the run's place in its bucket.  Bound by
// the 24 bytes moved per key and the shared-memory round trip; with stable
// ranks from match instructions, per-tile counts and their scans, and keys
// folded for the children, a pass over 32e6 keys took 0.31 ms; now 0.15 to
// 0.19 ms.
constexpr int SC_NT = 512, SC_IPT = LT_TILE / SC_NT;
constexpr size_t SCATTER_SMEM = (size_t)LT_TILE * (8 + 4 + 2);

__global__ void __launch_bounds__(SC_NT, 2) k_scatter(SortState S, const Seg* segs, uint32_t nseg) {
    extern __shared__ __align__(16) unsigned char sm_scatter[];
    unsigned long long* skey = (unsigned long long*)sm_scatter;
    uint32_t* sord = (uint32_t*)(skey + LT_TILE);
    uint16_t* sdig = (uint16_t*)(sord + LT_TILE);
    __shared__ uint32_t cnt[DIGIT_MAX], tloff[DIGIT_MAX], wsum[SC_NT / 32];
    __shared__ uint2 dst[DIGIT_MAX];  // place of the digit's run minus its place in the tile; whether its bucket is one string
    __shared__ BucketBits B;
    const uint32_t t = blockIdx.x;
    if (t >= S.counters[8]) return;
    const uint32_t D = 1u << S.dbits;
    const uint32_t si = find_seg(S.tile0, nseg, t);
    const Seg& sg = segs[si];
    const uint32_t start = sg.start, end = start + sg.size, flags = sg.flags, par = flags & F_PARITY;
    const uint32_t tb = start + (t - S.tile0[si]) * LT_TILE;
    const uint32_t te = min(end, tb + LT_TILE);
    const uint32_t tn = te - tb;
    if (sg.stay) {  // the segment stays where it is (its ids must exist)
        if (S.iota)
            for (uint32_t i = tb + threadIdx.x; i < te; i += SC_NT) S.ord[par][i] = i;
        return;
    }
    const unsigned long long* key = S.key[par];
    uint64_t k[SC_IPT];
    uint32_t o[SC_IPT];
#pragma unroll
    for (int j = 0; j < SC_IPT; ++j) {
        const uint32_t i = tb + j * SC_NT + threadIdx.x;
        k[j] = i < te ? key[i] : 0;
        o[j] = i < te ? ord_of(S, par, i) : 0;
    }
    if (threadIdx.x < sizeof(BucketBits) / 4) ((uint32_t*)&B)[threadIdx.x] = ((const uint32_t*)&sg.bits)[threadIdx.x];
    const bool ended = sg.ended;
#pragma unroll
    for (uint32_t x = 0; x < DIGIT_MAX / SC_NT; ++x) cnt[x * SC_NT + threadIdx.x] = 0;
    __syncthreads();
    uint32_t d[SC_IPT];
    digits_of(B, k, d);
#pragma unroll
    for (int j = 0; j < SC_IPT; ++j)
        if (tb + j * SC_NT + threadIdx.x < te) d[j] |= atomicAdd(&cnt[d[j]], 1u) << DIGIT_BITS_MAX;
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    constexpr int PER = DIGIT_MAX / SC_NT;
    uint32_t c[PER], x = 0;
#pragma unroll
    for (int q = 0; q < PER; ++q) x += c[q] = cnt[threadIdx.x * PER + q];
    const uint32_t mine = x;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    uint32_t at = x - mine;
#pragma unroll
    for (int ww = 0; ww < SC_NT / 32; ++ww)
        if (ww < w) at += wsum[ww];
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        const uint32_t dg = threadIdx.x * PER + q;
        tloff[dg] = at;
        if (c[q]) {  // then dg < D
            const uint32_t* bk = S.bucket + (uint64_t)si * (D + 1) + dg;
            const uint32_t base = atomicAdd(&S.cursor[(uint64_t)si * D + dg], c[q]);
            dst[dg] = make_uint2(base - at, bk[1] - bk[0] == 1);
        }
        at += c[q];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < SC_IPT; ++j) {
        if (tb + j * SC_NT + threadIdx.x >= te) continue;
        const uint32_t dg = d[j] & (DIGIT_MAX - 1), lp = tloff[dg] + (d[j] >> DIGIT_BITS_MAX);
        skey[lp] = ended && dg == 0 ? (uint64_t)o[j] : k[j];  // equal strings go on by id
        sord[lp] = o[j];
        sdig[lp] = (uint16_t)dg;
    }
    __syncthreads();
    uint32_t* ord_dst = S.ord[par ^ 1u];
    unsigned long long* key_dst = S.key[par ^ 1u];
    for (uint32_t i = threadIdx.x; i < tn; i += SC_NT) {
        const uint2 to = dst[sdig[i]];
        const uint32_t at = to.x + i;
        if (at < start || at >= end) {  // never taken when the counts agree
            atomicExch(&S.counters[10], 1u);
            continue;
        }
        const uint32_t oo = sord[i];
        if (to.y) {
            S.ord_out[at] = oo;
        } else {
            ord_dst[at] = oo;
            key_dst[at] = skey[i];
        }
    }
}


// ------------------------------------------------------------ small sort ----
// Segments of 2..small_max strings finish inside one CTA (the tail the MSD
// passes hand over, like the reference's insertion-sort / multikey tail), those
// of up to 32 in one warp.  A group of strings is sorted by a 64-bit key:
//   plain  : 8 bytes of each string from the group's depth;
//   pseudo : each string's LCP l (from the depth) with one of the group, the
//            pivot, as a 16-bit code that orders as the strings do, then the 6
//            bytes behind it: a group whose 8-byte keys all agree goes on with
//            these, since its strings often agree for long (suffixes of copied
//            text, shared heads) and then leave the pivot at many depths;
//   id     : the strings are equal; they keep ascending ids.
// Equal keys that do not hold their strings' end form the next groups.
//
// A CTA takes groups of more than 32 strings through one bucket pass each: the
// most significant bits in which the group's keys differ, as many as two
// buckets per string need, pick a bucket; shared atomics count them and hand
// out places (the order inside a bucket does not matter, every bucket is
// sorted by (key, id) afterwards); buckets of 2..8 strings are sorted by one
// thread each, up to 64 by a warp, larger ones return to the CTA's stack.
// The first pass, which is all that most segments need, stands by itself: the
// rest is one call behind it, whose registers would else cut into the first
// pass's (1e8 strings in segments of about 700: 1.32 ms inlined, 1.18 ms as a
// call, 1.03 ms with the five blocks per SM that then fit).
//
// What bounds the groups that go deeper is latency, not instructions: a group
// of the CTA takes a dozen barriers, of the warps a chain of loads per round.
// So warps claim groups from a list, several small ones at a time in their 64
// elements, and all lanes of a comparison step on together (text with repeats,
// 9e6 strings: 32 elements and one group per warp, comparisons beyond 32 bytes
// one lane after another: 5.4 ms; this: 3.8; groups up to 128 by a warp: 4.1).
// Over keys with enough differing bits nearly all buckets hold one string, so
// a string costs about 60 thread instructions; the stable byte passes with
// match instructions and bitonic networks that this replaces took 26 warp
// instructions per string.  B200, 32e6 strings in segments of about 700:
// 1.12 -> 0.29 ms; a 4e6-string request whose segments are chains of nested
// prefixes: 0.61 -> 0.13 ms; 9e6 suffixes of copied text: 9.2 -> 3.8 ms.
constexpr unsigned FULL = 0xffffffffu;
enum GroupKind : uint32_t { G_PLAIN = 0, G_TIE = 1, G_ID = 2, G_PSEUDO = 3 };  // G_TIE: keys still to be made
// Pivot code of a string with LCP l: l below the pivot, CODE_MID for strings
// equal to it (or to CODE_CAP bytes of it), 0xBFFF - l above it.
constexpr uint32_t CODE_MID = 0x4000u, CODE_TOP = 0xBFFFu, CODE_CAP = 0x3FFEu;
constexpr uint32_t TINY_MAX = 8;  // largest bucket one thread sorts
constexpr uint32_t MID_MAX = 64;  // largest group that one warp sorts

// LCP part of a pivot code (the pivot's own is above all others).
__device__ __forceinline__ uint32_t code_l(uint32_t c) { return c <= CODE_MID ? c : CODE_TOP - c; }

// The key whose differing bits choose a group's buckets: above the pivot the
// code counts down, so its LCP bits are flipped back.  In the key itself the
// bits that then do not differ follow from the two highest ones.
__device__ __forceinline__ uint64_t level_key(uint64_t k, bool pseudo) {
    return pseudo && (k >> 63) ? k ^ 0x3FFFull << 48 : k;
}

// Bytes before the end that a key holds: plain, index of its first zero byte
// (8: none); pseudo, index among its last six (6: none).
__device__ __forceinline__ uint32_t key_end(uint64_t k, bool pseudo) {
    return pseudo ? zero_byte(k | 0xFFFF000000000000ull) - 2 : zero_byte(k);
}
__device__ __forceinline__ bool key_ended(uint64_t k, bool pseudo) { return key_end(k, pseudo) < (pseudo ? 6u : 8u); }

// LCP of two strings of a group of depth d whose keys differ.
__device__ __forceinline__ uint32_t group_lcp(uint64_t x, uint64_t y, uint32_t d, bool pseudo) {
    if (!pseudo) return d + key_lcp(x, y);
    const uint32_t cx = (uint32_t)(x >> 48), cy = (uint32_t)(y >> 48);
    if (cx != cy) return d + min(code_l(cx), code_l(cy));
    return d + code_l(cx) + key_lcp(x, y) - 2;
}

// Depth up to which strings with the equal, not ended key k agree.
__device__ __forceinline__ uint32_t tie_depth(uint64_t k, uint32_t d, bool pseudo) {
    if (!pseudo) return d + 8;
    const uint32_t c = (uint32_t)(k >> 48);
    return c == CODE_MID ? d + CODE_CAP : d + code_l(c) + 6;
}

struct StrRef {
    uint64_t off;
    uint32_t len;
};

__device__ __forceinline__ StrRef ref_of(const ArenaDev& a, uint32_t id) {
    StrRef r;
    str_of(a, id, r.off, r.len);
    return r;
}

// Each active lane's LCP with its own pivot h, both strings sharing their
// first d bytes; at most d + CODE_CAP.  Lanes take 32 bytes of their own pair
// at a time; once at most four are still equal these go one after another, the
// whole warp reading 256 bytes of a pair at a time.  Every lane of the warp
// calls it.
__device__ __forceinline__ uint32_t warp_lcp(const uint8_t* chars, StrRef x, StrRef h, uint32_t d, bool active) {
    uint32_t l = d;
    bool open = active;
    uint32_t todo;
    do {
        if (open) {
            const uint32_t at = l;
            uint64_t u[4], v[4];
            key_words<4>(chars, x.off, x.len, at, 4, u);
            key_words<4>(chars, h.off, h.len, at, 4, v);
            l = at + 32;
#pragma unroll
            for (int w = 3; w >= 0; --w) {  // the first word that differs or ends wins
                if (u[w] != v[w]) {
                    l = at + 8 * w + key_lcp(u[w], v[w]);
                    open = false;
                } else if (zero_byte(u[w]) < 8) {
                    l = at + 8 * w + zero_byte(u[w]);
                    open = false;
                }
            }
            if (l >= d + CODE_CAP) {
                l = d + CODE_CAP;
                open = false;
            }
        }
        todo = __ballot_sync(FULL, open);
    } while (__popc(todo) > 4);
    const uint32_t lane = threadIdx.x & 31;
    for (; todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1;
        const uint64_t ox = __shfl_sync(FULL, x.off, src), oh = __shfl_sync(FULL, h.off, src);
        const uint32_t lx = __shfl_sync(FULL, x.len, src), lh = __shfl_sync(FULL, h.len, src);
        const uint32_t cap = __shfl_sync(FULL, d, src) + CODE_CAP;
        uint32_t at = __shfl_sync(FULL, l, src);
        for (;; at += 256) {
            if (at >= cap) {
                at = cap;
                break;
            }
            const uint32_t p = at + 8 * lane;
            const uint64_t u = key8(chars, ox, lx, p), v = key8(chars, oh, lh, p);
            const uint32_t e = u != v ? key_lcp(u, v) : zero_byte(u);
            const uint32_t hit = __ballot_sync(FULL, e < 8);
            if (hit) {
                const int f = __ffs(hit) - 1;
                at = min(at + 8 * f + __shfl_sync(FULL, e, f), cap);
                break;
            }
        }
        if (lane == (uint32_t)src) l = at;
    }
    return l;
}

// The pseudo key of string x against pivot h, l their LCP, d the group's
// depth.
__device__ __forceinline__ uint64_t pseudo_key(const ArenaDev& a, StrRef x, StrRef h, uint32_t l, uint32_t d) {
    if (l >= d + CODE_CAP) return (uint64_t)CODE_MID << 48 | 0x010101010101ull;  // no end in sight
    const uint64_t bx = key8(a.chars, x.off, x.len, l), bh = key8(a.chars, h.off, h.len, l);
    const uint32_t xb = (uint32_t)(bx >> 56), hb = (uint32_t)(bh >> 56);
    if (xb == hb) return (uint64_t)CODE_MID << 48;  // both end: equal strings
    const uint32_t c = xb < hb ? l - d : CODE_TOP - (l - d);
    return (uint64_t)c << 48 | bx >> 16;
}

// Pseudo key of string x against pivot h of a group of depth d, and
// whether the comparison ended at the cap; every lane of the warp calls it.
struct PivotKey {
    uint64_t key;
    bool capped;
};
__device__ __forceinline__ PivotKey pivot_key(const ArenaDev& a, StrRef x, StrRef h, uint32_t d, bool active) {
    const uint32_t l = warp_lcp(a.chars, x, h, d, active);
    PivotKey r{0, false};
    if (active) {
        r.key = pseudo_key(a, x, h, l, d);
        r.capped = l >= d + CODE_CAP;
    }
    return r;
}

// Compare-exchange network on (grp, key, id) over the first P (a power of two)
// elements of a warp's 32 * I; element 32 * q + lane is item q of the lane.
template <int I>
__device__ __forceinline__ void warp_network(uint32_t P, uint32_t (&grp)[I], uint64_t (&key)[I], uint32_t (&id)[I]) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll 1
    for (uint32_t k = 2; k <= P; k <<= 1) {
#pragma unroll 1
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            if (I > 1 && j >= 32) {
#pragma unroll
                for (int q = 0; q < I; ++q) {
#pragma unroll
                    for (int r = q + 1; r < I; ++r) {
                        if ((uint32_t)(q ^ r) * 32 != j) continue;
                        const bool less = grp[r] < grp[q] || (grp[r] == grp[q] && (key[r] < key[q] || (key[r] == key[q] && id[r] < id[q])));
                        if (less == ((q * 32 & k) == 0)) {
                            const uint32_t tg = grp[q], to = id[q];
                            const uint64_t tk = key[q];
                            grp[q] = grp[r];
                            key[q] = key[r];
                            id[q] = id[r];
                            grp[r] = tg;
                            key[r] = tk;
                            id[r] = to;
                        }
                    }
                }
                continue;
            }
#pragma unroll
            for (int q = 0; q < I; ++q) {
                if (I > 1 && (uint32_t)q * 32 >= P) break;
                const uint64_t pk = __shfl_xor_sync(FULL, key[q], j);
                const uint32_t po = __shfl_xor_sync(FULL, id[q], j), pg = __shfl_xor_sync(FULL, grp[q], j);
                const bool want_min = (((q * 32 + lane) & k) == 0) == ((lane & j) == 0);
                const bool less = pg < grp[q] || (pg == grp[q] && (pk < key[q] || (pk == key[q] && po < id[q])));
                if (less == want_min) {
                    grp[q] = pg;
                    key[q] = pk;
                    id[q] = po;
                }
            }
        }
    }
}

// Groups of one warp, back to back in its n <= 32 * I elements.  An element
// holds the element at which its group starts (grp), the group's depth and
// kind, its own place pos (with its LCP at lcp[pos]), a string of the group
// and, unless kind is G_TIE or G_ID, the string's key.  On return the ids of
// each group are in order and every element but a group's first has its LCP
// with its predecessor (the depth itself for G_ID).
//
// All groups go through each round together: sort by (group, key, id), then
// every run of equal keys that has not ended becomes a group of its own and
// compares with its first string.
template <int I>
__device__ __forceinline__ void warp_groups(const ArenaDev& a, uint32_t n, uint32_t (&grp)[I], uint32_t (&dep)[I],
                                            uint32_t (&kind)[I], const uint32_t (&pos)[I], uint64_t (&key)[I],
                                            uint32_t (&id)[I], uint32_t* lcp) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t P = n <= 2 ? 2u : 1u << (32 - __clz(n - 1));
    static_assert(I <= 2, "places are 6 bits");
    uint32_t rs[I];  // start of the element's run
    bool unres[I];   // the run goes on
    bool sort = false;
#pragma unroll
    for (int q = 0; q < I; ++q) {
        const bool valid = q * 32 + lane < n;
        if (!valid) {
            grp[q] = 0xFFFFFFFFu;
            id[q] = 0xFFFFFFFFu;
            kind[q] = G_TIE;
        }
        if (kind[q] == G_TIE || kind[q] == G_ID) key[q] = 0;
        rs[q] = grp[q];
        unres[q] = valid && kind[q] == G_TIE;
        sort = sort || kind[q] != G_TIE;
    }
    sort = __any_sync(FULL, sort);
    for (;;) {
        if (sort) {
            warp_network<I>(P, grp, key, id);
            uint32_t heads[I];
            bool head[I];
#pragma unroll
            for (int q = 0; q < I; ++q) {
                const uint32_t e = q * 32 + lane;
                uint64_t qk = __shfl_up_sync(FULL, key[q], 1);
                if (I > 1 && q > 0) {
                    const uint64_t last = __shfl_sync(FULL, key[q > 0 ? q - 1 : 0], 31);
                    if (lane == 0) qk = last;
                }
                const bool valid = e < n, inner = valid && e != grp[q];
                const bool pseudo = kind[q] == G_PSEUDO;
                head[q] = !inner || qk != key[q];
                if (inner && kind[q] != G_TIE) {
                    if (kind[q] == G_ID) lcp[pos[q]] = dep[q];
                    else if (qk != key[q]) lcp[pos[q]] = group_lcp(qk, key[q], dep[q], pseudo);
                    else if (key_ended(key[q], pseudo)) lcp[pos[q]] = ref_of(a, id[q]).len;  // equal strings
                }
                heads[q] = __ballot_sync(FULL, head[q]);
            }
#pragma unroll
            for (int q = 0; q < I; ++q) {
                const uint32_t e = q * 32 + lane;
                const bool valid = e < n;
#pragma unroll
                for (int r = 0; r <= q; ++r) {
                    const uint32_t m = r < q ? heads[r] : heads[q] & ((2u << lane) - 1u);
                    if (m) rs[q] = r * 32 + 31u - __clz(m);
                }
                const bool next_head = lane < 31 ? (heads[q] >> (lane + 1) & 1u) != 0
                                                 : (q + 1 < I ? (heads[q + 1 < I ? q + 1 : 0] & 1u) != 0 : true);
                unres[q] = valid && kind[q] != G_ID && !(head[q] && next_head) &&
                           (kind[q] == G_TIE || !key_ended(key[q], kind[q] == G_PSEUDO));
                if (valid) grp[q] = unres[q] ? rs[q] : e;  // a resolved string stays at its place
            }
        }
        bool any = false;
#pragma unroll
        for (int q = 0; q < I; ++q) any = any || unres[q];
        if (!__any_sync(FULL, any)) return;
        // every unresolved run goes on against its first string, the one with
        // the longest string against that: where one common part is shared up
        // to different depths, the longest string likely shares the most of it
        // and leaves none of the others together (a chain of 64 strings: 6
        // rounds against any of them, 1 or 2 against the longest)
        StrRef x[I], h[I];
        uint32_t pv[I], best = 0;
#pragma unroll
        for (int q = 0; q < I; ++q) {
            x[q] = StrRef{0, 0};
            if (unres[q]) {
                x[q] = ref_of(a, id[q]);
                best = max(best, min(x[q].len, 0x3FFFFFFu) << 6 | (q * 32 + lane));
            }
        }
        best = __reduce_max_sync(FULL, best) & 63u;
        uint32_t best_run = __shfl_sync(FULL, rs[0], best & 31u);
        if (I > 1) {
            const uint32_t t = __shfl_sync(FULL, rs[I - 1], best & 31u);
            if (best >= 32) best_run = t;
        }
#pragma unroll
        for (int q = 0; q < I; ++q) pv[q] = unres[q] && rs[q] == best_run ? best : rs[q];
#pragma unroll
        for (int q = 0; q < I; ++q) {
            h[q] = StrRef{0, 0};
#pragma unroll
            for (int r = 0; r < I; ++r) {
                const uint64_t off = __shfl_sync(FULL, x[r].off, pv[q] & 31u);
                const uint32_t len = __shfl_sync(FULL, x[r].len, pv[q] & 31u);
                if (pv[q] >> 5 == (uint32_t)r) h[q] = StrRef{off, len};
            }
        }
        bool capped[I];
#pragma unroll
        for (int q = 0; q < I; ++q) capped[q] = false;
#pragma unroll 1
        for (int q = 0; q < I; ++q) {  // one copy of the comparison's code: warps are at different places in it
            StrRef qx = x[0], qh = h[0];
            uint32_t qd = dep[0], qt = kind[0], qr = pv[0];
            uint64_t qk = key[0];
            bool qu = unres[0];
#pragma unroll
            for (int r = 1; r < I; ++r)
                if (r == q) {
                    qx = x[r];
                    qh = h[r];
                    qd = dep[r];
                    qt = kind[r];
                    qr = pv[r];
                    qk = key[r];
                    qu = unres[r];
                }
            if (I > 1 && !__any_sync(FULL, qu)) continue;
            if (qt != G_TIE) qd = tie_depth(qk, qd, qt == G_PSEUDO);
            const bool cmp = qu && q * 32 + lane != qr;
            const PivotKey t = pivot_key(a, qx, qh, qd, cmp);
#pragma unroll
            for (int r = 0; r < I; ++r)
                if (r == q && qu) {
                    dep[r] = qd;
                    kind[r] = G_PSEUDO;
                    key[r] = cmp ? t.key : (uint64_t)CODE_MID << 48;
                    capped[r] = cmp && t.capped;
                }
        }
        // a run's pivot keeps to those that agree with it up to the cap
#pragma unroll
        for (int q = 0; q < I; ++q)
            for (uint32_t m = __ballot_sync(FULL, capped[q]); m; m &= m - 1) {
                const uint32_t f = __shfl_sync(FULL, pv[q], __ffs(m) - 1);
#pragma unroll
                for (int r = 0; r < I; ++r)
                    if (f == r * 32 + lane) key[r] |= 0x010101010101ull;
            }
        sort = true;
    }
}

// Segments of 2..32 strings: one warp each, four per CTA.
__global__ void __launch_bounds__(128) k_warp_segs(const __grid_constant__ SortState S, const SmallSeg* segs, uint32_t nseg) {
    for (uint32_t si = blockIdx.x * 4 + (threadIdx.x >> 5); si < nseg; si += gridDim.x * 4) {
        const uint32_t lane = threadIdx.x & 31;
        const SmallSeg seg = segs[si];
        const uint32_t* src = S.ord[seg.flags & F_PARITY];
        uint32_t id = 0;
        uint64_t key = 0;
        if (lane < seg.size) {
            id = src[seg.start + lane];
            if (seg.flags & F_ID) key = 0;
            else key = (seg.flags & F_KEYS) ? S.key[seg.flags & F_PARITY][seg.start + lane] : key8_of(S.a, id, seg.depth);
        }
        uint32_t grp1[1] = {0}, dep1[1] = {seg.depth}, kind1[1] = {(seg.flags & F_ID) ? (uint32_t)G_ID : (uint32_t)G_PLAIN};
        const uint32_t pos1[1] = {lane};
        uint64_t key1[1] = {key};
        uint32_t id1[1] = {id};
        warp_groups<1>(S.a, seg.size, grp1, dep1, kind1, pos1, key1, id1, S.lcp_out + seg.start);
        if (lane < seg.size) S.ord_out[seg.start + lane] = id1[0];
    }
}

// A group on the CTA's stack or the warps' list: positions [start, start +
// size) of the segment, packed with the kind.
__device__ __forceinline__ uint2 group_pack(uint32_t start, uint32_t size, uint32_t kind, uint32_t depth) {
    return make_uint2(start | (size - 1) << 12 | kind << 24, depth);
}
__device__ __forceinline__ uint32_t group_start(uint2 g) { return g.x & 0xFFFu; }
__device__ __forceinline__ uint32_t group_size(uint2 g) { return ((g.x >> 12) & 0xFFFu) + 1; }
__device__ __forceinline__ uint32_t group_kind(uint2 g) { return g.x >> 24; }

template <int CAP, int NT>
struct SegSmem {
    static constexpr int NW = NT / 32;
    static constexpr int NB = CAP <= 256 ? 1024 : CAP <= 1024 ? 2048 : 4096;  // buckets
    unsigned long long key[CAP];
    __align__(16) uint16_t cnt[NB + 8];  // bucket counts, then starts (the last one the group's size)
    uint32_t id[CAP];
    uint2 wl[CAP / 2];         // groups for the warps
    uint32_t tl[CAP / 2];      // the pass's buckets of 2..TINY_MAX strings
    uint2 stk[CAP / MID_MAX + 2];  // groups for the CTA
    // per pass: OR and AND of the warps' keys, the warps' counts, the LCP sums of the pivot's candidates
    unsigned long long orv[NW], andv[NW];
    uint32_t sum[NW], piv[8];
    BucketBits bits;
    uint32_t ns, nw, nt, claim;  // lengths of stk, wl and tl; groups of wl taken
};

// The keys of a group that goes deeper: pivot, then every string's pseudo key.
template <int CAP, int NT>
__device__ __forceinline__ void cta_pivot_keys(const SortState& S, SegSmem<CAP, NT>& M, uint32_t bs, uint32_t bn, uint32_t dep) {
    constexpr int NW = NT / 32, IPT = CAP / NT;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // the pivot: of 8 evenly spaced strings the one with the largest sum of LCPs
    // (256 bytes at most) with the others
    for (uint32_t c = w; c < 8; c += NW) {
        const StrRef x = ref_of(S.a, M.id[bs + c * bn / 8]);
        const uint64_t kx = key8(S.a.chars, x.off, x.len, dep + 8 * lane);
        uint32_t sum = 0;
#pragma unroll 4
        for (uint32_t q = 0; q < 8; ++q) {
            const StrRef y = ref_of(S.a, M.id[bs + q * bn / 8]);
            const uint64_t ky = key8(S.a.chars, y.off, y.len, dep + 8 * lane);
            const uint32_t e = kx != ky ? key_lcp(kx, ky) : 8u;
            const uint32_t hit = __ballot_sync(FULL, e < 8);
            const int f = hit ? __ffs(hit) - 1 : 0;
            const uint32_t ef = __shfl_sync(FULL, e, f);
            sum += hit ? 8 * f + ef : 256u;
        }
        if (lane == 0) M.piv[c] = sum << 3 | c;
    }
    __syncthreads();
    uint32_t best = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) best = max(best, M.piv[c]);
    const uint32_t pid = M.id[bs + (best & 7u) * bn / 8];
    const StrRef h = ref_of(S.a, pid);
#pragma unroll 1
    for (int j = 0; j < IPT; ++j) {
        const uint32_t i = threadIdx.x + j * NT;
        if (i - lane >= bn) break;  // the same for the whole warp
        const bool v = i < bn;
        StrRef x{0, 0};
        uint32_t oj = v ? M.id[bs + i] : 0u;
        if (v) x = ref_of(S.a, oj);
        const uint32_t l = warp_lcp(S.a.chars, x, h, dep, v);
        if (v) M.key[bs + i] = pseudo_key(S.a, x, h, l, dep);
    }
}

// The groups on the warps' list, claimed up to 8 at a time; as many of these
// together as fit into a warp's 64 elements.
template <int CAP, int NT>
__device__ __forceinline__ void warps_sort_groups(const SortState& S, SegSmem<CAP, NT>& M, uint32_t* lcp) {
    const uint32_t ng = M.nw, lane = threadIdx.x & 31, per = min(8u, 1 + ng / (NT / 16));
    for (;;) {
        uint32_t e0 = 0;
        if (lane == 0) e0 = atomicAdd(&M.claim, per);
        e0 = __shfl_sync(FULL, e0, 0);
        if (e0 >= ng) break;
        uint2 g = make_uint2(0, 0);
        uint32_t left = min(per, ng - e0), sz = 0;  // lane t < left: the t-th group still to be sorted
        if (lane < left) {
            g = M.wl[e0 + lane];
            sz = group_size(g);
        }
        while (left) {
            uint32_t end = sz;  // inclusive sums of the sizes
#pragma unroll
            for (int off = 1; off < 8; off <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL, end, off);
                if (lane >= (uint32_t)off) end += y;
            }
            const uint32_t take = __popc(__ballot_sync(FULL, lane < left && end <= 64));
            const uint32_t n = __shfl_sync(FULL, end, take - 1);
            uint32_t grp[2], dep[2], kind[2], pos[2], id[2];
            uint64_t key[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const uint32_t e = q * 32 + lane;
                uint32_t t = 0;  // the element's group
                for (uint32_t r = 0; r + 1 < take; ++r) t += e >= __shfl_sync(FULL, end, r);
                const uint32_t gx = __shfl_sync(FULL, g.x, t);
                grp[q] = __shfl_sync(FULL, end - sz, t);
                dep[q] = __shfl_sync(FULL, g.y, t);
                kind[q] = gx >> 24;
                pos[q] = (gx & 0xFFFu) + e - grp[q];
                id[q] = e < n ? M.id[pos[q]] : 0u;
                key[q] = e < n ? M.key[pos[q]] : 0ull;
            }
            warp_groups<2>(S.a, n, grp, dep, kind, pos, key, id, lcp);
#pragma unroll
            for (int q = 0; q < 2; ++q)
                if (q * 32 + lane < n) M.id[pos[q]] = id[q];
            left -= take;
            g.x = __shfl_down_sync(FULL, g.x, take);
            g.y = __shfl_down_sync(FULL, g.y, take);
            sz = __shfl_down_sync(FULL, sz, take);
            if (lane >= left) sz = 0;
        }
    }
}

// Whether a bucket of c out of n strings goes on by a pivot although its plain
// keys still differ: more than three in four together look like a chain of
// nested prefixes, from which passes over plain keys peel a byte or two each,
// a pivot pass nearly all.  (1000 strings with shared parts of random length:
// five plain passes of 5 us before the first pivot pass of 15.)
__device__ __forceinline__ bool chained(uint32_t c, uint32_t n) { return c > MID_MAX && 4 * c > 3 * n; }

// The first pass from the buckets' starts (cnt) on; br holds a string's bucket
// and its place there.  What bounds it is the shared memory's throughput: the
// counts, places and keys of random buckets take a wavefront for every two or
// three strings.  So counts are 16 bits wide, a string reads its bucket's start
// once, buckets join the list by one atomic per warp, and the LCPs are taken in
// sorted order, from neighbouring keys to neighbouring places (at the buckets'
// first strings, in the order of the input, they cost a random key and a
// scattered store each).  1e8 strings: 1.03 -> 1.00 ms, and 0.89 ms with the
// six blocks per SM that the smaller counts allow (seven or eight: 0.92).
// Inside the groups still to be sorted the LCPs written here are not yet right;
// sort_rest replaces them.
template <int CAP, int NT>
__device__ __forceinline__ void first_pass_rest(const SortState& S, SegSmem<CAP, NT>& M, uint32_t bn, uint32_t dep,
                                                uint32_t kind, const uint32_t (&o)[CAP / NT],
                                                const uint64_t (&k)[CAP / NT], const uint32_t (&br)[CAP / NT],
                                                uint32_t* lcp) {
    constexpr int IPT = CAP / NT;
    const uint32_t lane = threadIdx.x & 31;
    const bool all = M.bits.all != 0;
    bool bad = false;
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
        uint32_t s0 = 0, c = 0;  // its bucket's start and, for the first one there, size
        if (threadIdx.x + j * NT < bn) {
            const uint32_t b = br[j] & 0xFFFFu;
            s0 = M.cnt[b];
            const uint32_t at = s0 + (br[j] >> 16);
            if (at < bn) {  // only the counts' sum bounds a place, always so
                M.key[at] = k[j];
                M.id[at] = o[j];
                if (at == s0) c = M.cnt[b + 1] - s0;
            } else {
                bad = true;
            }
        }
        const bool tiny = c >= 2 && c <= TINY_MAX;
        const uint32_t peers = __ballot_sync(FULL, tiny);
        if (peers) {
            uint32_t at = 0;
            if (lane == (uint32_t)__ffs(peers) - 1) at = atomicAdd(&M.nt, __popc(peers));
            at = __shfl_sync(FULL, at, __ffs(peers) - 1);
            if (tiny) M.tl[at + __popc(peers & ((1u << lane) - 1u))] = s0 | c << 16;
        }
        if (c > TINY_MAX) {
            uint32_t gk = kind, gd = dep;
            if (kind == G_PLAIN && chained(c, bn)) gk = G_TIE;
            if (kind != G_ID && all) {  // one key in the bucket
                const bool ended = key_ended(k[j], false);
                gk = ended ? G_ID : G_TIE;
                gd = ended ? dep + key_end(k[j], false) : dep + 8;
            }
            const uint2 g = group_pack(s0, c, gk, gd);
            if (c <= MID_MAX) M.wl[atomicAdd(&M.nw, 1u)] = g;
            else M.stk[atomicAdd(&M.ns, 1u)] = g;
        }
    }
    if (bad) atomicExch(&S.counters[10], 1u);
    __syncthreads();
    // buckets of 2..TINY_MAX strings: insertion sort on (key, id), then the
    // runs that go deeper
    const uint32_t nt = M.nt;
    for (uint32_t e = threadIdx.x; e < nt; e += NT) {
        const uint32_t s0 = M.tl[e] & 0xFFFFu, c = M.tl[e] >> 16;
        uint32_t same = 0;  // neighbours that were found equal
        for (uint32_t x = 1; x < c; ++x) {
            const uint64_t kx = M.key[s0 + x];
            const uint32_t ox = M.id[s0 + x];
            uint32_t y = x;
            for (; y > 0; --y) {
                const uint64_t ky = M.key[s0 + y - 1];
                const uint32_t oy = M.id[s0 + y - 1];
                same |= ky == kx;
                if (ky < kx || (ky == kx && oy < ox)) break;
                M.key[s0 + y] = ky;
                M.id[s0 + y] = oy;
            }
            if (y != x) {
                M.key[s0 + y] = kx;
                M.id[s0 + y] = ox;
            }
        }
        if (!same) continue;
        uint64_t kp = M.key[s0];
        uint32_t r0 = 0;  // start of the run of equal keys
        for (uint32_t x = 1; x <= c; ++x) {
            const uint64_t kx = x < c ? M.key[s0 + x] : ~kp;
            if (kx == kp) continue;
            if (x - r0 > 1 && !key_ended(kp, false))
                M.wl[atomicAdd(&M.nw, 1u)] = group_pack(s0 + r0, x - r0, G_TIE, dep + 8);
            kp = kx;
            r0 = x;
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
        const uint32_t i = threadIdx.x + j * NT;
        if (i == 0 || i >= bn) continue;
        const uint64_t kp = M.key[i - 1], kx = M.key[i];
        if (kind == G_ID) lcp[i] = dep;
        else if (kp != kx) lcp[i] = dep + key_lcp(kp, kx);
        else if (key_ended(kx, false)) lcp[i] = dep + key_end(kx, false);  // equal strings
    }
}

// One bucket pass over the CTA's group at [bs, bs + bn): thread t holds its
// strings t, t + NT, ... (o) and their keys (k).  Every count in cnt is zero
// before and, unless FIRST, after.  FIRST: the whole segment, not yet in shared
// memory, with plain keys or ids.
template <int CAP, int NT, bool FIRST>
__device__ __forceinline__ void cta_pass(const SortState& S, SegSmem<CAP, NT>& M, uint32_t bs, uint32_t bn, uint32_t dep,
                                         uint32_t kind, const uint32_t (&o)[CAP / NT], const uint64_t (&k)[CAP / NT],
                                         uint32_t* lcp) {
    constexpr int NW = NT / 32, IPT = CAP / NT, NB = SegSmem<CAP, NT>::NB, PER = NB / NT;
    const ArenaDev& a = S.a;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t br[IPT];
    const bool pseudo = !FIRST && kind == G_PSEUDO;
    // the bits in which the keys differ
    uint64_t vo = 0, va = ~0ull;
#pragma unroll
    for (int j = 0; j < IPT; ++j)
        if (threadIdx.x + j * NT < bn) {
            const uint64_t t = level_key(k[j], pseudo);
            vo |= t;
            va &= t;
        }
    const uint32_t olo = __reduce_or_sync(FULL, (uint32_t)vo), ohi = __reduce_or_sync(FULL, (uint32_t)(vo >> 32));
    const uint32_t alo = __reduce_and_sync(FULL, (uint32_t)va);
    const uint32_t ahi = __reduce_and_sync(FULL, (uint32_t)(va >> 32));
    if (lane == 0) {
        M.orv[w] = (uint64_t)ohi << 32 | olo;
        M.andv[w] = (uint64_t)ahi << 32 | alo;
    }
    __syncthreads();
    if (w == 0) {
        uint64_t x = lane < NW ? M.orv[lane] : 0ull, y = lane < NW ? M.andv[lane] : ~0ull;
        const uint32_t dl = __reduce_or_sync(FULL, (uint32_t)x) ^ __reduce_and_sync(FULL, (uint32_t)y);
        const uint32_t dh = __reduce_or_sync(FULL, (uint32_t)(x >> 32)) ^ __reduce_and_sync(FULL, (uint32_t)(y >> 32));
        if (lane == 0) {
            constexpr uint32_t most = 31u - (uint32_t)__builtin_clz(NB);
            const uint64_t diff = (uint64_t)dh << 32 | dl;
            M.bits.nruns = 0;
            if (diff)
                bucket_bits(M.bits, diff, pseudo ? most : min(32u - (uint32_t)__clz(bn - 1) + 1u, most));
        }
    }
    __syncthreads();
    if (M.bits.nruns == 0) {  // one key: equal strings, or the group goes deeper
        if (FIRST) {
#pragma unroll
            for (int j = 0; j < IPT; ++j) {
                const uint32_t i = threadIdx.x + j * NT;
                if (i < bn) M.id[i] = o[j];
            }
        }
        if (threadIdx.x == 0) {
            const uint64_t k0 = k[0];
            const uint2 g = key_ended(k0, pseudo) ? group_pack(bs, bn, G_ID, ref_of(a, o[0]).len)
                                                  : group_pack(bs, bn, G_TIE, tie_depth(k0, dep, pseudo));
            if (bn <= MID_MAX) M.wl[M.nw++] = g;
            else M.stk[M.ns++] = g;
        }
        __syncthreads();
        return;
    }
    {
        const uint32_t lo = M.bits.lo, nr = M.bits.nruns;
        uint32_t x[IPT];
#pragma unroll
        for (int j = 0; j < IPT; ++j) {
            x[j] = (uint32_t)(k[j] >> lo);
            br[j] = 0;
        }
        for (uint32_t r = 0; r < nr; ++r) {
            const uint32_t sh = M.bits.sh[r], mask = M.bits.mask[r];
            if (M.bits.wide) {
#pragma unroll
                for (int j = 0; j < IPT; ++j) br[j] |= (uint32_t)(k[j] >> (lo + sh)) & mask;
            } else {
#pragma unroll
                for (int j = 0; j < IPT; ++j) br[j] |= (x[j] >> sh) & mask;
            }
        }
    }
    // counts; br: the bucket and, above it, the place inside it
#pragma unroll
    for (int j = 0; j < IPT; ++j)
        if (threadIdx.x + j * NT < bn) {
            const uint32_t half = (br[j] & 1u) * 16;
            br[j] |= atomicAdd(reinterpret_cast<uint32_t*>(M.cnt) + (br[j] >> 1), 1u << half) >> half << 16;
        }
    __syncthreads();
    {
        uint32_t v[PER], sum = 0;
#pragma unroll
        for (int q = 0; q < PER; q += 8) {
            const uint4 c = *reinterpret_cast<const uint4*>(&M.cnt[threadIdx.x * PER + q]);
            const uint32_t p[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                v[q + 2 * h] = p[h] & 0xFFFFu;
                v[q + 2 * h + 1] = p[h] >> 16;
                sum += v[q + 2 * h] + v[q + 2 * h + 1];
            }
        }
        uint32_t x = sum;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, x, off);
            if (lane >= (uint32_t)off) x += y;
        }
        if (lane == 31) M.sum[w] = x;
        __syncthreads();
        uint32_t run = x - sum;
#pragma unroll
        for (int q = 0; q < NW; ++q)
            if ((uint32_t)q < w) run += M.sum[q];
#pragma unroll
        for (int q = 0; q < PER; q += 8) {
            uint32_t p[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                p[h] = run | (run + v[q + 2 * h]) << 16;
                run += v[q + 2 * h] + v[q + 2 * h + 1];
            }
            *reinterpret_cast<uint4*>(&M.cnt[threadIdx.x * PER + q]) = make_uint4(p[0], p[1], p[2], p[3]);
        }
        if (threadIdx.x == NT - 1) M.cnt[NB] = (uint16_t)run;
    }
    __syncthreads();
    if (FIRST) {
        first_pass_rest<CAP, NT>(S, M, bn, dep, kind, o, k, br, lcp);
        return;
    }
    // places (a thread holds its strings, so the group is permuted in
    // place); only the counts' sum bounds a place, never taken else
    bool bad = false;
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
        if (threadIdx.x + j * NT >= bn) continue;
        const uint32_t at = M.cnt[br[j] & 0xFFFFu] + (br[j] >> 16);
        if (at >= bn) {
            bad = true;
            continue;
        }
        M.key[bs + at] = k[j];
        M.id[bs + at] = o[j];
    }
    if (bad) atomicExch(&S.counters[10], 1u);
    __syncthreads();
    // each bucket's first string: the LCP with the bucket before (any
    // of its strings), and who sorts the bucket
    const bool all = M.bits.all != 0, mixed = pseudo && M.bits.mixed;
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
        if (threadIdx.x + j * NT >= bn || (br[j] >> 16) != 0) continue;
        const uint32_t b = br[j] & 0xFFFFu, s0 = M.cnt[b], c = M.cnt[b + 1] - s0;
        if (s0) {
            uint64_t kp = M.key[bs + s0 - 1], kn = k[j];
            if (mixed) {  // the codes next to the boundary: the last of the bucket before, this one's first
                const uint32_t bp = bucket_of_key(M.bits, kp);
                for (uint32_t x = s0 - 1; x > 0 && bucket_of_key(M.bits, M.key[bs + x - 1]) == bp; --x)
                    kp = max(kp, (uint64_t)M.key[bs + x - 1]);
                for (uint32_t x = 0; x < c; ++x) kn = min(kn, (uint64_t)M.key[bs + s0 + x]);
            }
            lcp[bs + s0] = kind == G_ID ? dep : group_lcp(kp, kn, dep, pseudo);
        }
        if (c < 2) continue;
        if (c <= TINY_MAX) {
            M.tl[atomicAdd(&M.nt, 1u)] = s0 | c << 16;
            continue;
        }
        uint32_t gk = kind, gd = dep;
        if (kind == G_PLAIN && chained(c, bn)) gk = G_TIE;
        if (kind != G_ID && all) {  // one key in the bucket
            const bool ended = key_ended(k[j], pseudo);
            gk = ended ? G_ID : G_TIE;
            gd = ended ? ref_of(a, o[j]).len : tie_depth(k[j], dep, pseudo);
        }
        const uint2 g = group_pack(bs + s0, c, gk, gd);
        if (c <= MID_MAX) M.wl[atomicAdd(&M.nw, 1u)] = g;
        else M.stk[atomicAdd(&M.ns, 1u)] = g;
    }
    __syncthreads();
    // buckets of 2..TINY_MAX strings: insertion sort on (key, id), then
    // the neighbours' LCPs and the runs that go deeper
    const uint32_t nt = M.nt;
    for (uint32_t e = threadIdx.x; e < nt; e += NT) {
        const uint32_t s0 = bs + (M.tl[e] & 0xFFFFu), c = M.tl[e] >> 16;
        for (uint32_t x = 1; x < c; ++x) {
            const uint64_t kx = M.key[s0 + x];
            const uint32_t ox = M.id[s0 + x];
            uint32_t y = x;
            for (; y > 0; --y) {
                const uint64_t ky = M.key[s0 + y - 1];
                const uint32_t oy = M.id[s0 + y - 1];
                if (ky < kx || (ky == kx && oy < ox)) break;
                M.key[s0 + y] = ky;
                M.id[s0 + y] = oy;
            }
            M.key[s0 + y] = kx;
            M.id[s0 + y] = ox;
        }
        if (kind == G_ID) {
            for (uint32_t x = 1; x < c; ++x) lcp[s0 + x] = dep;
            continue;
        }
        uint64_t kp = M.key[s0];
        uint32_t r0 = 0;  // start of the run of equal keys
        for (uint32_t x = 1; x <= c; ++x) {
            const uint64_t kx = x < c ? M.key[s0 + x] : ~kp;
            if (kx == kp) continue;
            if (x - r0 > 1) {
                if (key_ended(kp, pseudo)) {
                    const uint32_t len = ref_of(a, M.id[s0 + r0]).len;
                    for (uint32_t y = r0 + 1; y < x; ++y) lcp[s0 + y] = len;
                } else {
                    M.wl[atomicAdd(&M.nw, 1u)] = group_pack(s0 + r0, x - r0, G_TIE, tie_depth(kp, dep, pseudo));
                }
            }
            if (x < c) lcp[s0 + x] = group_lcp(kp, kx, dep, pseudo);
            kp = kx;
            r0 = x;
        }
    }
    // the next pass counts from zero
#pragma unroll
    for (int q = 0; q < PER; q += 8)
        *reinterpret_cast<uint4*>(&M.cnt[8 * threadIdx.x + q * NT]) = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    if (threadIdx.x == 0) M.nt = 0;  // pushed to again only after the next pass's barriers
}

// Everything after a segment's first pass: the CTA's stack of groups, then the
// warps' list.
template <int CAP, int NT>
__device__ __noinline__ void sort_rest(const SortState& S, uint32_t* lcp) {
    constexpr int IPT = CAP / NT, PER = SegSmem<CAP, NT>::NB / NT;
    extern __shared__ __align__(16) unsigned char smem[];
    SegSmem<CAP, NT>& M = *reinterpret_cast<SegSmem<CAP, NT>*>(smem);
#pragma unroll
    for (int q = 0; q < PER; q += 8)
        *reinterpret_cast<uint4*>(&M.cnt[8 * threadIdx.x + q * NT]) = make_uint4(0u, 0u, 0u, 0u);
    if (threadIdx.x == 0) M.nt = 0;
    __syncthreads();
    while (M.ns) {
        const uint2 g = M.stk[M.ns - 1];
        const uint32_t bs = group_start(g), bn = group_size(g), dep = g.y;
        uint32_t kind = group_kind(g);
        __syncthreads();
        if (threadIdx.x == 0) --M.ns;  // read again only after the pass's barriers
        if (kind == G_TIE) {
            cta_pivot_keys<CAP, NT>(S, M, bs, bn, dep);
            kind = G_PSEUDO;  // a thread reads back only the keys it wrote
        }
        uint32_t o[IPT];
        uint64_t k[IPT];
#pragma unroll
        for (int j = 0; j < IPT; ++j) {
            const uint32_t i = threadIdx.x + j * NT;
            o[j] = i < bn ? M.id[bs + i] : 0u;
            k[j] = i < bn ? (kind == G_ID ? o[j] : M.key[bs + i]) : 0ull;
        }
        cta_pass<CAP, NT, false>(S, M, bs, bn, dep, kind, o, k, lcp);
    }
    if (M.nw) warps_sort_groups<CAP, NT>(S, M, lcp);
}

template <int CAP, int NT>
__global__ void __launch_bounds__(NT, CAP >= 4096 ? 2 : CAP >= 1024 ? 6 : 8) k_seg_sort(const __grid_constant__ SortState S,
                                                                                       const SmallSeg* segs,
                                                                                       uint32_t nseg) {
    constexpr int IPT = CAP / NT, PER = SegSmem<CAP, NT>::NB / NT;
    extern __shared__ __align__(16) unsigned char smem[];
    SegSmem<CAP, NT>& M = *reinterpret_cast<SegSmem<CAP, NT>*>(smem);
    for (uint32_t bi = blockIdx.x; bi < nseg; bi += gridDim.x) {
        const SmallSeg seg = segs[bi];
        const uint32_t start = seg.start, size = seg.size;
        uint32_t* lcp = S.lcp_out + start;
        uint32_t o[IPT];
        uint64_t k[IPT];
        const uint32_t* src = S.ord[seg.flags & F_PARITY] + start;
        const unsigned long long* ksrc = S.key[seg.flags & F_PARITY] + start;
#pragma unroll
        for (int j = 0; j < IPT; ++j) {
            const uint32_t i = threadIdx.x + j * NT;
            o[j] = i < size ? src[i] : 0u;
            k[j] = i < size && (seg.flags & F_KEYS) ? ksrc[i] : 0ull;
        }
        if (seg.flags & F_ID) {
#pragma unroll
            for (int j = 0; j < IPT; ++j) k[j] = o[j];
        } else if (!(seg.flags & F_KEYS)) {
#pragma unroll
            for (int j = 0; j < IPT; ++j)
                if (threadIdx.x + j * NT < size) k[j] = key8_of(S.a, o[j], seg.depth);
        }
#pragma unroll
        for (int q = 0; q < PER; q += 8)
            *reinterpret_cast<uint4*>(&M.cnt[8 * threadIdx.x + q * NT]) = make_uint4(0u, 0u, 0u, 0u);
        if (threadIdx.x == 0) M.ns = M.nw = M.nt = M.claim = 0;
        cta_pass<CAP, NT, true>(S, M, 0, size, seg.depth, (seg.flags & F_ID) ? G_ID : G_PLAIN, o, k, lcp);
        if (M.ns | M.nw) sort_rest<CAP, NT>(S, lcp);
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < size; i += NT) S.ord_out[start + i] = M.id[i];
        __syncthreads();  // shared memory is reused by the next segment
    }
}

template <int CAP, int NT>
static int launch_seg_sort(const SortState& S, const SmallSeg* segs, uint32_t n, const char* name, cudaStream_t st) {
    if (!n) return DSSS_OK;
    constexpr size_t shm = sizeof(SegSmem<CAP, NT>);
    static std::atomic<uint64_t> configured{0};
    DSSS_TRY(set_smem_once(configured, k_seg_sort<CAP, NT>, (int)shm));
    DSSS_LAUNCH(name, st, k_seg_sort<CAP, NT><<<n, NT, shm, st>>>(S, segs, n));
    DSSS_CUDA(cudaGetLastError());
    return DSSS_OK;
}


// ------------------------------------------------------------------ host ----
// One block: per large segment its first tile (exclusive prefix over the
// list), the total into counters[8]; resets the next list's counts.
__global__ void __launch_bounds__(1024) k_seg_offsets(SortState S, const Seg* segs, uint32_t nseg) {
    __shared__ uint32_t wsum[32];
    const uint32_t per = (nseg + 1023) / 1024;
    const uint32_t b = min(nseg, threadIdx.x * per), e = min(nseg, b + per);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t tt = 0;
    for (uint32_t i = b; i < e; ++i) tt += (segs[i].size + LT_TILE - 1) / LT_TILE;
    uint32_t x = tt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    uint32_t rt = x - tt, total = 0;
    for (int k = 0; k < 32; ++k) {
        if (k < w) rt += wsum[k];
        total += wsum[k];
    }
    for (uint32_t i = b; i < e; ++i) {
        S.tile0[i] = rt;
        rt += (segs[i].size + LT_TILE - 1) / LT_TILE;
    }
    if (threadIdx.x == 0) {
        const bool over = total > S.cap_tiles;
        S.counters[8] = over ? 0u : total;  // nothing runs past the plan; the guard stops the loop
        if (over) S.counters[10] = 1;
        S.counters[0] = 0;   // large segments of the next pass
        S.counters[11] = 0;  // of them, without keys or with a pivot pass
    }
}

static uint32_t clamp_small_max(uint32_t m) {
    if (m == 0) m = (uint32_t)tune(TUNE_SORT_SMALL_MAX);
    return (m == 0 || m > (uint32_t)bin_cap(NBINS - 1)) ? (uint32_t)bin_cap(NBINS - 1) : (m < 2 ? 2 : m);
}

// Tables of the passes: per possible large segment its record twice and three
// rows of D words.  Large segments are disjoint and hold more than small_max
// strings each, so the strings bound their number (and that of a bin's small
// ones), whatever the number of parts.  The rows take 3 bytes per string at the
// default cutoff, 12 at 1024 and 48 at 256; below that a segment needs no wide
// digit.  (Digits of 8 bits at 256: 12 bytes, but 32e6 strings of D/N 0.25 took
// 6.8 ms instead of 5.4.)
void layout_sort(Carve& c, SortLayout& L, uint64_t n, uint32_t p, uint32_t small_max) {
    small_max = clamp_small_max(small_max);
    uint64_t N = n ? n : 1;
    L.small_max = small_max;
    L.ord[0] = c.take<uint32_t>(N);
    L.ord[1] = c.take<uint32_t>(N);
    L.key[0] = c.take<unsigned long long>(N);
    L.key[1] = c.take<unsigned long long>(N);
    L.cap_large = N / (small_max + 1) + 1;
    L.cap_tiles = N / LT_TILE + L.cap_large + 1;
    L.large[0] = c.take<unsigned char>(L.cap_large * sizeof(Seg));
    L.large[1] = c.take<unsigned char>(L.cap_large * sizeof(Seg));
    for (int b = 0; b < NBINS; ++b) {
        L.cap_small[b] = N / (b ? bin_cap(b - 1) + 1 : 2) + 1;
        L.small[b] = c.take<unsigned char>(L.cap_small[b] * sizeof(SmallSeg));
    }
    L.tile0 = c.take<uint32_t>(L.cap_large);
    L.dbits = small_max >= 256 ? DIGIT_BITS_MAX : 8;
    const uint64_t D = 1ull << L.dbits;
    L.hist = c.take<uint32_t>(L.cap_large * D);
    L.bucket = c.take<uint32_t>(L.cap_large * (D + 1));
    L.cursor = c.take<uint32_t>(L.cap_large * D);
    L.counters = c.take<uint32_t>(16);
    L.pb = c.take<uint64_t>(p + 1);
}

int sort_strings(const SortLayout& L, ArenaDev& a, uint64_t n, uint32_t p, const uint64_t* pb_host,
                 const uint32_t* ids_in, uint32_t* ord_out, uint32_t* lcp_out, uint32_t* pin, cudaStream_t st,
                 ulonglong2* handles, const uint32_t* seg_depth) {
    if (n == 0) return DSSS_OK;
    SortState S;
    S.a = a;
    S.ord[0] = L.ord[0];
    S.ord[1] = L.ord[1];
    S.key[0] = L.key[0];
    S.key[1] = L.key[1];
    S.ord_out = ord_out;
    S.lcp_out = lcp_out;
    Seg* large[2] = {(Seg*)L.large[0], (Seg*)L.large[1]};
    S.large[0] = large[0];
    S.large[1] = large[1];
    for (int b = 0; b < NBINS; ++b) {
        S.small[b] = (SmallSeg*)L.small[b];
        S.cap_small[b] = L.cap_small[b];
    }
    S.tile0 = L.tile0;
    S.hist = L.hist;
    S.bucket = L.bucket;
    S.cursor = L.cursor;
    S.dbits = L.dbits;
    S.counters = L.counters;
    S.small_max = L.small_max;
    S.pivot = tune(TUNE_SORT_PIVOT) ? 1u : 0u;
    S.n = n;
    S.cap_large = L.cap_large;
    S.cap_tiles = L.cap_tiles;
    S.seg_depth = seg_depth;
    // the first lists' sizes follow from the bounds: nothing to read back
    uint32_t nlarge = 0, nsmall[NBINS] = {};
    for (uint32_t q = 0; q < p; ++q) {
        const uint64_t size = pb_host[q + 1] - pb_host[q];
        if (size > S.small_max) ++nlarge;
        else if (size > 1) ++nsmall[bin_of((uint32_t)size)];
    }
    const bool all_large = !nsmall[0] && !nsmall[1] && !nsmall[2] && !nsmall[3];
    S.iota = !ids_in && all_large;
    static std::atomic<uint64_t> scatter_configured{0};
    DSSS_TRY(set_smem_once(scatter_configured, k_scatter, (int)SCATTER_SMEM));
    DSSS_CUDA(cudaMemsetAsync(L.counters, 0, 16 * sizeof(uint32_t), st));
    if (!S.iota) DSSS_LAUNCH("k_init_ids", st, k_init_ids<<<grid_for(n, 256), 256, 0, st>>>(S.ord[0], ids_in, n));
    const bool one = p == 1 && pb_host[0] == 0 && pb_host[1] == n;
    if (!one) DSSS_CUDA(cudaMemcpyAsync(L.pb, pb_host, (p + 1) * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
    DSSS_LAUNCH("k_init_segs", st, k_init_segs<<<grid_for(p, 128), 128, 0, st>>>(S, one ? nullptr : L.pb, p));
    DSSS_CUDA(cudaGetLastError());
    int cur = 0;
    uint32_t guard = 0;
    // whether the list holds a segment without keys (the first pass, a pivot
    // pass, equal strings): only then the passes that make keys run
    bool keyless = true;
    uint64_t rows = 0;  // zeroed rows of hist; a pass leaves those it uses zero again
    while (nlarge) {
        if (++guard > (1u << 24)) return fail(DSSS_EDEVICE, "string sort made no progress");
        if (nlarge > L.cap_large) return fail(DSSS_EDEVICE, "string sort: large-segment list overflow");
        if (nlarge > rows) {
            // for the segments there are, with room for the next passes' (all
            // rows of 1e8 strings are 100 MB, 1.6 GB at a cutoff of 256)
            const uint64_t to = std::min<uint64_t>(L.cap_large, std::max<uint64_t>(4ull * nlarge, 256));
            DSSS_CUDA(cudaMemsetAsync(L.hist + (rows << L.dbits), 0, ((to - rows) << L.dbits) * sizeof(uint32_t), st));
            rows = to;
        }
        Seg* segs = large[cur];
        Seg* next = large[cur ^ 1];
        // an upper bound for the grids (kernels exit past the real count)
        const unsigned tiles = (unsigned)std::min<uint64_t>(L.cap_tiles, n / LT_TILE + nlarge + 1);
        DSSS_LAUNCH("k_seg_offsets", st, k_seg_offsets<<<1, 1024, 0, st>>>(S, segs, nlarge));
        if (keyless) {
            DSSS_LAUNCH("k_spec", st, k_spec<<<std::min<uint32_t>(nlarge, 148 * 16), 256, 0, st>>>(S, segs, nlarge));
            DSSS_LAUNCH("k_prefix", st, k_prefix<<<tiles, LT_NT, 0, st>>>(S, segs, nlarge));
            if (guard > 1) DSSS_LAUNCH("k_pivot", st, k_pivot<<<tiles, LT_NT, 0, st>>>(S, segs, nlarge));
            DSSS_LAUNCH("k_keys_diff", st, k_keys_diff<<<tiles, LT_NT, 0, st>>>(S, segs, nlarge));
        }
        DSSS_LAUNCH("k_hist", st, k_hist<<<tiles, LT_NT, 0, st>>>(S, segs, nlarge));
        if (S.dbits == 8) DSSS_LAUNCH("k_seg_scan", st, k_seg_scan<1><<<nlarge, 256, 0, st>>>(S, segs, next));
        else DSSS_LAUNCH("k_seg_scan", st, k_seg_scan<4><<<nlarge, 256, 0, st>>>(S, segs, next));
        DSSS_LAUNCH("k_scatter", st, k_scatter<<<tiles, SC_NT, SCATTER_SMEM, st>>>(S, segs, nlarge));
        DSSS_CUDA(cudaGetLastError());
        DSSS_CUDA(cudaMemcpyAsync(pin, L.counters, 16 * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
        DSSS_CUDA(cudaStreamSynchronize(st));
        nlarge = pin[0];
        keyless = pin[11] != 0;
        if (pin[10]) return fail(DSSS_EDEVICE, "string sort: internal consistency guard tripped");
        cur ^= 1;
        S.iota = 0;
        if (nlarge && keyless && handles && !a.h) {
            // keys are gathered from here on: one 16-byte read per string
            DSSS_TRY(make_handles(a, handles, st));
            a.h = S.a.h = handles;
        }
        for (int b = 0; b < NBINS; ++b) nsmall[b] = pin[1 + b];
    }
    for (int b = 0; b < NBINS; ++b)
        if (nsmall[b] > L.cap_small[b]) return fail(DSSS_EDEVICE, "string sort: small-segment list overflow");
    if (nsmall[0]) {
        DSSS_LAUNCH("k_warp_segs", st, k_warp_segs<<<(nsmall[0] + 3) / 4, 128, 0, st>>>(S, S.small[0], nsmall[0]));
        DSSS_CUDA(cudaGetLastError());
    }
    DSSS_TRY((launch_seg_sort<256, 128>(S, S.small[1], nsmall[1], "k_seg_sort256", st)));
    DSSS_TRY((launch_seg_sort<1024, 256>(S, S.small[2], nsmall[2], "k_seg_sort1024", st)));
    DSSS_TRY((launch_seg_sort<4096, 512>(S, S.small[3], nsmall[3], "k_seg_sort4096", st)));
    DSSS_CUDA(cudaMemcpyAsync(pin, L.counters, 16 * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    DSSS_CUDA(cudaStreamSynchronize(st));
    if (pin[10]) return fail(DSSS_EDEVICE, "string sort: internal consistency guard tripped");
    return DSSS_OK;
}

}  // namespace dsss
