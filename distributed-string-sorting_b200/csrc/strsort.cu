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
//   hist     : warp-aggregated 256-bin histogram of that byte per 4096-element tile;
//   scan     : per segment, bucket starts and per-tile offsets (chunked);
//   scatter  : stable scatter of ids (and keys of children that stay large).
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

constexpr int LT_NT = 256, LT_IPT = 8, LT_TILE = LT_NT * LT_IPT;
constexpr int CHUNK_TILES = 32;
constexpr uint32_t PREFIX_CAP = 256;
// F_KEYS: the key array holds the segment's keys at Seg.depth; F_PIVOT: the
// next pass is a pivot pass; F_PSEUDO: the keys are pivot pseudo keys.
constexpr uint32_t F_PARITY = 1u, F_KEYS = 2u, F_PIVOT = 4u, F_PSEUDO = 8u;
constexpr uint32_t PIVOT_CAP = 127;  // pseudo key byte 0 holds codes 0 .. 2 * PIVOT_CAP

struct Seg {
    uint32_t start, size, depth, flags;
    uint32_t newdepth;
    uint32_t first_digit;
    unsigned long long diff;
    // speculated common-prefix depth + 1 (0: none) and the OR of key ^ key0
    // over the keys k_prefix wrote at that depth (segments without keys)
    uint32_t spec;
    // this pass's digit: the key byte at the first difference (nspl = 0), or
    // the bucket among nspl sampled splitters (table spl_slot; bucket-start
    // LCPs into the fix list from fix0)
    uint32_t nspl;
    unsigned long long spec_diff;
    uint32_t spl_slot, fix0;
    // pivot pass: the pivot's string id (NO_PIVOT: the segment's first string)
    uint32_t piv, pad;
    // OR and AND of the keys the previous pass's scatter wrote for this
    // segment (children with keys, when the child table is kept): the bits
    // that differ among its keys are kor ^ kand
    unsigned long long kor, kand;
};

// Sampled splitters.  Where the key byte at a large segment's first
// difference takes few values (letters, DNA), a byte digit splits the segment
// only a few ways per pass.  Instead, the distinct keys among every 8th of an
// evenly spaced, sorted sample of SPL_SAMPLE keys become m <= 255 splitters.
// With more than SPL_EQ_MAX of them a key's bucket is the number of
// splitters below it (about 1/256 of the segment each; two splitters are
// keys of the segment in different buckets, so it splits).  With fewer (few
// distinct keys: frequent ones), bucket 2j holds the keys between splitters
// j-1 and j and bucket 2j+1 the keys equal to splitter j, so every sampled
// key lands in an equality bucket and the others elsewhere.  Equal keys
// always share a bucket, and two neighbours across a bucket boundary have
// different keys, so their LCP is the depth plus the LCP of the two keys; it
// is written once the final order is known (k_lcp_fix).
constexpr int SPL_SAMPLE = 2048;
constexpr uint32_t SPL_MAX = 255, SPL_STRIDE = 256, SPL_EQ_MAX = 127;
constexpr uint32_t SPL_MIN_FLOOR = 4096;  // smallest sort_split_min other than 0 (off)
constexpr uint32_t FIX_NONE = 0xFFFFFFFFu;
constexpr uint32_t NO_PIVOT = 0xFFFFFFFFu;

constexpr int NBINS = 4;
__host__ __device__ constexpr int bin_cap(int b) { return b == 0 ? 32 : b == 1 ? 256 : b == 2 ? 1024 : 4096; }
__device__ __forceinline__ int bin_of(uint32_t size) {
    return size <= 32 ? 0 : size <= 256 ? 1 : size <= 1024 ? 2 : 3;
}

// Counters block (device): [0] n_large_next, [1..4] n_small per bin, [5]
// fix-list slots reserved, [6] splitter tables of the pass, [8] total tiles,
// [9] total chunks, [10] error flag (a guard tripped), [11] large segments of
// the next pass without keys or with a pivot pass.
struct SortState {
    ArenaDev a;
    uint32_t* ord[2];
    unsigned long long* key[2];
    uint32_t* ord_out;
    uint32_t* lcp_out;
    Seg* large[2];
    Seg* small[NBINS];
    uint32_t* tile0;
    uint32_t* chunk0;
    uint32_t* tmp_counts;
    uint32_t* tile_hist;
    uint32_t* chunk_pre;
    uint32_t* bucket;  // 257 per large segment
    uint32_t* counters;
    // child table (optional, 256 per large segment): the next list's slot of
    // digit d's child when it is large and keeps the keys (~0u otherwise); the
    // scatter then folds the keys it writes into that child's kor / kand
    uint32_t* child;
    Seg* nxt;  // the next pass's list (the scatter's children)
    uint32_t small_max;
    uint32_t pivot;  // pivot passes enabled
    uint32_t bits;   // plain keys split on their top differing bits: 0 never, 1 always, 2 on narrow bytes
    uint32_t first;     // the first pass over the arena (host-driven passes)
    uint64_t cap_large, cap_small, cap_tiles, cap_chunks;
    // sampled splitters: segments of at least split_min strings (0: never);
    // cap_spl tables of SPL_STRIDE keys per pass; the fix list holds
    // (position, depth) pairs of bucket starts whose LCP k_lcp_fix writes
    uint32_t split_min;
    const uint32_t* seg_depth;  // optional: each segment's shared prefix length
    unsigned long long* spl;
    uint32_t* fix;
    uint64_t cap_spl, cap_fix;
};

__device__ __forceinline__ uint32_t find_seg(const uint32_t* first, uint32_t nseg, uint32_t t) {
    // last s with first[s] <= t
    uint32_t lo = 0, hi = nseg;
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (first[mid] <= t) lo = mid;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ void push_small(const SortState& S, uint32_t start, uint32_t size, uint32_t depth,
                                           uint32_t flags) {
    int b = bin_of(size);
    uint32_t slot = atomicAdd(&S.counters[1 + b], 1u);
    if (slot >= S.cap_small) {
        atomicExch(&S.counters[10], 1u);
        return;
    }
    Seg s;
    s.start = start;
    s.size = size;
    s.depth = depth;
    s.flags = flags;
    s.newdepth = 0xFFFFFFFFu;
    s.first_digit = 0;
    s.diff = 0;
    s.spec = 0;
    s.nspl = 0;
    s.spl_slot = 0;
    s.fix0 = 0;
    s.piv = NO_PIVOT;
    s.pad = 0;
    s.spec_diff = 0;
    s.kor = 0;
    s.kand = ~0ull;
    S.small[b][slot] = s;
}

// Returns the segment's slot in dst (~0u when the list is full).
__device__ __forceinline__ uint32_t push_large(const SortState& S, Seg* dst, uint32_t start, uint32_t size,
                                               uint32_t depth, uint32_t flags) {
    uint32_t slot = atomicAdd(&S.counters[0], 1u);
    if (slot >= S.cap_large) {
        atomicExch(&S.counters[10], 1u);
        return 0xFFFFFFFFu;
    }
    if (!(flags & F_KEYS) || (flags & F_PIVOT)) atomicAdd(&S.counters[11], 1u);
    Seg s;
    s.start = start;
    s.size = size;
    s.depth = depth;
    s.flags = flags;
    s.newdepth = 0xFFFFFFFFu;
    s.first_digit = 0;
    s.diff = 0;
    s.spec = 0;
    s.nspl = 0;
    s.spl_slot = 0;
    s.fix0 = 0;
    s.piv = NO_PIVOT;
    s.pad = 0;
    s.spec_diff = 0;
    s.kor = 0;
    s.kand = ~0ull;
    dst[slot] = s;
    return slot;
}

// ------------------------------------------------------------------ init ----
__global__ void k_init_ids(uint32_t* ord, const uint32_t* in, uint64_t n) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) ord[i] = in ? in[i] : (uint32_t)i;
}

__global__ void k_init_segs(SortState S, const uint64_t* pb, uint32_t p) {
    uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= p) return;
    uint32_t start = (uint32_t)pb[q], size = (uint32_t)(pb[q + 1] - pb[q]);
    if (size == 0) return;
    S.lcp_out[start] = 0;
    if (size == 1) {
        S.ord_out[start] = S.ord[0][start];
        return;
    }
    // a segment whose strings are known to share their first bytes starts there
    const uint32_t d = S.seg_depth ? S.seg_depth[q] : 0u;
    if (size > S.small_max) push_large(S, S.large[0], start, size, d, 0);
    else push_small(S, start, size, d, 0);
}

// --------------------------------------------------------- tile indexing ----
__global__ void k_tile_counts(const Seg* segs, uint32_t nseg, uint32_t* tiles, uint32_t* chunks) {
    uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nseg) return;
    uint32_t t = (segs[s].size + LT_TILE - 1) / LT_TILE;
    tiles[s] = t;
    chunks[s] = (t + CHUNK_TILES - 1) / CHUNK_TILES;
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
        if (sg.flags & F_KEYS) continue;
        const uint32_t* ord = S.ord[sg.flags & F_PARITY];
        const uint32_t d0 = sg.depth;
        uint32_t l = 0xFFFFFFFFu;
        const uint32_t m = sg.size < 256u ? sg.size : 256u;
        if (threadIdx.x < m) {
            uint64_t off0, off;
            uint32_t len0, len;
            str_of(S.a, ord[sg.start], off0, len0);
            const uint32_t i = sg.start + (uint32_t)((uint64_t)threadIdx.x * sg.size / m);
            str_of(S.a, ord[i], off, len);
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

__global__ void __launch_bounds__(LT_NT, 4) k_prefix(SortState S, Seg* segs, uint32_t nseg) {
    if (!segs) {  // graph mode: this pass's list and count live on the device
        segs = S.large[S.counters[12]];
        nseg = S.counters[13];
    }
    const uint32_t t = blockIdx.x;
    if (t >= S.counters[8]) return;
    const uint32_t si = find_seg(S.tile0, nseg, t);
    Seg& sg = segs[si];
    if (sg.flags & (F_KEYS | F_PIVOT)) return;
    const uint32_t par = sg.flags & F_PARITY;
    const uint32_t* ord = S.ord[par];
    const uint32_t tb = sg.start + (t - S.tile0[si]) * LT_TILE;
    const uint32_t te = min(sg.start + sg.size, tb + LT_TILE);
    const uint32_t d0 = sg.depth, cap = d0 + PREFIX_CAP;
    const uint32_t s0 = ord[sg.start];
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
            const uint32_t s = ord[i];
            str_of(S.a, s, off, len);
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
        const uint32_t s = ord[i];
        str_of(S.a, s, off, len);
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
    if (!segs) {  // graph mode: this pass's list and count live on the device
        segs = S.large[S.counters[12]];
        nseg = S.counters[13];
    }
    const uint32_t t = blockIdx.x;
    if (t >= S.counters[8]) return;
    const uint32_t si = find_seg(S.tile0, nseg, t);
    Seg& sg = segs[si];
    if (sg.flags & F_PIVOT) return;  // keys and diff come from k_pivot
    if (!(sg.flags & F_KEYS) && sg.spec && sg.newdepth == sg.spec - 1) {
        // the speculated depth was the common prefix: k_prefix wrote the keys
        if (t == S.tile0[si] && threadIdx.x == 0) sg.diff = sg.spec_diff;
        return;
    }
    const uint32_t par = sg.flags & F_PARITY;
    const bool valid = sg.flags & F_KEYS;
    const uint32_t depth = valid ? sg.depth : sg.newdepth;
    const uint32_t* ord = S.ord[par];
    unsigned long long* key = S.key[par];
    const uint32_t tb = sg.start + (t - S.tile0[si]) * LT_TILE;
    const uint32_t te = min(sg.start + sg.size, tb + LT_TILE);
    uint64_t k0;
    if (valid) {
        k0 = key[sg.start];
    } else {
        uint32_t s0 = ord[sg.start];
        k0 = key8_of(S.a, s0, depth);
    }
    uint64_t df = 0;
    if (valid) {
        // the tile's keys all in flight before any is used
        uint64_t k[LT_IPT];
#pragma unroll
        for (int j = 0; j < LT_IPT; ++j) {
            const uint32_t i = tb + j * LT_NT + threadIdx.x;
            k[j] = i < te ? key[i] : k0;
        }
#pragma unroll
        for (int j = 0; j < LT_IPT; ++j) df |= k[j] ^ k0;
    } else {
        // KD_ILP independent gathers in flight per thread
        for (uint32_t i0 = tb + threadIdx.x; i0 < te; i0 += KD_ILP * LT_NT) {
            uint32_t s[KD_ILP];
            uint64_t off[KD_ILP];
            uint32_t len[KD_ILP];
#pragma unroll
            for (int q = 0; q < KD_ILP; ++q) {
                const uint32_t i = i0 + q * LT_NT;
                s[q] = i < te ? ord[i] : 0u;
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
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) df |= __shfl_xor_sync(0xffffffffu, df, o);
    if ((threadIdx.x & 31) == 0 && df) atomicOr(&sg.diff, (unsigned long long)df);
}

// ------------------------------------------------------ sampled splitters ----
// Per large segment with keys (not a pivot pass) of at least split_min
// strings: the sample's byte-digit histogram at the first difference decides
// whether splitters pay (its largest bucket holds more than 1/64 of the
// sample, four times what a splitter bucket holds); if so, the sorted
// sample's every 8th key, distinct, become the splitters.  One block of
// SPL_SAMPLE / 2 threads per segment.
__global__ void __launch_bounds__(SPL_SAMPLE / 2) k_split_sample(SortState S, Seg* segs, uint32_t nseg) {
    if (!segs) {  // graph mode: this pass's list and count live on the device
        segs = S.large[S.counters[12]];
        nseg = S.counters[13];
    }
    __shared__ unsigned long long sk[SPL_SAMPLE];
    __shared__ uint32_t bcnt[256];
    __shared__ uint32_t s_fix0, s_nres;
    for (uint32_t si = blockIdx.x; si < nseg; si += gridDim.x) {
        Seg& sg = segs[si];
        const bool use = S.split_min && sg.size >= S.split_min && sg.diff != 0 && !(sg.flags & (F_PIVOT | F_PSEUDO));
        if (!use) {  // the same for the whole block
            if (threadIdx.x == 0) sg.nspl = 0;
            continue;
        }
        const unsigned long long* key = S.key[sg.flags & F_PARITY];
        const uint32_t shift = 56 - 8 * (uint32_t)(__clzll(sg.diff) >> 3);
        if (threadIdx.x < 256) bcnt[threadIdx.x] = 0;
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < (uint32_t)SPL_SAMPLE; j += blockDim.x) {
            const unsigned long long k = key[sg.start + (uint32_t)((uint64_t)j * sg.size / SPL_SAMPLE)];
            sk[j] = k;
            atomicAdd(&bcnt[(uint32_t)(k >> shift) & 0xFFu], 1u);
        }
        __syncthreads();
        // bitonic sort of the sample, ascending: thread t compares index i
        // (bit j clear) with i | j
        for (uint32_t k = 2; k <= (uint32_t)SPL_SAMPLE; k <<= 1) {
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                const uint32_t i = ((threadIdx.x & ~(j - 1)) << 1) | (threadIdx.x & (j - 1));
                const unsigned long long a = sk[i], b = sk[i | j];
                if ((a > b) == ((i & k) == 0)) {
                    sk[i] = b;
                    sk[i | j] = a;
                }
                __syncthreads();
            }
        }
        if (threadIdx.x == 0) {
            uint32_t mx = 0;
            for (int d = 0; d < 256; ++d) mx = max(mx, bcnt[d]);
            uint32_t m = 0, slot = 0, fix0 = 0, nres = 0;
            if (64 * mx > (uint32_t)SPL_SAMPLE) {
                slot = atomicAdd(&S.counters[6], 1u);
                if (slot < S.cap_spl) {
                    unsigned long long* spl = S.spl + (uint64_t)slot * SPL_STRIDE;
                    for (uint32_t q = 0; q < SPL_MAX; ++q) {
                        const unsigned long long c = sk[(q + 1) * (SPL_SAMPLE / SPL_STRIDE) - 1];
                        if (m == 0 || c != spl[m - 1]) spl[m++] = c;
                    }
                    for (uint32_t q = m; q < SPL_STRIDE; ++q) spl[q] = ~0ull;
                    // bucket-start slots in the fix list, one per bucket
                    nres = m > SPL_EQ_MAX ? m + 1 : 2 * m + 1;
                    fix0 = atomicAdd(&S.counters[5], nres);
                    if ((uint64_t)fix0 + nres > S.cap_fix) m = 0;
                }
            }
            s_fix0 = fix0;
            s_nres = nres;
            sg.nspl = m;
            sg.spl_slot = slot;
            sg.fix0 = fix0;
        }
        __syncthreads();
        // every reserved fix slot starts empty (also a reservation past the
        // list's end, as far as the list goes)
        if (s_nres) {
            const uint64_t e = min((uint64_t)s_fix0 + s_nres, S.cap_fix);
            for (uint64_t f = (uint64_t)s_fix0 + threadIdx.x; f < e; f += blockDim.x) S.fix[2 * f] = FIX_NONE;
        }
        __syncthreads();  // the sample buffer is reused by the next segment
    }
}

// Bucket of key k among m sorted splitters (the table padded to SPL_STRIDE
// with ~0): j = the number of splitters below k (at most m, eight fixed
// steps); with more than SPL_EQ_MAX splitters j, else 2j, or 2j + 1 when k
// equals splitter j.
__device__ __forceinline__ uint32_t spl_bucket(const unsigned long long* spl, uint32_t m, unsigned long long k) {
    uint32_t j = 0;
#pragma unroll
    for (uint32_t step = SPL_STRIDE / 2; step; step >>= 1)
        if (spl[j + step - 1] < k) j += step;
    if (m > SPL_EQ_MAX) return j;
    return 2 * j + (j < m && spl[j] == k ? 1u : 0u);
}

// LCPs at the bucket starts of splitter passes, once the order is final: the
// two neighbours have different keys at depth d.
__global__ void __launch_bounds__(256) k_lcp_fix(SortState S) {
    const uint64_t m = min((uint64_t)S.counters[5], S.cap_fix);
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t f = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; f < m; f += stride) {
        const uint32_t pos = S.fix[2 * f];
        if (pos == FIX_NONE) continue;
        uint32_t l = S.fix[2 * f + 1];
        const uint32_t x = S.ord_out[pos - 1], y = S.ord_out[pos];
        for (;;) {
            const uint64_t kx = key8_of(S.a, x, l), ky = key8_of(S.a, y, l);
            if (kx != ky) {
                l += key_lcp(kx, ky);
                break;
            }
            const uint32_t z = zero_byte(kx);
            if (z < 8) {
                l += z;
                break;
            }
            l += 8;
        }
        S.lcp_out[pos] = l;
    }
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

// Pseudo key of string (off, len) against the pivot (off0, len0), both
// sharing their first d0 bytes.
__device__ __forceinline__ uint64_t pivot_key(const uint8_t* chars, uint64_t off, uint32_t len, uint64_t off0,
                                              uint32_t len0, uint32_t d0) {
    uint32_t code = PIVOT_CAP, byte = 0;
    bool done = false;
    for (uint32_t c = 0; c < PIVOT_CAP && !done; c += 16) {
        // 16 bytes per step: two independent 8-byte compares
        uint64_t x[2], y[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            x[q] = key8(chars, off, len, d0 + c + 8 * q);
            y[q] = key8(chars, off0, len0, d0 + c + 8 * q);
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (done) continue;
            if (x[q] != y[q]) {
                const uint32_t j = key_lcp(x[q], y[q]);
                const uint32_t l = c + 8 * q + j;
                if (l < PIVOT_CAP) {
                    const uint32_t bx = (uint32_t)(x[q] >> (56 - 8 * j)) & 0xFFu;
                    const uint32_t by = (uint32_t)(y[q] >> (56 - 8 * j)) & 0xFFu;
                    code = bx < by ? l : 2 * PIVOT_CAP - l;
                    byte = bx;
                }
                done = true;
            } else if (zero_byte(x[q]) < 8) {
                done = true;  // equal to the pivot
            }
        }
    }
    return (uint64_t)code << 56 | (uint64_t)byte << 48;
}

__global__ void __launch_bounds__(LT_NT) k_pivot(SortState S, Seg* segs, uint32_t nseg) {
    if (!segs) {  // graph mode: this pass's list and count live on the device
        segs = S.large[S.counters[12]];
        nseg = S.counters[13];
    }
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
    uint64_t off0;
    uint32_t len0;
    str_of(S.a, sg.piv == NO_PIVOT ? ord[sg.start] : sg.piv, off0, len0);
    const uint64_t k0 = (uint64_t)PIVOT_CAP << 56;
    uint64_t df = 0;
    for (uint32_t i = tb + threadIdx.x; i < te; i += LT_NT) {
        uint64_t off;
        uint32_t len;
        str_of(S.a, ord[i], off, len);
        const uint64_t k = pivot_key(S.a.chars, off, len, off0, len0, sg.depth);
        key[i] = k;
        df |= k ^ k0;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) df |= __shfl_xor_sync(0xffffffffu, df, o);
    if ((threadIdx.x & 31) == 0 && df) atomicOr(&sg.diff, (unsigned long long)df);
}

// ------------------------------------------------------------------ hist ----
__device__ __forceinline__ uint32_t digit_of(uint64_t k, uint32_t shift) { return (uint32_t)(k >> shift) & 0xFFu; }

// The digit of a pass over plain keys: the (up to) eight most significant
// bits in which the segment's keys differ, packed in key order.  Every bit
// above the lowest of them that is not one of them is the same in all keys,
// so the digit orders the keys as their first bytes do.  Where the key byte
// at the first difference varies in all eight bits this is that byte; over a
// small alphabet (letters vary in 5 or 6 bits of a byte, DNA in 4) a digit
// covers more than one key byte, and a pass splits up to 256 ways instead of
// as many ways as the byte has values.  sh[j]: the right shift that brings
// digit bit j (most significant first) to bit 0.
struct BitDigit {
    uint32_t nb;     // bits in the digit (1..8)
    uint32_t sh[8];
    bool whole;      // one whole key byte: (k >> sh[7]) & 0xFF
};

// Whether a pass over plain keys splits on bits: knob sort_bits 1 always, 2
// where the first differing key byte varies in at most four bits (DNA, or a
// leading digit with few values), 3 the same in the first pass only, 0
// never; and only for segments of more than four times the small-segment
// cutoff (a 256-way split of a segment just above the cutoff leaves children
// of a few strings each, whose segment records cost more than sorting them).
__device__ __forceinline__ bool use_bits(uint32_t mode, uint64_t diff, uint32_t shift, uint32_t size,
                                         uint32_t small_max, uint32_t first) {
    if ((uint64_t)size <= 4ull * small_max) return false;
    const bool narrow = __popc((uint32_t)(diff >> shift) & 0xFFu) <= 4;
    return mode == 1 || (mode == 2 && narrow) || (mode == 3 && first && narrow);
}

__device__ __forceinline__ BitDigit bit_digit_spec(uint64_t diff) {
    BitDigit d;
    d.nb = 0;
    uint64_t x = diff;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        d.sh[j] = 0;
        if (x) {
            const uint32_t at = 63u - (uint32_t)__clzll(x);
            d.sh[j] = at;
            x &= ~(1ull << at);
            ++d.nb;
        }
    }
    d.whole = d.nb == 8 && (d.sh[0] & 7u) == 7u && d.sh[7] + 7u == d.sh[0];
    return d;
}

// Digit lookup in shared memory: for each key byte that holds digit bits,
// tab[q][v] is the digit bits of byte value v, packed and moved to their place
// in the digit; a key's digit is the OR over those bytes (usually two).
struct BitTables {
    uint8_t tab[8][256];
    uint32_t n;      // key bytes holding digit bits
    uint32_t sh[8];  // right shift of each such byte
};

// Builds the tables of digit d; every thread of the block calls it, and a
// barrier follows before the first lookup.
__device__ __forceinline__ void bit_tables_build(BitTables& T, const BitDigit& d) {
    uint64_t chosen = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if ((uint32_t)j < d.nb) chosen |= 1ull << d.sh[j];
    for (uint32_t v = threadIdx.x; v < 256; v += blockDim.x) {
        uint32_t q = 0, below = (uint32_t)__popcll(chosen);
        for (int J = 0; J < 8; ++J) {
            const uint32_t sh = 56u - 8u * (uint32_t)J;
            const uint32_t sel = (uint32_t)(chosen >> sh) & 0xFFu;
            if (!sel) continue;
            below -= (uint32_t)__popc(sel);  // digit bits in later key bytes
            uint32_t x = 0;                  // the bits of v that sel selects, packed
            for (int bit = 7; bit >= 0; --bit)
                if ((sel >> bit) & 1u) x = (x << 1) | ((v >> bit) & 1u);
            T.tab[q][v] = (uint8_t)(x << below);
            if (v == 0) T.sh[q] = sh;
            ++q;
        }
        if (v == 0) T.n = q;
    }
}

__device__ __forceinline__ uint32_t bit_digit(uint64_t k, const BitDigit& d, const BitTables& T) {
    if (d.whole) return (uint32_t)(k >> d.sh[7]) & 0xFFu;
    uint32_t v = 0;
    for (uint32_t q = 0; q < T.n; ++q) v |= T.tab[q][(uint32_t)(k >> T.sh[q]) & 0xFFu];
    return v;
}

// Key byte (from the key's first byte) that holds digit bit h (0: least
// significant): two keys whose digits first differ in bit h share exactly
// that many bytes past the segment depth.
__device__ __forceinline__ uint32_t bit_digit_byte(const BitDigit& d, uint32_t h) {
    uint32_t byte = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if ((uint32_t)j + 1 + h == d.nb) byte = (63u - d.sh[j]) >> 3;
    return byte;
}

// BITS: the bit-digit form (its tables and registers only where the knob asks
// for it; the byte form keeps the occupancy of a 32-register kernel).
template <bool BITS>
__global__ void __launch_bounds__(LT_NT) k_hist(SortState S, const Seg* segs, uint32_t nseg) {
    if (!segs) {  // graph mode: this pass's list and count live on the device
        segs = S.large[S.counters[12]];
        nseg = S.counters[13];
    }
    // one 256-bin histogram per warp (shared-memory atomics contend only
    // inside a warp), summed per digit at the end
    __shared__ uint32_t hist[LT_NT / 32][256];
    __shared__ unsigned long long s_spl[SPL_STRIDE];
    const uint32_t t = blockIdx.x;
    if (t >= S.counters[8]) return;
    const uint32_t si = find_seg(S.tile0, nseg, t);
    const Seg sg = segs[si];
    if (sg.diff == 0) return;
    const uint32_t shift = 56 - 8 * (uint32_t)(__clzll(sg.diff) >> 3);
    const uint32_t m = sg.nspl;
    // plain keys split on their top differing bits, pivot pseudo keys on a byte
    const bool bits = BITS && !m && !(sg.flags & (F_PIVOT | F_PSEUDO)) && use_bits(S.bits, sg.diff, shift, sg.size, S.small_max, S.first);
    const BitDigit bd = bit_digit_spec(bits ? (uint64_t)sg.diff : (0xFFull << shift));
    __shared__ BitTables bt;
    if (BITS && !bd.whole) bit_tables_build(bt, bd);
    const unsigned long long* key = S.key[sg.flags & F_PARITY];
#pragma unroll
    for (int w = 0; w < LT_NT / 32; ++w) hist[w][threadIdx.x] = 0;
    if (m)
        for (uint32_t q = threadIdx.x; q < SPL_STRIDE; q += LT_NT) s_spl[q] = S.spl[(uint64_t)sg.spl_slot * SPL_STRIDE + q];
    __syncthreads();
    const uint32_t tb = sg.start + (t - S.tile0[si]) * LT_TILE;
    const uint32_t te = min(sg.start + sg.size, tb + LT_TILE);
    uint32_t* wh = hist[threadIdx.x >> 5];
    // the tile's keys loaded before any is counted (one DRAM wait, not LT_IPT)
    uint64_t k[LT_IPT];
#pragma unroll
    for (int j = 0; j < LT_IPT; ++j) {
        const uint32_t i = tb + j * LT_NT + threadIdx.x;
        k[j] = i < te ? key[i] : 0;
    }
#pragma unroll
    for (int j = 0; j < LT_IPT; ++j) {
        const uint32_t i = tb + j * LT_NT + threadIdx.x;
        if (i < te)
            atomicAdd(&wh[m ? spl_bucket(s_spl, m, k[j]) : BITS ? bit_digit(k[j], bd, bt) : digit_of(k[j], shift)], 1u);
    }
    __syncthreads();
    uint32_t c = 0;
#pragma unroll
    for (int w = 0; w < LT_NT / 32; ++w) c += hist[w][threadIdx.x];
    S.tile_hist[(uint64_t)t * 256 + threadIdx.x] = c;
}

// ------------------------------------------------------------ chunk sums ----
__global__ void k_chunk_sum(SortState S, const Seg* segs, uint32_t nseg) {
    if (!segs) {  // graph mode: this pass's list and count live on the device
        segs = S.large[S.counters[12]];
        nseg = S.counters[13];
    }
    const uint32_t c = blockIdx.x;
    if (c >= S.counters[9]) return;
    const uint32_t si = find_seg(S.chunk0, nseg, c);
    const Seg sg = segs[si];
    if (sg.diff == 0) return;
    const uint32_t ntiles = (sg.size + LT_TILE - 1) / LT_TILE;
    const uint32_t t0 = S.tile0[si] + (c - S.chunk0[si]) * CHUNK_TILES;
    const uint32_t t1 = min(S.tile0[si] + ntiles, t0 + CHUNK_TILES);
    // each tile's count becomes its exclusive prefix inside the chunk (one
    // read for the scatter instead of the chunk's earlier tiles); every load
    // of the chunk in flight before the first store
    uint32_t v[CHUNK_TILES];
#pragma unroll
    for (int q = 0; q < CHUNK_TILES; ++q)
        v[q] = t0 + q < t1 ? S.tile_hist[(uint64_t)(t0 + q) * 256 + threadIdx.x] : 0u;
    uint32_t s = 0;
#pragma unroll
    for (int q = 0; q < CHUNK_TILES; ++q) {
        if (t0 + q < t1) S.tile_hist[(uint64_t)(t0 + q) * 256 + threadIdx.x] = s;
        s += v[q];
    }
    S.chunk_pre[(uint64_t)c * 256 + threadIdx.x] = s;
}

// ----------------------------------------------------------- segment scan ----
__global__ void __launch_bounds__(256) k_seg_scan(SortState S, Seg* segs, uint32_t nseg, Seg* next) {
    __shared__ uint32_t sh[32];
    __shared__ uint32_t s_first;
    if (!segs) {  // graph mode: this pass's list and count live on the device
        const uint32_t c = S.counters[12];
        segs = S.large[c];
        next = S.large[c ^ 1u];
        nseg = S.counters[13];
    }
    const uint32_t si = blockIdx.x;
    if (si >= nseg) return;
    Seg& sg = segs[si];
    const uint32_t par = sg.flags & F_PARITY;
    const bool pseudo = (sg.flags & (F_PIVOT | F_PSEUDO)) != 0;
    const uint32_t depth = (sg.flags & (F_KEYS | F_PIVOT)) ? sg.depth : sg.newdepth;
    const uint32_t d = threadIdx.x;
    if (sg.diff == 0) {
        // Every key equal: byte-identical strings if the key holds their end,
        // else continue deeper without keys.
        const uint64_t k0 = S.key[par][sg.start];
        const uint32_t* ord = S.ord[par];
        uint32_t fin = 0xFFFFFFFFu, cont = 0, cflags = par;
        if (pseudo) {
            const uint32_t code = (uint32_t)(k0 >> 56), byte = (uint32_t)(k0 >> 48) & 0xFFu;
            if (code == PIVOT_CAP) {
                uint64_t o0;
                uint32_t l0;
                str_of(S.a, ord[sg.start], o0, l0);
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
        if (fin != 0xFFFFFFFFu) {
            for (uint32_t i = threadIdx.x; i < sg.size; i += blockDim.x) {
                S.ord_out[sg.start + i] = ord[sg.start + i];
                if (i) S.lcp_out[sg.start + i] = fin;
            }
        } else if (threadIdx.x == 0) {
            push_large(S, next, sg.start, sg.size, cont, cflags);
        }
        return;
    }
    const uint32_t b = (uint32_t)(__clzll(sg.diff) >> 3);
    const uint32_t c0 = S.chunk0[si];
    const uint32_t ntiles = (sg.size + LT_TILE - 1) / LT_TILE;
    const uint32_t nch = (ntiles + CHUNK_TILES - 1) / CHUNK_TILES;
    // the digit's column of chunk sums, eight loads in flight (a segment of
    // n strings has n / 64 Ki chunks, walked by one block)
    uint32_t run = 0;
    for (uint32_t c = 0; c < nch; c += 8) {
        uint32_t v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = c + q < nch ? S.chunk_pre[(uint64_t)(c0 + c + q) * 256 + d] : 0u;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (c + q < nch) S.chunk_pre[(uint64_t)(c0 + c + q) * 256 + d] = run;
            run += v[q];
        }
    }
    const uint32_t total = run;
    // block exclusive scan over the 256 digits
    const int lane = d & 31, w = d >> 5;
    uint32_t x = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[w] = x;
    if (d == 0) s_first = 256;
    __syncthreads();
    uint32_t wb = 0;
    for (int k = 0; k < w; ++k) wb += sh[k];
    const uint32_t excl = wb + x - total;
    if (total) atomicMin(&s_first, d);
    uint32_t* bk = S.bucket + (uint64_t)si * 257;
    bk[d] = sg.start + excl;
    if (d == 255) bk[256] = sg.start + sg.size;
    __syncthreads();
    if (d == 0) {
        sg.first_digit = s_first;
        sg.depth = depth;
    }
    uint32_t* child = S.child ? S.child + (uint64_t)si * 256 + d : nullptr;
    if (child) *child = 0xFFFFFFFFu;  // set below for a large child that keeps the keys
    if (total < 2) return;
    const uint32_t cs = sg.start + excl;
    const uint32_t np = par ^ 1u;
    if (sg.nspl) {
        // splitter buckets: children keep the keys at this depth (an
        // equality bucket's keys are all equal: its next pass goes deeper)
        if (total > S.small_max) {
            const uint32_t slot = push_large(S, next, cs, total, depth, np | F_KEYS);
            if (child) *child = slot;
        } else {
            push_small(S, cs, total, depth, np | F_KEYS);
        }
    } else if (!pseudo) {
        // digit 0 holds the strings that end at byte b, unless byte b has a
        // constant nonzero part (then no string ends there and digit 0 is an
        // ordinary bucket)
        bool ended_ok = true;
        if (S.bits) {
            const uint32_t shift = 56 - 8 * b;
            const uint64_t k0 = S.key[par][sg.start];
            ended_ok = (((k0 >> shift) & 0xFFu) & ~((sg.diff >> shift) & 0xFFu)) == 0;
        }
        if (d == 0 && ended_ok) return;  // strings that end here: written by the scatter
        // children keep the parent's keys: their first b+1 key bytes are now
        // common; one that keeps most of the parent gets a pivot pass
        if (total > S.small_max) {
            if (S.pivot && 2 * (uint64_t)total > sg.size) {
                push_large(S, next, cs, total, depth + b + 1, np | F_PIVOT);
            } else {
                const uint32_t slot = push_large(S, next, cs, total, depth, np | F_KEYS);
                if (child) *child = slot;
            }
        } else {
            push_small(S, cs, total, depth, np | F_KEYS);
        }
    } else if (b == 0) {
        // split by pivot code (only the pivot pass's own segment): large children keep the pseudo keys, small
        // ones restart from the depth their strings share
        if (total > S.small_max) {
            const uint32_t slot = push_large(S, next, cs, total, depth, np | F_KEYS | F_PSEUDO);
            if (child) *child = slot;
        } else {
            uint32_t cd = depth + pivot_l(d);
            if (d == PIVOT_CAP) {
                uint64_t o0;
                uint32_t l0;
                str_of(S.a, sg.piv == NO_PIVOT ? S.ord[par][sg.start] : sg.piv, o0, l0);
                cd = min(depth + PIVOT_CAP, l0);
            }
            push_small(S, cs, total, cd, np);
        }
    } else {
        // split by the byte after the shared d + l bytes; byte 0: strings that
        // end there, written by the scatter
        if (d == 0) return;
        const uint32_t cd = depth + pivot_l((uint32_t)(S.key[par][sg.start] >> 56)) + 1;
        if (total > S.small_max) push_large(S, next, cs, total, cd, np | (S.pivot && 2 * (uint64_t)total > sg.size ? F_PIVOT : 0u));
        else push_small(S, cs, total, cd, np);
    }
}

// --------------------------------------------------------------- scatter ----
// Ranks are stable within the tile (warp-aggregated per digit); the tile is
// first reordered by digit in shared memory so that the global writes of each
// digit's run are contiguous.
constexpr size_t SCATTER_SMEM = (size_t)LT_TILE * (8 + 4 + 1);

__global__ void __launch_bounds__(LT_NT, 4) k_scatter(SortState S, const Seg* segs, uint32_t nseg) {
    if (!segs) {  // graph mode: this pass's list and count live on the device
        segs = S.large[S.counters[12]];
        nseg = S.counters[13];
    }
    extern __shared__ __align__(16) unsigned char sm_scatter[];
    unsigned long long* skey = (unsigned long long*)sm_scatter;
    uint32_t* sord = (uint32_t*)(skey + LT_TILE);
    uint8_t* sdig = (uint8_t*)(sord + LT_TILE);
    __shared__ uint32_t base[256];
    __shared__ uint32_t bstart[257];
    __shared__ uint32_t tloff[256];
    __shared__ uint32_t wcnt[LT_NT / 32][256];
    __shared__ uint32_t wsum[LT_NT / 32];
    __shared__ uint32_t schild[256];
    __shared__ uint32_t actm[LT_NT / 32];  // per warp: the digits (d & 7 == warp) whose keys it folds
    __shared__ unsigned long long s_spl[SPL_STRIDE];
    const uint32_t t = blockIdx.x;
    if (t >= S.counters[8]) return;
    const uint32_t si = find_seg(S.tile0, nseg, t);
    const Seg sg = segs[si];
    if (sg.diff == 0) return;
    const uint32_t par = sg.flags & F_PARITY;
    const uint32_t b = (uint32_t)(__clzll(sg.diff) >> 3);
    const uint32_t shift = 56 - 8 * b;
    const uint32_t depth = sg.depth;
    const uint32_t m = sg.nspl;  // splitter buckets (0: the byte digit)
    const bool pseudo = (sg.flags & (F_PIVOT | F_PSEUDO)) != 0;
    // plain keys split on their top differing bits, pivot pseudo keys on a byte
    const bool bits = S.bits && !m && !pseudo && use_bits(S.bits, sg.diff, shift, sg.size, S.small_max, S.first);
    const BitDigit bd = bit_digit_spec(bits ? (uint64_t)sg.diff : (0xFFull << shift));
    __shared__ BitTables bt;
    if (!bd.whole) bit_tables_build(bt, bd);  // the barrier after the block's set-up follows
    // digit 0 holds the strings that end at byte b unless byte b has a
    // constant nonzero part
    bool ended_ok = true;
    if (bits) {
        const uint64_t k0 = S.key[par][sg.start];
        ended_ok = (((k0 >> shift) & 0xFFu) & ~((sg.diff >> shift) & 0xFFu)) == 0;
    }
    // LCP inside the group of strings that end here and at bucket starts
    // (pivot code splits: d + min(l, l') from the two codes)
    const bool code_split = pseudo && b == 0;
    const uint32_t lcp_here = pseudo ? depth + pivot_l((uint32_t)(S.key[par][sg.start] >> 56)) : depth + b;
    const uint32_t tloc = t - S.tile0[si];
    const uint32_t c = S.chunk0[si] + tloc / CHUNK_TILES;
    {
        const uint32_t d = threadIdx.x;
        const uint32_t* bk = S.bucket + (uint64_t)si * 257;
        // k_chunk_sum left the tile's prefix inside its chunk in tile_hist
        base[d] = bk[d] + S.chunk_pre[(uint64_t)c * 256 + d] + S.tile_hist[(uint64_t)t * 256 + d];
        bstart[d] = bk[d];
        if (d == 0) bstart[256] = bk[256];
        if (S.child) schild[d] = S.child[(uint64_t)si * 256 + d];
        if (d < LT_NT / 32) actm[d] = 0;
#pragma unroll
        for (int w = 0; w < LT_NT / 32; ++w) wcnt[w][d] = 0;
        if (m)
            for (uint32_t q = d; q < SPL_STRIDE; q += LT_NT) s_spl[q] = S.spl[(uint64_t)sg.spl_slot * SPL_STRIDE + q];
    }
    __syncthreads();
    const uint32_t* ord = S.ord[par];
    const unsigned long long* key = S.key[par];
    uint32_t* ord_dst = S.ord[par ^ 1u];
    unsigned long long* key_dst = S.key[par ^ 1u];
    const uint32_t tb = sg.start + tloc * LT_TILE;
    const uint32_t te = min(sg.start + sg.size, tb + LT_TILE);
    const uint32_t tn = te - tb;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t wb = tb + (uint32_t)w * 32 * LT_IPT;
    uint64_t k[LT_IPT];
    uint32_t o[LT_IPT];
    uint32_t rk[LT_IPT];
#pragma unroll
    for (int j = 0; j < LT_IPT; ++j) {
        const uint32_t i = wb + j * 32 + lane;
        k[j] = i < te ? key[i] : 0;
        o[j] = i < te ? ord[i] : 0;
    }
#pragma unroll
    for (int j = 0; j < LT_IPT; ++j) {
        const uint32_t i = wb + j * 32 + lane;
        const uint32_t dg = i < te ? (m ? spl_bucket(s_spl, m, k[j]) : bit_digit(k[j], bd, bt)) : 0x100u + lane;
        const uint32_t peers = __match_any_sync(0xffffffffu, dg);
        const uint32_t r = __popc(peers & ((1u << lane) - 1));
        const uint32_t prev = dg < 256 ? wcnt[w][dg] : 0;
        __syncwarp();
        if (dg < 256 && lane == __ffs(peers) - 1) wcnt[w][dg] = prev + __popc(peers);
        __syncwarp();
        rk[j] = (dg & 0xFFu) << 24 | (prev + r);  // the digit kept for the placement below
    }
    __syncthreads();
    {
        // exclusive over warps per digit, then over digits within the tile
        const uint32_t d = threadIdx.x;
        uint32_t run = 0;
#pragma unroll
        for (int ww = 0; ww < LT_NT / 32; ++ww) {
            const uint32_t v = wcnt[ww][d];
            wcnt[ww][d] = run;
            run += v;
        }
        uint32_t x = run;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
            if (lane >= off) x += y;
        }
        if (lane == 31) wsum[w] = x;
        __syncthreads();
        uint32_t wpre = 0;
        for (int ww = 0; ww < w; ++ww) wpre += wsum[ww];
        tloff[d] = wpre + x - run;
        if (S.child && run && schild[d] < S.cap_large) atomicOr(&actm[d & 7], 1u << (d >> 3));
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < LT_IPT; ++j) {
        const uint32_t i = wb + j * 32 + lane;
        if (i >= te) continue;
        const uint32_t dg = rk[j] >> 24;
        const uint32_t lp = tloff[dg] + wcnt[w][dg] + (rk[j] & 0xFFFFFFu);
        if (lp >= tn) {  // never taken when the counts agree
            atomicExch(&S.counters[10], 1u);
            continue;
        }
        skey[lp] = k[j];
        sord[lp] = o[j];
        sdig[lp] = (uint8_t)dg;
    }
    __syncthreads();
    if (S.child) {
        // the OR and AND of the keys each large child that keeps them gets
        // from this tile (one warp per digit, over the digit's run in shared
        // memory): its next pass needs no key read to find the byte where its
        // keys differ
        for (uint32_t m = actm[w]; m; m &= m - 1) {
            const uint32_t dg = ((uint32_t)(__ffs(m) - 1) << 3) | (uint32_t)w;
            const uint32_t r0 = tloff[dg], r1 = dg < 255 ? tloff[dg + 1] : tn;
            unsigned long long vo = 0, va = ~0ull;
            for (uint32_t x = r0 + lane; x < r1; x += 32) {
                const unsigned long long v = skey[x];
                vo |= v;
                va &= v;
            }
            const uint32_t olo = __reduce_or_sync(0xffffffffu, (uint32_t)vo);
            const uint32_t ohi = __reduce_or_sync(0xffffffffu, (uint32_t)(vo >> 32));
            const uint32_t alo = __reduce_and_sync(0xffffffffu, (uint32_t)va);
            const uint32_t ahi = __reduce_and_sync(0xffffffffu, (uint32_t)(va >> 32));
            if (lane == 0) {
                const uint32_t slot = schild[dg];
                atomicOr(&S.nxt[slot].kor, ((unsigned long long)ohi << 32) | olo);
                atomicAnd(&S.nxt[slot].kand, ((unsigned long long)ahi << 32) | alo);
            }
        }
    }
    for (uint32_t x = threadIdx.x; x < tn; x += LT_NT) {
        const uint32_t dg = sdig[x];
        const uint32_t dest = base[dg] + (x - tloff[dg]);
        const uint32_t bs = bstart[dg], cnt = bstart[dg + 1] - bs;
        if (dest < bs || dest >= bs + cnt) {  // never taken when the counts agree
            atomicExch(&S.counters[10], 1u);
            continue;
        }
        const uint32_t oo = sord[x];
        const bool ended = !m && dg == 0 && !code_split && ended_ok;
        if (ended || cnt == 1) {
            S.ord_out[dest] = oo;
            if (ended && dest != bs) S.lcp_out[dest] = lcp_here;
        } else {
            ord_dst[dest] = oo;
            key_dst[dest] = skey[x];
        }
        if (m) {
            // a splitter bucket's start: its LCP once the order is final
            if (dest == bs && dg != sg.first_digit) {
                S.fix[2 * ((uint64_t)sg.fix0 + dg)] = dest;
                S.fix[2 * ((uint64_t)sg.fix0 + dg) + 1] = depth;
            }
        } else if (dest == bs && dg != sg.first_digit) {
            uint32_t l = lcp_here;
            if (code_split || !bd.whole) {
                uint32_t pd = dg - 1;  // previous non-empty bucket (exists: dg is not the first)
                while (pd > 0 && bstart[pd] == bs) --pd;
                // pivot codes: d + min(l, l'); bit digits: the byte of the
                // highest bit in which the two buckets' digits differ
                l = code_split ? depth + min(pivot_l(dg), pivot_l(pd))
                               : depth + bit_digit_byte(bd, 31u - (uint32_t)__clz(dg ^ pd));
            }
            S.lcp_out[dest] = l;
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
// thread each, up to 32 by a warp, larger ones return to the CTA's stack.
// Over keys with enough differing bits nearly all buckets hold one string, so
// a string costs about 60 thread instructions; the stable byte passes with
// match instructions and bitonic networks that this replaces took 26 warp
// instructions per string.  B200, 32e6 strings in segments of about 700:
// 1.12 -> 0.49 ms; a 4e6-string request whose segments are chains of nested
// prefixes: 0.61 -> 0.18 ms; 9e6 suffixes of copied text: 9.2 -> 6.5 ms.
constexpr unsigned FULL = 0xffffffffu;
enum GroupKind : uint32_t { G_PLAIN = 0, G_TIE = 1, G_ID = 2, G_PSEUDO = 3 };  // G_TIE: keys still to be made
// Pivot code of a string with LCP l: l below the pivot, CODE_MID for strings
// equal to it (or to CODE_CAP bytes of it), 0xBFFF - l above it.
constexpr uint32_t CODE_MID = 0x4000u, CODE_TOP = 0xBFFFu, CODE_CAP = 0x3FFEu;
constexpr uint32_t TINY_MAX = 8;  // largest bucket one thread sorts

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
// first d bytes; at most d + CODE_CAP.  32 bytes per lane first; lanes still
// equal then go one after another, the whole warp reading 256 bytes of a pair
// at a time.  Every lane of the warp calls it.
__device__ __forceinline__ uint32_t warp_lcp(const ArenaDev& a, StrRef x, StrRef h, uint32_t d, bool active) {
    uint32_t l = d;
    bool open = active;
    if (active) {
        uint64_t u[4], v[4];
        key_words<4>(a.chars, x.off, x.len, d, 4, u);
        key_words<4>(a.chars, h.off, h.len, d, 4, v);
        l = d + 32;
#pragma unroll
        for (int w = 3; w >= 0; --w) {  // the first word that differs or ends wins
            if (u[w] != v[w]) {
                l = d + 8 * w + key_lcp(u[w], v[w]);
                open = false;
            } else if (zero_byte(u[w]) < 8) {
                l = d + 8 * w + zero_byte(u[w]);
                open = false;
            }
        }
    }
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t todo = __ballot_sync(FULL, open); todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1;
        const uint64_t ox = __shfl_sync(FULL, x.off, src), oh = __shfl_sync(FULL, h.off, src);
        const uint32_t lx = __shfl_sync(FULL, x.len, src), lh = __shfl_sync(FULL, h.len, src);
        const uint32_t d0 = __shfl_sync(FULL, d, src);
        uint32_t at = d0 + 32;
        for (;; at += 256) {
            if (at >= d0 + CODE_CAP) {
                at = d0 + CODE_CAP;
                break;
            }
            const uint32_t p = at + 8 * lane;
            const uint64_t u = key8(a.chars, ox, lx, p), v = key8(a.chars, oh, lh, p);
            const uint32_t e = u != v ? key_lcp(u, v) : zero_byte(u);
            const uint32_t hit = __ballot_sync(FULL, e < 8);
            if (hit) {
                const int f = __ffs(hit) - 1;
                at = min(at + 8 * f + __shfl_sync(FULL, e, f), d0 + CODE_CAP);
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

// Compare-exchange network over the first P (a power of two) lanes.
template <bool GRP>
__device__ __forceinline__ void warp_network(uint32_t P, uint32_t& grp, uint64_t& key, uint32_t& id, uint32_t& dep) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (uint32_t k = 2; k <= 32; k <<= 1) {
        if (k > P) break;
#pragma unroll
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            const uint64_t pk = __shfl_xor_sync(FULL, key, j);
            const uint32_t po = __shfl_xor_sync(FULL, id, j);
            const bool want_min = ((lane & k) == 0) == ((lane & j) == 0);
            if (GRP) {
                const uint32_t pg = __shfl_xor_sync(FULL, grp, j), pd = __shfl_xor_sync(FULL, dep, j);
                const bool less = pg < grp || (pg == grp && (pk < key || (pk == key && po < id)));
                if (less == want_min) {
                    grp = pg;
                    key = pk;
                    id = po;
                    dep = pd;
                }
            } else {
                const bool less = pk < key || (pk == key && po < id);
                if (less == want_min) {
                    key = pk;
                    id = po;
                }
            }
        }
    }
}

// A group of size <= 32: lane i < size holds an id and, unless kind is G_TIE
// or G_ID, its key.  On return lane i holds the i-th smallest string; lcp[i]
// (1 <= i < size) gets the LCP with the predecessor (depth itself for G_ID).
__device__ __forceinline__ void warp_group(const ArenaDev& a, uint32_t size, uint32_t depth, uint32_t kind,
                                           uint64_t key, uint32_t& id, uint32_t* lcp) {
    const uint32_t lane = threadIdx.x & 31;
    const bool valid = lane < size;
    const uint32_t P = size <= 2 ? 2u : 1u << (32 - __clz(size - 1));
    uint32_t grp = valid ? 0u : 0xFFFFFFFFu;
    uint32_t dep = depth;
    bool pseudo = kind == G_PSEUDO;
    if (!valid) {
        key = ~0ull;
        id = 0xFFFFFFFFu;
    } else if (kind == G_ID) {
        key = 0;
    }
    bool unres = valid && kind == G_TIE;
    uint32_t rs = 0;
    bool first = true;
    for (;;) {
        if (kind != G_TIE || !first) {
            if (first) warp_network<false>(P, grp, key, id, dep);
            else warp_network<true>(P, grp, key, id, dep);
            const uint32_t qg = __shfl_up_sync(FULL, grp, 1);
            const uint64_t qk = __shfl_up_sync(FULL, key, 1);
            const bool head = lane == 0 || qg != grp || qk != key;
            if (kind == G_ID) {
                if (valid && lane > 0) lcp[lane] = depth;
                return;
            }
            // dep of a resolved string is no longer used; neighbours in one
            // group share it
            if (valid && lane > 0 && qg == grp) {
                if (qk != key) lcp[lane] = group_lcp(qk, key, dep, pseudo);
                else if (key_ended(key, pseudo)) lcp[lane] = ref_of(a, id).len;  // equal strings
            }
            const uint32_t heads = __ballot_sync(FULL, head);
            rs = 31u - __clz(heads & ((2u << lane) - 1u));
            const bool next_head = lane == 31 ? true : ((heads >> (lane + 1)) & 1u) != 0;
            const bool multi = !head || (!next_head && lane + 1 < size);
            unres = valid && multi && !key_ended(key, pseudo);
            if (valid) grp = rs;
        }
        if (!__any_sync(FULL, unres)) return;
        // every unresolved run goes on against its head
        const uint32_t nd = first && kind == G_TIE ? depth : tie_depth(key, dep, pseudo);
        const uint32_t hid = __shfl_sync(FULL, id, rs);
        StrRef x{0, 0}, h{0, 0};
        if (unres) {
            x = ref_of(a, id);
            h = ref_of(a, hid);
        }
        const bool cmp = unres && lane != rs;
        const uint32_t l = warp_lcp(a, x, h, nd, cmp);
        // resolved strings keep a key that orders them among themselves
        if (unres) {
            dep = nd;
            key = cmp ? pseudo_key(a, x, h, l, nd) : (uint64_t)CODE_MID << 48;
        } else if (valid) {
            key = 0;  // alone in its group, or equal strings in id order
        }
        // the head shares its end with the strings that equal it, or the cap
        const uint32_t capped = __ballot_sync(FULL, cmp && l >= nd + CODE_CAP);
        const uint32_t run = __match_any_sync(FULL, unres ? rs : 32u + lane);
        if (unres && lane == rs && (capped & run)) key |= 0x010101010101ull;
        pseudo = true;
        first = false;
    }
}

// Segments of 2..32 strings: one warp each, four per CTA.
// dcount (graph mode): the segment count on the device; blocks stride over it.
__global__ void __launch_bounds__(128) k_warp_segs(SortState S, const Seg* segs, uint32_t nseg, const uint32_t* dcount) {
    if (dcount) nseg = *dcount;
    for (uint32_t si = blockIdx.x * 4 + (threadIdx.x >> 5); si < nseg; si += gridDim.x * 4) {
        const uint32_t lane = threadIdx.x & 31;
        const Seg seg = segs[si];
        const uint32_t* src = S.ord[seg.flags & F_PARITY];
        uint32_t id = 0;
        uint64_t key = 0;
        if (lane < seg.size) {
            id = src[seg.start + lane];
            key = (seg.flags & F_KEYS) ? S.key[seg.flags & F_PARITY][seg.start + lane] : key8_of(S.a, id, seg.depth);
        }
        warp_group(S.a, seg.size, seg.depth, G_PLAIN, key, id, S.lcp_out + seg.start);
        if (lane < seg.size) S.ord_out[seg.start + lane] = id;
    }
}

// The bits that pick a bucket: up to `want` of the most significant bits of
// diff, in at most 8 runs of neighbouring bits.  A key's bucket is the OR over
// the runs of ((key >> lo) >> sh) & mask; every bit above lo that is not
// chosen is the same in all keys, so buckets order as keys do.
// In a pseudo group whose code bits are all chosen, a bucket holds one code;
// otherwise (LCPs over thousands of bytes) `mixed` is set.
struct BucketBits {
    uint32_t lo, nruns, wide, all;  // wide: the bits span more than 32; all: every differing bit is chosen
    uint32_t mixed;
    uint32_t sh[8], mask[8];
};

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

// A group on the CTA's stack or the warps' list: positions [start, start +
// size) of the segment, packed with the kind.
__device__ __forceinline__ uint2 group_pack(uint32_t start, uint32_t size, uint32_t kind, uint32_t depth) {
    return make_uint2(start | (size - 1) << 12 | kind << 24, depth);
}
__device__ __forceinline__ uint32_t group_start(uint2 g) { return g.x & 0xFFFu; }
__device__ __forceinline__ uint32_t group_size(uint2 g) { return ((g.x >> 12) & 0xFFFu) + 1; }
__device__ __forceinline__ uint32_t group_kind(uint2 g) { return g.x >> 24; }

template <int CAP>
struct SegSmem {
    static constexpr int NB = CAP <= 256 ? 1024 : CAP <= 1024 ? 2048 : 4096;  // buckets
    unsigned long long key[CAP];
    uint32_t cnt[NB + 4];  // bucket counts, then starts (the last one the group's size)
    uint32_t id[CAP];
    uint2 wl[CAP / 2];         // groups for the warps
    uint32_t tl[CAP / 2];      // the pass's buckets of 2..TINY_MAX strings
    uint2 stk[CAP / 32 + 2];   // groups for the CTA
};

template <int CAP, int NT>
__global__ void __launch_bounds__(NT, CAP >= 4096 ? 2 : CAP >= 1024 ? 4 : 8) k_seg_sort(SortState S, const Seg* segs,
                                                                                       uint32_t nseg,
                                                                                       const uint32_t* dcount) {
    constexpr int NW = NT / 32, IPT = CAP / NT, NB = SegSmem<CAP>::NB, PER = NB / NT;
    extern __shared__ __align__(16) unsigned char smem[];
    SegSmem<CAP>& M = *reinterpret_cast<SegSmem<CAP>*>(smem);
    __shared__ unsigned long long s_or[NW], s_and[NW];
    __shared__ uint32_t s_sum[NW], s_ns, s_nw, s_nt, s_piv[8];
    __shared__ uint2 s_cur;
    __shared__ BucketBits s_bits;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (dcount) nseg = *dcount;
    for (uint32_t bi = blockIdx.x; bi < nseg; bi += gridDim.x) {
        const Seg seg = segs[bi];
        const uint32_t start = seg.start, size = seg.size;
        uint32_t* lcp = S.lcp_out + start;
        {
            const uint32_t* src = S.ord[seg.flags & F_PARITY] + start;
            const unsigned long long* ksrc = S.key[seg.flags & F_PARITY] + start;
            uint32_t o[IPT];
            uint64_t k[IPT];
#pragma unroll
            for (int j = 0; j < IPT; ++j) {
                const uint32_t i = threadIdx.x + j * NT;
                o[j] = i < size ? src[i] : 0u;
                k[j] = i < size && (seg.flags & F_KEYS) ? ksrc[i] : 0ull;
            }
            if (!(seg.flags & F_KEYS)) {
#pragma unroll
                for (int j = 0; j < IPT; ++j)
                    if (threadIdx.x + j * NT < size) k[j] = key8_of(S.a, o[j], seg.depth);
            }
#pragma unroll
            for (int j = 0; j < IPT; ++j) {
                const uint32_t i = threadIdx.x + j * NT;
                if (i < size) {
                    M.id[i] = o[j];
                    M.key[i] = k[j];
                }
            }
        }
        for (uint32_t x = threadIdx.x; x < NB; x += NT) M.cnt[x] = 0;
        if (threadIdx.x == 0) {
            const uint2 g = group_pack(0, size, G_PLAIN, seg.depth);
            s_nw = size <= 32;
            s_ns = size > 32;
            s_nt = 0;
            if (size <= 32) M.wl[0] = g;
            else M.stk[0] = g;
        }
        __syncthreads();
        while (s_ns) {
            if (threadIdx.x == 0) s_cur = M.stk[s_ns - 1];
            __syncthreads();
            const uint32_t bs = group_start(s_cur), bn = group_size(s_cur), dep = s_cur.y;
            uint32_t kind = group_kind(s_cur);
            if (threadIdx.x == 0) --s_ns;  // read again only after the next barrier
            uint64_t k[IPT];
            uint32_t o[IPT], br[IPT];
#pragma unroll
            for (int j = 0; j < IPT; ++j) {
                const uint32_t i = threadIdx.x + j * NT;
                o[j] = i < bn ? M.id[bs + i] : 0u;
                k[j] = i < bn ? (kind == G_ID ? (uint64_t)o[j] : M.key[bs + i]) : 0ull;
            }
            if (kind == G_TIE) {
                // the pivot: of 8 evenly spaced strings the one with the
                // largest sum of LCPs (256 bytes at most) with the others
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
                    if (lane == 0) s_piv[c] = sum << 3 | c;
                }
                __syncthreads();
                uint32_t best = 0;
#pragma unroll
                for (int c = 0; c < 8; ++c) best = max(best, s_piv[c]);
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
                    const uint32_t l = warp_lcp(S.a, x, h, dep, v);
                    if (v) M.key[bs + i] = pseudo_key(S.a, x, h, l, dep);
                }
                // a thread reads back only the keys it wrote
#pragma unroll
                for (int j = 0; j < IPT; ++j) {
                    const uint32_t i = threadIdx.x + j * NT;
                    if (i < bn) k[j] = M.key[bs + i];
                }
                kind = G_PSEUDO;
            }
            const bool pseudo = kind == G_PSEUDO;
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
                s_or[w] = (uint64_t)ohi << 32 | olo;
                s_and[w] = (uint64_t)ahi << 32 | alo;
            }
            __syncthreads();
            uint64_t diff;
            {
                uint64_t x = s_or[0], y = s_and[0];
#pragma unroll
                for (int v = 1; v < NW; ++v) {
                    x |= s_or[v];
                    y &= s_and[v];
                }
                diff = x ^ y;
            }
            if (diff == 0) {  // one key: equal strings, or the group goes deeper
                if (threadIdx.x == 0) {
                    const uint64_t k0 = k[0];
                    M.stk[s_ns++] = key_ended(k0, pseudo) ? group_pack(bs, bn, G_ID, ref_of(S.a, o[0]).len)
                                                          : group_pack(bs, bn, G_TIE, tie_depth(k0, dep, pseudo));
                }
                __syncthreads();
                continue;
            }
            if (threadIdx.x == 0) {
                constexpr uint32_t most = 31u - (uint32_t)__builtin_clz(NB);
                bucket_bits(s_bits, diff, pseudo ? most : min(32u - (uint32_t)__clz(bn - 1) + 1u, most));
            }
            __syncthreads();
            {
                const uint32_t lo = s_bits.lo, nr = s_bits.nruns;
                uint32_t x[IPT];
#pragma unroll
                for (int j = 0; j < IPT; ++j) {
                    x[j] = (uint32_t)(k[j] >> lo);
                    br[j] = 0;
                }
                for (uint32_t r = 0; r < nr; ++r) {
                    const uint32_t sh = s_bits.sh[r], mask = s_bits.mask[r];
                    if (s_bits.wide) {
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
                if (threadIdx.x + j * NT < bn) br[j] |= atomicAdd(&M.cnt[br[j]], 1u) << 16;
            __syncthreads();
            {
                uint32_t v[PER], sum = 0;
#pragma unroll
                for (int q = 0; q < PER; q += 4) {
                    const uint4 c = *reinterpret_cast<const uint4*>(&M.cnt[threadIdx.x * PER + q]);
                    v[q] = c.x;
                    v[q + 1] = c.y;
                    v[q + 2] = c.z;
                    v[q + 3] = c.w;
                    sum += c.x + c.y + c.z + c.w;
                }
                uint32_t x = sum;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const uint32_t y = __shfl_up_sync(FULL, x, off);
                    if (lane >= (uint32_t)off) x += y;
                }
                if (lane == 31) s_sum[w] = x;
                __syncthreads();
                uint32_t run = x - sum;
#pragma unroll
                for (int q = 0; q < NW; ++q)
                    if ((uint32_t)q < w) run += s_sum[q];
#pragma unroll
                for (int q = 0; q < PER; q += 4) {
                    uint4 c;
                    c.x = run;
                    c.y = c.x + v[q];
                    c.z = c.y + v[q + 1];
                    c.w = c.z + v[q + 2];
                    run = c.w + v[q + 3];
                    *reinterpret_cast<uint4*>(&M.cnt[threadIdx.x * PER + q]) = c;
                }
                if (threadIdx.x == NT - 1) M.cnt[NB] = run;
            }
            __syncthreads();
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
            const bool all = s_bits.all != 0, mixed = pseudo && s_bits.mixed;
#pragma unroll
            for (int j = 0; j < IPT; ++j) {
                if (threadIdx.x + j * NT >= bn || (br[j] >> 16) != 0) continue;
                const uint32_t b = br[j] & 0xFFFFu, s0 = M.cnt[b], c = M.cnt[b + 1] - s0;
                if (s0) {
                    uint64_t kp = M.key[bs + s0 - 1], kn = k[j];
                    if (mixed) {  // the codes next to the boundary: the last of the bucket before, this one's first
                        const uint32_t bp = bucket_of_key(s_bits, kp);
                        for (uint32_t x = s0 - 1; x > 0 && bucket_of_key(s_bits, M.key[bs + x - 1]) == bp; --x)
                            kp = max(kp, (uint64_t)M.key[bs + x - 1]);
                        for (uint32_t x = 0; x < c; ++x) kn = min(kn, (uint64_t)M.key[bs + s0 + x]);
                    }
                    lcp[bs + s0] = kind == G_ID ? dep : group_lcp(kp, kn, dep, pseudo);
                }
                if (c < 2) continue;
                if (c <= TINY_MAX) {
                    M.tl[atomicAdd(&s_nt, 1u)] = s0 | c << 16;
                    continue;
                }
                uint32_t gk = kind, gd = dep;
                if (kind != G_ID && all) {  // one key in the bucket
                    const bool ended = key_ended(k[j], pseudo);
                    gk = ended ? G_ID : G_TIE;
                    gd = ended ? ref_of(S.a, o[j]).len : tie_depth(k[j], dep, pseudo);
                }
                const uint2 g = group_pack(bs + s0, c, gk, gd);
                if (c <= 32) M.wl[atomicAdd(&s_nw, 1u)] = g;
                else M.stk[atomicAdd(&s_ns, 1u)] = g;
            }
            __syncthreads();
            // buckets of 2..TINY_MAX strings: insertion sort on (key, id), then
            // the neighbours' LCPs and the runs that go deeper
            const uint32_t nt = s_nt;
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
                            const uint32_t len = ref_of(S.a, M.id[s0 + r0]).len;
                            for (uint32_t y = r0 + 1; y < x; ++y) lcp[s0 + y] = len;
                        } else {
                            M.wl[atomicAdd(&s_nw, 1u)] = group_pack(s0 + r0, x - r0, G_TIE, tie_depth(kp, dep, pseudo));
                        }
                    }
                    if (x < c) lcp[s0 + x] = group_lcp(kp, kx, dep, pseudo);
                    kp = kx;
                    r0 = x;
                }
            }
            // the next pass counts from zero
            for (uint32_t x = threadIdx.x; x < NB; x += NT) M.cnt[x] = 0;
            __syncthreads();
            if (threadIdx.x == 0) s_nt = 0;  // pushed to again only after the next pass's barriers
        }
        const uint32_t nwl = s_nw;
        for (uint32_t e = w; e < nwl; e += NW) {
            const uint2 g = M.wl[e];
            const uint32_t ws = group_start(g), wn = group_size(g);
            uint64_t key = 0;
            uint32_t id = 0;
            if (lane < wn) {
                id = M.id[ws + lane];
                key = M.key[ws + lane];
            }
            warp_group(S.a, wn, g.y, group_kind(g), key, id, lcp + ws);
            if (lane < wn) M.id[ws + lane] = id;
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < size; i += NT) S.ord_out[start + i] = M.id[i];
        __syncthreads();  // shared memory is reused by the next segment
    }
}

template <int CAP>
constexpr size_t seg_sort_smem() {
    return sizeof(SegSmem<CAP>);
}

template <int CAP, int NT>
static int launch_seg_sort(const SortState& S, const Seg* segs, uint32_t n, const char* name, cudaStream_t st) {
    if (!n) return DSSS_OK;
    constexpr size_t shm = seg_sort_smem<CAP>();
    static std::atomic<uint64_t> configured{0};
    DSSS_TRY(set_smem_once(configured, k_seg_sort<CAP, NT>, (int)shm));
    DSSS_LAUNCH(name, st, k_seg_sort<CAP, NT><<<n, NT, shm, st>>>(S, segs, n, nullptr));
    DSSS_CUDA(cudaGetLastError());
    return DSSS_OK;
}


// ------------------------------------------------------- graph mode ----
// For n up to sort_graph_max_n (off by default) the MSD passes run as one CUDA graph: the pass
// is the body of a conditional WHILE node, the number of large segments and
// the parity of their list live on the device (counters[13], [12]), grids are
// the layout's capacities (blocks past the real tiles exit), and a one-thread
// kernel at the end of each pass sets the loop condition — no host round trip
// per pass.  The small-segment sorters then stride over the device counts.

// One block: per large segment its first tile and chunk (exclusive prefix
// over the list), totals into counters[8], [9]; resets the next-list count.
__global__ void __launch_bounds__(1024) k_seg_offsets(SortState S, Seg* segs, uint32_t nseg) {
    __shared__ uint32_t st_[1024], sc_[1024];
    if (!segs) {
        segs = S.large[S.counters[12]];
        nseg = S.counters[13];
    }
    const uint32_t per = (nseg + 1023) / 1024;
    const uint32_t b = min(nseg, threadIdx.x * per), e = min(nseg, b + per);
    uint32_t tt = 0, tc = 0;
    for (uint32_t i = b; i < e; ++i) {
        const uint32_t t = (segs[i].size + LT_TILE - 1) / LT_TILE;
        tt += t;
        tc += (t + CHUNK_TILES - 1) / CHUNK_TILES;
    }
    st_[threadIdx.x] = tt;
    sc_[threadIdx.x] = tc;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {
        const uint32_t vt = threadIdx.x >= (unsigned)off ? st_[threadIdx.x - off] : 0;
        const uint32_t vc = threadIdx.x >= (unsigned)off ? sc_[threadIdx.x - off] : 0;
        __syncthreads();
        st_[threadIdx.x] += vt;
        sc_[threadIdx.x] += vc;
        __syncthreads();
    }
    uint32_t rt = st_[threadIdx.x] - tt, rc = sc_[threadIdx.x] - tc;
    for (uint32_t i = b; i < e; ++i) {
        const uint32_t t = (segs[i].size + LT_TILE - 1) / LT_TILE;
        // keys folded by the previous scatter: the bits where they differ
        if (S.child && (segs[i].flags & (F_KEYS | F_PIVOT)) == F_KEYS) segs[i].diff = segs[i].kor ^ segs[i].kand;
        S.tile0[i] = rt;
        S.chunk0[i] = rc;
        rt += t;
        rc += (t + CHUNK_TILES - 1) / CHUNK_TILES;
    }
    if (threadIdx.x == 1023) {
        S.counters[8] = st_[1023];
        S.counters[9] = sc_[1023];
        if (st_[1023] > S.cap_tiles || sc_[1023] > S.cap_chunks) {
            S.counters[8] = 0;  // nothing runs; the guard stops the loop
            S.counters[9] = 0;
            S.counters[10] = 1;
        }
        S.counters[0] = 0;   // large segments of the next pass
        S.counters[11] = 0;  // of them, without keys or with a pivot pass
        S.counters[6] = 0;   // splitter tables of this pass
    }
}

__global__ void k_loop_init(SortState S, cudaGraphConditionalHandle h) {
    S.counters[12] = 0;
    S.counters[13] = S.counters[0];
    S.counters[14] = 0;
    cudaGraphSetConditional(h, S.counters[13] > 0 ? 1u : 0u);
}

// Ends a pass: the next list becomes current; loop while it is not empty,
// no guard tripped and the pass count stays sane.
__global__ void k_pass_end(SortState S, cudaGraphConditionalHandle h) {
    uint32_t next = S.counters[0];
    if (next > S.cap_large) {
        S.counters[10] = 1;
        next = 0;
    }
    S.counters[12] ^= 1u;
    S.counters[13] = next;
    const uint32_t passes = ++S.counters[14];
    if (passes > (1u << 20)) S.counters[10] = 1;
    cudaGraphSetConditional(h, (next > 0 && S.counters[10] == 0) ? 1u : 0u);
}

// Two streams per host thread and device to capture on (the caller's stream
// may be the legacy default stream, which cannot be captured); the graph is
// then launched on the caller's stream.
static int capture_streams(cudaStream_t* cap, cudaStream_t* body) {
    constexpr int MAXDEV = 64;
    thread_local cudaStream_t tl[MAXDEV][2] = {};
    int dev = 0;
    DSSS_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= MAXDEV) return fail(DSSS_ENOTSUP, "device %d out of range", dev);
    for (int k = 0; k < 2; ++k)
        if (!tl[dev][k]) DSSS_CUDA(cudaStreamCreateWithFlags(&tl[dev][k], cudaStreamNonBlocking));
    *cap = tl[dev][0];
    *body = tl[dev][1];
    return DSSS_OK;
}

static int sort_strings_graph(const SortLayout& L, SortState S, uint64_t n, uint32_t p, const uint32_t* ids_in,
                              uint32_t* pin, cudaStream_t run_st) {
    cudaStream_t st = nullptr, bst = nullptr;
    DSSS_TRY(capture_streams(&st, &bst));
    struct Res {
        cudaGraph_t g = nullptr;
        cudaGraphExec_t x = nullptr;
        ~Res() {
            if (x) cudaGraphExecDestroy(x);
            if (g) cudaGraphDestroy(g);
        }
    } res;
    const unsigned tiles = (unsigned)L.cap_tiles, chunks = (unsigned)L.cap_chunks, large = (unsigned)L.cap_large;
    DSSS_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    cudaMemsetAsync(L.counters, 0, 16 * sizeof(uint32_t), st);
    k_init_ids<<<grid_for(n, 256), 256, 0, st>>>(S.ord[0], ids_in, n);
    k_init_segs<<<grid_for(p, 128), 128, 0, st>>>(S, L.pb, p);
    cudaStreamCaptureStatus cs;
    cudaGraph_t g = nullptr;
    const cudaGraphNode_t* deps = nullptr;
    size_t ndeps = 0;
    cudaError_t e = cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, &deps, &ndeps);
    cudaGraphConditionalHandle h{};
    if (e == cudaSuccess) e = cudaGraphConditionalHandleCreate(&h, g, 0, 0);
    if (e == cudaSuccess) k_loop_init<<<1, 1, 0, st>>>(S, h);
    if (e == cudaSuccess) e = cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, &deps, &ndeps);
    cudaGraphNodeParams np{};
    np.type = cudaGraphNodeTypeConditional;
    np.conditional.handle = h;
    np.conditional.type = cudaGraphCondTypeWhile;
    np.conditional.size = 1;
    cudaGraphNode_t cond = nullptr;
    if (e == cudaSuccess) e = cudaGraphAddNode(&cond, g, deps, ndeps, &np);
    if (e == cudaSuccess) e = cudaStreamUpdateCaptureDependencies(st, &cond, 1, cudaStreamSetCaptureDependencies);
    if (e == cudaSuccess) {
        // the loop body: one MSD pass, captured on a second stream into the body graph
        cudaGraph_t body = np.conditional.phGraph_out[0];
        e = cudaStreamBeginCaptureToGraph(bst, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            k_seg_offsets<<<1, 1024, 0, bst>>>(S, nullptr, 0);
            k_prefix<<<tiles, LT_NT, 0, bst>>>(S, nullptr, 0);
            k_pivot<<<tiles, LT_NT, 0, bst>>>(S, nullptr, 0);
            k_keys_diff<<<tiles, LT_NT, 0, bst>>>(S, nullptr, 0);
            if (S.split_min) k_split_sample<<<148, SPL_SAMPLE / 2, 0, bst>>>(S, nullptr, 0);
            if (S.bits) k_hist<true><<<tiles, LT_NT, 0, bst>>>(S, nullptr, 0);
            else k_hist<false><<<tiles, LT_NT, 0, bst>>>(S, nullptr, 0);
            k_chunk_sum<<<chunks, 256, 0, bst>>>(S, nullptr, 0);
            k_seg_scan<<<large, 256, 0, bst>>>(S, nullptr, 0, nullptr);
            k_scatter<<<tiles, LT_NT, SCATTER_SMEM, bst>>>(S, nullptr, 0);
            k_pass_end<<<1, 1, 0, bst>>>(S, h);
            cudaGraph_t got = nullptr;
            e = cudaStreamEndCapture(bst, &got);
        }
    }
    if (e == cudaSuccess) {
        // small segments, striding over the device counts
        k_warp_segs<<<148 * 8, 128, 0, st>>>(S, S.small[0], 0, S.counters + 1);
        k_seg_sort<256, 128><<<148 * 8, 128, seg_sort_smem<256>(), st>>>(S, S.small[1], 0, S.counters + 2);
        k_seg_sort<1024, 256><<<148 * 4, 256, seg_sort_smem<1024>(), st>>>(S, S.small[2], 0, S.counters + 3);
        k_seg_sort<4096, 512><<<148 * 2, 512, seg_sort_smem<4096>(), st>>>(S, S.small[3], 0, S.counters + 4);
        if (S.split_min) k_lcp_fix<<<148 * 4, 256, 0, st>>>(S);
        cudaMemcpyAsync(pin, L.counters, 16 * sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
    }
    cudaGraph_t whole = nullptr;
    const cudaError_t e2 = cudaStreamEndCapture(st, &whole);
    res.g = whole;
    if (e != cudaSuccess || e2 != cudaSuccess)
        return fail(DSSS_EDEVICE, "string sort graph: %s", cudaGetErrorString(e != cudaSuccess ? e : e2));
    DSSS_CUDA(cudaGraphInstantiate(&res.x, whole, 0));
    {
        StageTimer t("graph:sort", run_st);
        DSSS_CUDA(cudaGraphLaunch(res.x, run_st));
    }
    DSSS_CUDA(cudaStreamSynchronize(run_st));
    if (pin[10]) return fail(DSSS_EDEVICE, "string sort: internal consistency guard tripped");
    return DSSS_OK;
}

// ------------------------------------------------------------------ host ----
static Seg* large_list(const SortLayout& L, int k) { return (Seg*)L.large[k]; }
static uint32_t clamp_small_max(uint32_t m) {
    if (m == 0) m = (uint32_t)tune(TUNE_SORT_SMALL_MAX);
    return (m == 0 || m > (uint32_t)bin_cap(NBINS - 1)) ? (uint32_t)bin_cap(NBINS - 1) : (m < 2 ? 2 : m);
}

void layout_sort(Carve& c, SortLayout& L, uint64_t n, uint32_t p, uint32_t small_max) {
    small_max = clamp_small_max(small_max);
    uint64_t N = n ? n : 1;
    L.ord[0] = c.take<uint32_t>(N);
    L.ord[1] = c.take<uint32_t>(N);
    L.key[0] = c.take<unsigned long long>(N);
    L.key[1] = c.take<unsigned long long>(N);
    L.cap_large = N / (small_max + 1) + p + 1;
    L.cap_small = N / 2 + p + 1;
    L.cap_tiles = N / LT_TILE + L.cap_large + 1;
    L.cap_chunks = L.cap_tiles / CHUNK_TILES + L.cap_large + 1;
    L.large[0] = c.take<unsigned char>(L.cap_large * sizeof(Seg));
    L.large[1] = c.take<unsigned char>(L.cap_large * sizeof(Seg));
    for (int b = 0; b < NBINS; ++b) L.small[b] = c.take<unsigned char>(L.cap_small * sizeof(Seg));
    L.tile0 = c.take<uint32_t>(L.cap_large);
    L.chunk0 = c.take<uint32_t>(L.cap_large);
    L.tmp_counts = c.take<uint32_t>(2 * L.cap_large);
    L.tile_hist = c.take<uint32_t>(L.cap_tiles * 256);
    L.chunk_pre = c.take<uint32_t>(L.cap_chunks * 256);
    L.bucket = c.take<uint32_t>(L.cap_large * 257);
    // the child table: 256 slots per large segment, about 4 bytes per string
    // once large segments hold more than 256 strings (smaller cut-offs keep
    // the per-pass key reads instead)
    L.child = small_max >= 256 ? c.take<uint32_t>(L.cap_large * 256) : nullptr;
    L.counters = c.take<uint32_t>(16);
    L.pb = c.take<uint64_t>(p + 1);
    L.scan = c.take<unsigned char>(scan_scratch_bytes(L.cap_large));
    // splitter tables: segments of at least SPL_MIN_FLOOR strings per pass;
    // fix list: (position, depth) pairs (when it runs short, passes keep the
    // byte digit)
    L.cap_spl = N / SPL_MIN_FLOOR + p + 1;
    L.spl = c.take<unsigned long long>(L.cap_spl * SPL_STRIDE);
    L.cap_fix = N / 16 + 65536;
    L.fix = c.take<uint32_t>(2 * L.cap_fix);
    L.pin = nullptr;
}

int sort_strings(const SortLayout& L, const ArenaDev& a, uint64_t n, uint32_t p, const uint64_t* pb_host,
                 const uint32_t* ids_in, uint32_t* ord_out, uint32_t* lcp_out, uint32_t small_max,
                 uint32_t* pin, cudaStream_t st, const uint32_t* seg_depth) {
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
    for (int b = 0; b < NBINS; ++b) S.small[b] = (Seg*)L.small[b];
    S.tile0 = L.tile0;
    S.chunk0 = L.chunk0;
    S.tmp_counts = L.tmp_counts;
    S.tile_hist = L.tile_hist;
    S.chunk_pre = L.chunk_pre;
    S.bucket = L.bucket;
    S.counters = L.counters;
    S.child = L.child;
    S.nxt = nullptr;
    S.small_max = clamp_small_max(small_max);
    S.pivot = tune(TUNE_SORT_PIVOT) ? 1u : 0u;
    S.bits = (uint32_t)tune(TUNE_SORT_BITS);
    S.first = 0;
    S.cap_large = L.cap_large;
    S.cap_small = L.cap_small;
    S.cap_tiles = L.cap_tiles;
    S.cap_chunks = L.cap_chunks;
    {
        const int64_t v = tune(TUNE_SORT_SPLIT_MIN);
        S.split_min = v <= 0 ? 0u : (uint32_t)std::min<int64_t>(std::max<int64_t>(v, SPL_MIN_FLOOR), 0xFFFFFFFFll);
    }
    S.seg_depth = seg_depth;
    S.spl = L.spl;
    S.fix = L.fix;
    S.cap_spl = L.cap_spl;
    S.cap_fix = L.cap_fix;
    static std::atomic<uint64_t> scatter_configured{0};
    DSSS_TRY(set_smem_once(scatter_configured, k_scatter, (int)SCATTER_SMEM));
    DSSS_CUDA(cudaMemcpyAsync(L.pb, pb_host, (p + 1) * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
    if (n <= (uint64_t)tune(TUNE_SORT_GRAPH)) {
        static std::atomic<uint64_t> c256{0}, c1024{0}, c4096{0};
        DSSS_TRY(set_smem_once(c256, k_seg_sort<256, 128>, (int)seg_sort_smem<256>()));
        DSSS_TRY(set_smem_once(c1024, k_seg_sort<1024, 256>, (int)seg_sort_smem<1024>()));
        DSSS_TRY(set_smem_once(c4096, k_seg_sort<4096, 512>, (int)seg_sort_smem<4096>()));
        S.large[0] = large_list(L, 0);
        S.large[1] = large_list(L, 1);
        S.child = nullptr;  // every pass of the graph reads the keys itself
        return sort_strings_graph(L, S, n, p, ids_in, pin, st);
    }
    DSSS_CUDA(cudaMemsetAsync(L.counters, 0, 16 * sizeof(uint32_t), st));
    DSSS_LAUNCH("k_init_ids", st, k_init_ids<<<grid_for(n, 256), 256, 0, st>>>(S.ord[0], ids_in, n));
    S.large[0] = large[0];
    S.large[1] = large[1];
    DSSS_LAUNCH("k_init_segs", st, k_init_segs<<<grid_for(p, 128), 128, 0, st>>>(S, L.pb, p));
    DSSS_CUDA(cudaGetLastError());
    DSSS_CUDA(cudaMemcpyAsync(pin, L.counters, 16 * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    DSSS_CUDA(cudaStreamSynchronize(st));
    uint32_t nlarge = pin[0];
    int cur = 0;
    uint32_t guard = 0;
    S.first = 1;
    // whether the list holds a segment without keys folded by the previous
    // scatter (no keys, a pivot pass, or the first pass): only then the
    // prefix, pivot and key passes run
    bool keyless = true;
    while (nlarge) {
        if (++guard > (1u << 24)) return fail(DSSS_EDEVICE, "string sort made no progress");
        Seg* segs = large[cur];
        Seg* next = large[cur ^ 1];
        // tile / chunk indexing
        // tile / chunk indexing (and the next list's count reset): one block
        DSSS_LAUNCH("k_seg_offsets", st, k_seg_offsets<<<1, 1024, 0, st>>>(S, segs, nlarge));
        // upper bounds for the grids (kernels exit past the real counts)
        uint64_t max_tiles = std::min<uint64_t>(L.cap_tiles, n / LT_TILE + nlarge + 1);
        uint64_t max_chunks = std::min<uint64_t>(L.cap_chunks, max_tiles / CHUNK_TILES + nlarge + 1);
        S.large[0] = segs;
        S.nxt = next;
        if (keyless) {
            DSSS_LAUNCH("k_spec", st, k_spec<<<std::min<uint32_t>(nlarge, 148 * 16), 256, 0, st>>>(S, segs, nlarge));
            DSSS_LAUNCH("k_prefix", st, k_prefix<<<(unsigned)max_tiles, LT_NT, 0, st>>>(S, segs, nlarge));
            DSSS_LAUNCH("k_pivot", st, k_pivot<<<(unsigned)max_tiles, LT_NT, 0, st>>>(S, segs, nlarge));
            DSSS_LAUNCH("k_keys_diff", st, k_keys_diff<<<(unsigned)max_tiles, LT_NT, 0, st>>>(S, segs, nlarge));
        }
        if (S.split_min)
            DSSS_LAUNCH("k_split_sample", st,
                        k_split_sample<<<std::min<uint32_t>(nlarge, 148 * 2), SPL_SAMPLE / 2, 0, st>>>(S, segs, nlarge));
        // the bit-digit histogram only in passes that can split on bits (its
        // tables and registers cost the byte form's occupancy)
        if (S.bits && (S.bits != 3 || S.first))
            DSSS_LAUNCH("k_hist", st, k_hist<true><<<(unsigned)max_tiles, LT_NT, 0, st>>>(S, segs, nlarge));
        else
            DSSS_LAUNCH("k_hist", st, k_hist<false><<<(unsigned)max_tiles, LT_NT, 0, st>>>(S, segs, nlarge));
        DSSS_LAUNCH("k_chunk_sum", st, k_chunk_sum<<<(unsigned)max_chunks, 256, 0, st>>>(S, segs, nlarge));
        DSSS_LAUNCH("k_seg_scan", st, k_seg_scan<<<nlarge, 256, 0, st>>>(S, segs, nlarge, next));
        DSSS_LAUNCH("k_scatter", st, k_scatter<<<(unsigned)max_tiles, LT_NT, SCATTER_SMEM, st>>>(S, segs, nlarge));
        DSSS_CUDA(cudaGetLastError());
        DSSS_CUDA(cudaMemcpyAsync(pin, L.counters, 16 * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
        DSSS_CUDA(cudaStreamSynchronize(st));
        nlarge = pin[0];
        keyless = !S.child || pin[11] != 0;
        if (pin[10]) return fail(DSSS_EDEVICE, "string sort: internal consistency guard tripped");
        if (nlarge > L.cap_large) return fail(DSSS_EDEVICE, "string sort: large-segment list overflow");
        cur ^= 1;
        S.first = 0;
    }
    for (int b = 0; b < NBINS; ++b)
        if (pin[1 + b] > L.cap_small) return fail(DSSS_EDEVICE, "string sort: small-segment list overflow");
    if (pin[1]) {
        DSSS_LAUNCH("k_warp_segs", st, k_warp_segs<<<(pin[1] + 3) / 4, 128, 0, st>>>(S, S.small[0], pin[1], nullptr));
        DSSS_CUDA(cudaGetLastError());
    }
    DSSS_TRY((launch_seg_sort<256, 128>(S, S.small[1], pin[2], "k_seg_sort256", st)));
    DSSS_TRY((launch_seg_sort<1024, 256>(S, S.small[2], pin[3], "k_seg_sort1024", st)));
    DSSS_TRY((launch_seg_sort<4096, 512>(S, S.small[3], pin[4], "k_seg_sort4096", st)));
    if (pin[5]) DSSS_LAUNCH("k_lcp_fix", st, k_lcp_fix<<<grid_for(std::min<uint64_t>(pin[5], L.cap_fix), 256), 256, 0, st>>>(S));
    DSSS_CUDA(cudaMemcpyAsync(pin, L.counters, 16 * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    DSSS_CUDA(cudaStreamSynchronize(st));
    if (pin[10]) return fail(DSSS_EDEVICE, "string sort: internal consistency guard tripped");
    return DSSS_OK;
}

}  // namespace dsss
