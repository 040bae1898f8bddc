// What every PE holds, cuts and receives, read off one global sorted order.
//
// The full path on one GPU sorts all strings once.  Position g of that order
// belongs to the PE that holds its string; a PE's local sorted order
// (radixsort_CI3 per PE, prefix_doubling.hpp:228) is the subsequence of its
// positions, and each position's rank in it is all that partitioning needs:
//   samples   : PE q's samples are the ranks floor(i * n_q / (nr + 1)), in
//               double arithmetic (samplingStrategies.hpp:57-89, 148-184);
//   order     : samples cut to their distinguishing prefixes (or to a length
//               that keeps equal cut samples adjacent) sort as their global
//               positions do, ties by (PE, index) included;
//   splitters : the sample of sorted rank k * (total / (nr' + 1))
//               (getSplitters, misc.hpp:89-189) is found by bisecting the
//               global order on the number of samples before a position;
//   bounds    : the reference's binary search of a splitter in PE q's strings
//               (misc.hpp:310-374) sees a probe as smaller, equal or greater
//               by its rank alone, once q's ranks below and inside the run of
//               strings equal to the splitter are known.
// No sample is gathered, sorted or compared (except where a splitter has
// equal neighbours), and nothing is read back between these steps.
//
// The receiving PEs' merged sequences are the global order itself unless
// equal strings on different PEs are cut on different sides of a splitter
// (flags[1]): then pe[g] and rank[g] already are the (index, PE) permutation.
#include <algorithm>
#include <cstring>

#include "dp.cuh"
#include "internal.cuh"
#include "project.cuh"
#include "util.cuh"

namespace dsss {

constexpr int PJ_NT = 256, PJ_IPT = 8, PJ_TILE = PJ_NT * PJ_IPT, PJ_NW = PJ_NT / 32;
constexpr unsigned PJ_FULL = 0xffffffffu;

// ------------------------------------------------------------- local orders --
// PE of every position and the PE counts of each tile.  The PE bounds are
// looked up in shared memory: the PE that equal parts would give, or one of
// its neighbours; PEs of very uneven sizes fall back to a binary search.
// Bound by the 4-byte id read and the 4-byte PE written per position (one pass
// where finding the PEs and counting them were two).
__global__ void __launch_bounds__(PJ_NT) k_pe_hist(const uint32_t* ord, uint64_t n, const uint64_t* pb, uint32_t npe,
                                                   uint32_t p, uint64_t tiles, uint32_t* pe, uint32_t* bucket,
                                                   uint32_t* hist) {
    extern __shared__ uint32_t spb[];
    uint32_t* h = spb + npe + 1;  // a row of npe counts per warp
    for (uint32_t q = threadIdx.x; q <= npe; q += PJ_NT) spb[q] = (uint32_t)pb[q];  // n < 2^32
    for (uint32_t q = threadIdx.x; q < npe * PJ_NW; q += PJ_NT) h[q] = 0;
    const uint64_t g0 = (uint64_t)blockIdx.x * PJ_TILE + threadIdx.x;
    uint32_t s[PJ_IPT];
#pragma unroll
    for (int j = 0; j < PJ_IPT; ++j) {
        const uint64_t g = g0 + (uint64_t)j * PJ_NT;
        s[j] = g < n ? ord[g] : 0u;
    }
    __syncthreads();
    const float scale = (float)npe / (float)max(spb[npe], 1u);
    uint32_t q[PJ_IPT];
#pragma unroll
    for (int j = 0; j < PJ_IPT; ++j) q[j] = min(npe - 1, (uint32_t)((float)s[j] * scale));
    uint32_t* hw = h + (threadIdx.x >> 5) * npe;
#pragma unroll
    for (int j = 0; j < PJ_IPT; ++j) {
        const uint64_t g = g0 + (uint64_t)j * PJ_NT;
        if (g >= n) continue;
        uint32_t r = q[j];
        if (spb[r] > s[j] || spb[r + 1] <= s[j]) {
            // off by one (r stays in range: spb[0] = 0, spb[npe] = n > s), or
            // further: the last r < npe with pb[r] <= s
            r = spb[r] > s[j] ? r - 1 : r + 1;
            if (spb[r] > s[j] || spb[r + 1] <= s[j]) {
                r = 0;
                for (uint32_t st = 1u << (31 - __clz(npe | 1u)); st; st >>= 1)
                    if (r + st < npe && spb[r + st] <= s[j]) r += st;
            }
        }
        pe[g] = p < npe ? r % p : r;
        if (bucket != pe) bucket[g] = r;
        atomicAdd(&hw[r], 1u);
    }
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < npe; b += PJ_NT) {
        uint32_t t = 0;
#pragma unroll
        for (int w = 0; w < PJ_NW; ++w) t += h[w * npe + b];
        hist[(uint64_t)b * tiles + blockIdx.x] = t;
    }
}

// Where a tile leaves the local LCPs open: per PE and tile the least LCP up to
// the PE's first string (PJ_NONE: it has none here) and from behind its last
// one to the tile's end, both PE-major, and each tile's least LCP.
struct LcpEdges {
    uint32_t *head, *tail, *tmin;
    unsigned long long* sum;
};
constexpr uint32_t PJ_NONE = 0xFFFFFFFFu;

// Stable scatter of every position's id (and distinguishing prefix, computed
// here from the LCPs) to its PE's local order, and its rank there.  The tile
// is reordered by PE in shared memory, so that each PE's run is written
// contiguously.  Bound by shared-memory latency (the stable rank), then by 24
// bytes moved per position.  Peers by ballots instead of a match instruction:
// 0.36 -> 0.25 ms on 32e6 strings and 64 PEs.
//
// Without DP it sums the PEs' local LCPs instead (the merge-sort path needs
// their average alone): two strings that follow one another on a PE have the
// least LCP of the global order between them, which blocks' prefix and suffix
// minima in shared memory give; what crosses tiles is left to
// k_local_lcp_edges.  Comparing the strings themselves again read every
// string's first bytes in random order: 8e6 strings 0.53 ms in all, now 0.17 ms.
template <bool DP>
constexpr size_t pj_scatter_smem(uint32_t P) {
    return (size_t)PJ_TILE * (DP ? 8 + 2 : 4 * 4 + 2 * 2) + (size_t)P * 4 * (3 + PJ_NW);
}

template <bool DP>
__global__ void __launch_bounds__(PJ_NT, 5) k_local_scatter(const uint32_t* bucket, const uint32_t* ord,
                                                            const uint32_t* lcp, const uint32_t* len,
                                                            const LenStats* stats, uint64_t n, uint32_t P,
                                                            uint64_t tiles, const uint32_t* off, const uint64_t* pb,
                                                            uint32_t* local_order,
                                                            uint32_t* dp, LcpEdges E, uint32_t* rank,
                                                            uint32_t* err) {
    extern __shared__ __align__(16) uint32_t pj_sm[];
    uint32_t* sid = pj_sm;                                       // PJ_TILE
    uint32_t* sdp = sid + PJ_TILE;                               // PJ_TILE; !DP: the tile's LCPs
    uint32_t* pmin = sdp + PJ_TILE;                              // PJ_TILE (!DP): least LCP from the block of 32's start
    uint32_t* smin = pmin + PJ_TILE;                             // PJ_TILE (!DP): least LCP to the block's end
    uint16_t* sbk = (uint16_t*)(sid + (DP ? 2 : 4) * PJ_TILE);   // PJ_TILE
    uint16_t* spos = sbk + PJ_TILE;                              // PJ_TILE (!DP)
    uint32_t* base = (uint32_t*)(sbk + (DP ? 1 : 2) * PJ_TILE);  // P
    uint32_t* first = base + P;                                  // P
    uint32_t* tloff = first + P;                                 // P
    uint32_t* wcnt = tloff + P;                                  // PJ_NW x P
    __shared__ uint32_t wsum[PJ_NW];
    for (uint32_t b = threadIdx.x; b < P; b += PJ_NT) {
        base[b] = off[(uint64_t)b * tiles + blockIdx.x];
        first[b] = (uint32_t)pb[b];  // where the PE's strings start
#pragma unroll
        for (int w = 0; w < PJ_NW; ++w) wcnt[w * P + b] = 0;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint64_t tb = (uint64_t)blockIdx.x * PJ_TILE;
    const uint32_t tn = (uint32_t)min((uint64_t)PJ_TILE, n - tb);
    const uint64_t wb = tb + (uint64_t)w * 32 * PJ_IPT;
    const uint32_t minlen = DP ? stats->min_len() : 0u;
    // everything the tile reads is in flight before the ranking starts
    uint32_t rk[PJ_IPT], bk[PJ_IPT], id[PJ_IPT], dv[PJ_IPT];
#pragma unroll
    for (int j = 0; j < PJ_IPT; ++j) {
        const uint64_t i = wb + j * 32 + lane;
        id[j] = i < n ? ord[i] : 0u;
        bk[j] = i < n ? bucket[i] : 0xFFFFFFFFu - lane;
        dv[j] = 0;
        if (DP) dv[j] = max(i && i < n ? lcp[i] : 0u, i + 1 < n ? lcp[i + 1] : 0u);
    }
    if (DP) {
#pragma unroll
        for (int j = 0; j < PJ_IPT; ++j) {
            uint64_t d = dp_depth_above(dv[j]);
            if (d > minlen && wb + j * 32 + lane < n) d = min(d, (uint64_t)len[id[j]]);
            dv[j] = (uint32_t)d;
        }
    } else {
#pragma unroll
        for (int j = 0; j < PJ_IPT; ++j) {
            const uint64_t i = wb + j * 32 + lane;
            const uint32_t t = w * 32 * PJ_IPT + j * 32 + lane, v = i < n ? lcp[i] : PJ_NONE;
            uint32_t up = v, down = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t x = __shfl_up_sync(PJ_FULL, up, o), y = __shfl_down_sync(PJ_FULL, down, o);
                if (lane >= o) up = min(up, x);
                if (lane + o < 32) down = min(down, y);
            }
            sdp[t] = v;
            pmin[t] = up;
            smin[t] = down;
        }
    }
    // the lanes with the same PE (one ballot per bit of the PE number), all
    // rounds independent of one another; then the warp's running counts
    uint32_t peers[PJ_IPT];
#pragma unroll
    for (int j = 0; j < PJ_IPT; ++j) peers[j] = same_lanes(bk[j], wb + j * 32 + lane < n, P);
#pragma unroll
    for (int j = 0; j < PJ_IPT; ++j) {
        const bool v = wb + j * 32 + lane < n;
        const uint32_t prev = v ? wcnt[w * P + bk[j]] : 0;
        __syncwarp();
        if (v && lane == __ffs(peers[j]) - 1) wcnt[w * P + bk[j]] = prev + __popc(peers[j]);
        __syncwarp();
        rk[j] = prev + __popc(peers[j] & ((1u << lane) - 1));
    }
    __syncthreads();
    // exclusive over warps per PE, then over PEs within the tile (each thread
    // a contiguous run of PEs, block scan of the run sums)
    const uint32_t per = (P + PJ_NT - 1) / PJ_NT;
    const uint32_t c0 = min(P, threadIdx.x * per), c1 = min(P, c0 + per);
    uint32_t sum = 0;
    for (uint32_t b = c0; b < c1; ++b) {
        uint32_t run = 0;
#pragma unroll
        for (int ww = 0; ww < PJ_NW; ++ww) {
            const uint32_t v = wcnt[ww * P + b];
            wcnt[ww * P + b] = run;
            run += v;
        }
        tloff[b] = run;
        sum += run;
    }
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(PJ_FULL, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    uint32_t run = x - sum;
    for (int ww = 0; ww < w; ++ww) run += wsum[ww];
    for (uint32_t b = c0; b < c1; ++b) {
        const uint32_t v = tloff[b];
        tloff[b] = run;
        run += v;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < PJ_IPT; ++j) {
        const uint64_t i = wb + j * 32 + lane;
        if (i >= n) continue;
        const uint32_t d = bk[j];
        const uint32_t in_tile = wcnt[w * P + d] + rk[j];
        const uint32_t lp = tloff[d] + in_tile;
        if (lp >= tn) {  // never taken when the counts agree
            atomicExch(err, 1u);
            continue;
        }
        sid[lp] = id[j];
        if (DP) sdp[lp] = dv[j];
        else spos[lp] = (uint16_t)(i - tb);
        sbk[lp] = (uint16_t)d;
        rank[i] = base[d] - first[d] + in_tile;
    }
    __syncthreads();
    for (uint32_t xx = threadIdx.x; xx < tn; xx += PJ_NT) {
        const uint32_t d = sbk[xx];
        const uint64_t dest = (uint64_t)base[d] + (xx - tloff[d]);
        if (dest >= n) {
            atomicExch(err, 1u);
            continue;
        }
        local_order[dest] = sid[xx];
        if (DP) dp[dest] = sdp[xx];
    }
    if (DP) return;
    // the least LCP over the tile's positions from .. to
    auto least = [&](uint32_t from, uint32_t to) {
        const uint32_t fb = from / 32, lb = to / 32;
        uint32_t m = PJ_NONE;
        if (fb == lb) {
            for (uint32_t t = from; t <= to; ++t) m = min(m, sdp[t]);
        } else {
            m = min(smin[from], pmin[to]);
            for (uint32_t b = fb + 1; b < lb; ++b) m = min(m, smin[b * 32]);
        }
        return m;
    };
    unsigned long long total = 0;
    for (uint32_t xx = threadIdx.x; xx < tn; xx += PJ_NT) {
        const uint32_t d = sbk[xx], t = spos[xx];
        const uint64_t cell = (uint64_t)d * tiles + blockIdx.x;
        if (xx > tloff[d]) total += least(spos[xx - 1] + 1u, t);
        else E.head[cell] = least(0, t);
        if (xx + 1 == tn || sbk[xx + 1] != d) E.tail[cell] = t + 1 < tn ? least(t + 1, tn - 1) : PJ_NONE;
    }
    for (uint32_t b = threadIdx.x; b < P; b += PJ_NT)
        if (tloff[b] == (b + 1 < P ? tloff[b + 1] : tn)) E.head[(uint64_t)b * tiles + blockIdx.x] = PJ_NONE;
    if (w == 0) {
        static_assert(PJ_TILE == 64 * 32, "two blocks per lane");
        const uint32_t m = __reduce_min_sync(PJ_FULL, min(smin[lane * 32], smin[(lane + 32) * 32]));
        if (lane == 0) E.tmin[blockIdx.x] = m;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) total += __shfl_xor_sync(PJ_FULL, total, o);
    if (lane == 0 && total) atomicAdd(E.sum, total);
}

// The local LCPs that cross tiles: one block per PE, a contiguous run of tiles
// per thread, the runs combined in order.  A run holds the least LCP up to its
// first string (all of it if it has none), the least one behind its last
// string, and the sum between.
struct LcpRun {
    uint32_t has, head, tail;
    unsigned long long sum;
};
__device__ __forceinline__ void lcp_run_append(LcpRun& a, const LcpRun& b) {
    a.sum += b.sum;
    if (a.has && b.has) a.sum += min(a.tail, b.head);
    if (!a.has) a.head = min(a.head, b.head);
    a.tail = b.has ? b.tail : min(a.tail, b.head);
    a.has |= b.has;
}

__global__ void __launch_bounds__(PJ_NT) k_local_lcp_edges(LcpEdges E, uint64_t tiles) {
    __shared__ LcpRun s_run[PJ_NW];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint64_t per = (tiles + PJ_NT - 1) / PJ_NT, t0 = threadIdx.x * per, t1 = min(tiles, t0 + per);
    const uint32_t *head = E.head + blockIdx.x * tiles, *tail = E.tail + blockIdx.x * tiles;
    LcpRun r{0u, PJ_NONE, PJ_NONE, 0ull};
    for (uint64_t t = t0; t < t1; ++t) {
        const uint32_t h = head[t];
        const LcpRun x{h != PJ_NONE, h != PJ_NONE ? h : E.tmin[t], h != PJ_NONE ? tail[t] : PJ_NONE, 0ull};
        lcp_run_append(r, x);
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        LcpRun x;
        x.has = __shfl_down_sync(PJ_FULL, r.has, o);
        x.head = __shfl_down_sync(PJ_FULL, r.head, o);
        x.tail = __shfl_down_sync(PJ_FULL, r.tail, o);
        x.sum = __shfl_down_sync(PJ_FULL, r.sum, o);
        if (lane + o < 32) lcp_run_append(r, x);  // what lanes not at a multiple of 2 o hold is not read again
    }
    if (lane == 0) s_run[w] = r;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 1; q < PJ_NW; ++q) lcp_run_append(r, s_run[q]);
        if (r.sum) atomicAdd(E.sum, r.sum);
    }
}

// --------------------------------------------------------------- splitters --
// Samples of a PE of nq strings (nr of them, dist = nq / (nr + 1) apart) at
// ranks below c: the number of i in 1..nr with floor(i * dist) < c.
__device__ __forceinline__ uint32_t samples_below(uint32_t c, uint32_t nr, double dist) {
    if (c == 0 || nr == 0) return 0;
    const double e = (double)c / dist;
    uint32_t i = e < (double)nr ? (uint32_t)e : nr;
    while (i > 0 && (uint64_t)((double)i * dist) >= c) --i;
    while (i < nr && (uint64_t)((double)(i + 1) * dist) < c) ++i;
    return i;
}

struct SplitArgs {
    ArenaDev a;
    uint64_t n, tiles;
    uint32_t p, factor;
    int indexed;
    const SetSplit* sets;
    const uint64_t* pb;
    const uint32_t *off, *ord, *lcp, *bucket, *rank;
    const unsigned long long* cut;
    uint32_t *bounds, *start, *flags;
};

// Whether the first T bytes of strings x and y (both at least T long) agree,
// by the 32 lanes of a warp, 8 bytes each per step.
__device__ __forceinline__ bool same_prefix(const uint8_t* chars, uint64_t ox, uint64_t oy, uint32_t T, uint32_t lane) {
    for (uint32_t d = 0; d < T; d += 256) {
        const uint32_t at = d + 8 * lane;
        const bool diff = at < T && key8(chars, ox, T, at) != key8(chars, oy, T, at);
        if (__any_sync(PJ_FULL, diff)) return false;
    }
    return true;
}

// Bisection of (lo, hi) by the block's warps, one probe each per round:
// pred(x) is evaluated by a whole warp and true for all x up to some point.
// Returns the last x in [lo, hi) with pred true, given pred(lo) (not
// evaluated).  Every thread of the block calls it.
template <typename F>
__device__ __forceinline__ uint64_t block_bisect(uint64_t lo, uint64_t hi, uint32_t* ok, F pred) {
    const uint32_t w = threadIdx.x >> 5;
    while (hi - lo > 1) {
        const uint64_t span = hi - lo;
        const uint64_t x = lo + span * (w + 1) / (PJ_NW + 1);
        const bool t = x == lo || pred(x);  // the same for the whole warp
        if ((threadIdx.x & 31) == 0) ok[w] = t;
        __syncthreads();
        uint64_t nl = lo, nh = hi;
#pragma unroll
        for (int k = 0; k < PJ_NW; ++k) {
            const uint64_t xk = lo + span * (k + 1) / (PJ_NW + 1);
            if (ok[k]) nl = max(nl, xk);
            else nh = min(nh, xk);
        }
        __syncthreads();
        lo = nl;
        hi = nh;
    }
    return lo;
}

// One block per receiver (set, k): for 1 <= k <= nspl the set's k-th splitter
// and bounds[.][k] of all its PEs, else the fixed bounds.  Latency-bound (a
// handful of dependent global reads per block, all blocks at once); the sample
// sort, its read-backs and the string searches that it replaces took 0.25 ms
// of the smallest call and 0.5 ms of one with 64 PEs.
__global__ void __launch_bounds__(PJ_NT) k_splitters(SplitArgs S) {
    extern __shared__ __align__(16) unsigned char pj_spl[];
    const uint32_t p = S.p, set = blockIdx.x / p, k = blockIdx.x % p;
    double* sdist = reinterpret_cast<double*>(pj_spl);         // p
    uint32_t* snr = reinterpret_cast<uint32_t*>(sdist + p);    // p
    uint32_t* row0 = snr + p;                                  // p: first slot of the PE's row in off
    uint32_t* cl = row0 + p;                                   // p: ranks below the splitter's run
    uint32_t* cu = cl + p;                                     // p: ranks up to the run's end
    __shared__ uint32_t ok[PJ_NW], ws[PJ_NW], s_before, s_minr, s_maxl;
    __shared__ unsigned long long s_g;
    const SetSplit sp = S.sets[set];
    const uint64_t* pb = S.pb + (uint64_t)set * p;
    const uint32_t* off = S.off + (uint64_t)set * p * S.tiles;
    uint32_t* bounds = S.bounds + (uint64_t)set * p * (p + 1);
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (k == 0 || k > sp.nspl) {
        for (uint32_t q = threadIdx.x; q < p; q += PJ_NT) {
            const uint32_t nq = (uint32_t)(pb[q + 1] - pb[q]);
            bounds[(uint64_t)q * (p + 1) + k] = k ? nq : 0u;
            if (k == 0) bounds[(uint64_t)q * (p + 1) + p] = nq;
        }
        if (threadIdx.x == 0) S.start[blockIdx.x] = 0xFFFFFFFFu;
        return;
    }
    for (uint32_t q = threadIdx.x; q < p; q += PJ_NT) {
        const uint64_t nq = pb[q + 1] - pb[q];
        const uint64_t nr = min((uint64_t)S.factor * (p - 1), nq);
        snr[q] = (uint32_t)nr;
        sdist[q] = (double)nq / (double)(nr + 1);
        row0[q] = off[(uint64_t)q * S.tiles];
    }
    if (threadIdx.x == 0) {
        s_before = 0;
        s_g = ~0ull;
        s_minr = 0xFFFFFFFFu;
        s_maxl = 0;
    }
    __syncthreads();
    // the last tile with at most r samples before it, r the splitter's rank
    const uint32_t r = k * sp.dist;
    const uint64_t t0 = sp.begin / PJ_TILE, t1 = (sp.end - 1) / PJ_TILE + 1;
    const uint64_t t = block_bisect(t0, t1, ok, [&](uint64_t x) {
        uint32_t c = 0;
        for (uint32_t q = lane; q < p; q += 32)
            c += samples_below(off[(uint64_t)q * S.tiles + x] - row0[q], snr[q], sdist[q]);
        return __reduce_add_sync(PJ_FULL, c) <= r;
    });
    // its samples before it, then the sample of rank r inside it
    {
        uint32_t c = 0;
        if (t > t0)  // nothing of the set lies before its first tile
            for (uint32_t q = threadIdx.x; q < p; q += PJ_NT)
                c += samples_below(off[(uint64_t)q * S.tiles + t] - row0[q], snr[q], sdist[q]);
        c = __reduce_add_sync(PJ_FULL, c);
        if (lane == 0 && c) atomicAdd(&s_before, c);
    }
    const uint64_t x0 = t * PJ_TILE + (uint64_t)threadIdx.x * PJ_IPT;
    uint32_t fl = 0, cnt = 0;
#pragma unroll
    for (int j = 0; j < PJ_IPT; ++j) {
        const uint64_t x = x0 + j;
        if (x < sp.begin || x >= sp.end) continue;
        const uint32_t q = S.bucket[x] - set * p, l = S.rank[x];
        if (samples_below(l + 1, snr[q], sdist[q]) != samples_below(l, snr[q], sdist[q])) {
            fl |= 1u << j;
            ++cnt;
        }
    }
    uint32_t pre = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(PJ_FULL, pre, o);
        if (lane >= (uint32_t)o) pre += y;
    }
    if (lane == 31) ws[w] = pre;
    __syncthreads();
    pre -= cnt;
    for (uint32_t v = 0; v < w; ++v) pre += ws[v];
    pre += s_before;
    if (r >= pre && r < pre + cnt) {
        for (int j = 0; j < PJ_IPT; ++j)
            if ((fl >> j) & 1u) {
                if (pre == r) s_g = x0 + j;
                ++pre;
            }
    }
    __syncthreads();
    const uint64_t g = s_g;
    if (g >= sp.end) {  // never taken when the counts agree
        if (threadIdx.x == 0) atomicExch(&S.flags[0], 1u);
        return;
    }
    // the splitter: string g cut to T bytes; [lo, hi) the positions whose
    // strings equal it
    const uint32_t id = S.ord[g];
    uint64_t off_s;
    uint32_t len;
    str_of(S.a, id, off_s, len);
    const uint32_t lg = g > sp.begin ? S.lcp[g] : 0u, lg1 = g + 1 < sp.end ? S.lcp[g + 1] : 0u;
    uint64_t T = S.cut ? 200 * (*S.cut / S.n + 5) : dp_depth_above(max(lg, lg1));
    T = min(T, (uint64_t)len);
    uint64_t lo = g, hi = T == len ? g + 1 : g;
    if (g > sp.begin && lg >= T && (T == len || S.cut)) {
        // the first position that shares T bytes with the splitter (searched
        // from g down: x counts back from g)
        lo = g - block_bisect(0, g - sp.begin + 1, ok, [&](uint64_t x) {
            uint64_t o;
            uint32_t l;
            str_of(S.a, S.ord[g - x], o, l);
            return l >= T && same_prefix(S.a.chars, o, off_s, (uint32_t)T, lane);
        });
        // a splitter shorter than its string equals only the strings of
        // exactly T bytes, which come first
        if (T < len) {
            uint64_t o;
            uint32_t l;
            str_of(S.a, S.ord[lo], o, l);
            hi = lo;
            if (l == T)
                hi = 1 + block_bisect(lo, g, ok, [&](uint64_t x) {
                    uint64_t ox;
                    uint32_t lx;
                    str_of(S.a, S.ord[x], ox, lx);
                    return lx == T;
                });
        }
    }
    if (T == len && g + 1 < sp.end && lg1 >= T) {
        hi = 1 + block_bisect(g, sp.end, ok, [&](uint64_t x) {
            uint64_t o;
            uint32_t l;
            str_of(S.a, S.ord[x], o, l);
            return l == T && same_prefix(S.a.chars, o, off_s, (uint32_t)T, lane);
        });
    }
    // every PE's ranks below lo and below hi
    const uint64_t tl = lo / PJ_TILE, th = hi / PJ_TILE;
    for (uint32_t q = threadIdx.x; q < p; q += PJ_NT) {
        cl[q] = off[(uint64_t)q * S.tiles + tl] - row0[q];
        cu[q] = hi >= sp.end ? (uint32_t)(pb[q + 1] - pb[q]) : off[(uint64_t)q * S.tiles + th] - row0[q];
    }
    __syncthreads();
    for (uint64_t x = max(tl * PJ_TILE, sp.begin) + threadIdx.x; x < lo; x += PJ_NT)
        atomicAdd(&cl[S.bucket[x] - set * p], 1u);
    if (hi < sp.end)
        for (uint64_t x = max(th * PJ_TILE, sp.begin) + threadIdx.x; x < hi; x += PJ_NT)
            atomicAdd(&cu[S.bucket[x] - set * p], 1u);
    __syncthreads();
    // the reference's search in each PE (binarySearch / binarySearchIndexed)
    uint32_t left_sum = 0;
    const uint64_t spl_index = pb[S.bucket[g] - set * p] + S.rank[g];
    for (uint32_t q = threadIdx.x; q < p; q += PJ_NT) {
        const uint64_t base = pb[q];
        uint32_t left = 0, right = (uint32_t)(pb[q + 1] - base);
        const uint32_t a = cl[q], b = cu[q];
        while (left != right) {
            const uint32_t m = left + (right - left) / 2;
            int res = m < a ? -1 : m >= b ? 1 : 0;
            // equal bytes compare by the global index, an int64 difference
            // narrowed to int (indexStringCompare, misc.hpp:335-345)
            if (res == 0 && S.indexed) res = (int)(int32_t)(uint32_t)(m + base - spl_index);
            if (res < 0) {
                left = m + 1;
            } else if (res == 0) {
                left = right = m;
            } else {
                right = m;
            }
        }
        bounds[(uint64_t)q * (p + 1) + k] = left;
        // inside the run: strings kept left of and right of the bound
        left_sum += left - a;
        if (b > left) atomicMin(&s_minr, q);
        if (left > a) atomicMax(&s_maxl, q + 1);
    }
    left_sum = __reduce_add_sync(PJ_FULL, left_sum);
    if (lane == 0) ws[w] = left_sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t c = 0;
        for (int v = 0; v < PJ_NW; ++v) c += ws[v];
        S.start[blockIdx.x] = (uint32_t)(lo + c);
        // a run lies in the order of its PEs: a string kept right before one
        // kept left (of a later PE) means that the receivers interleave
        if (s_maxl && s_minr < s_maxl - 1) atomicExch(&S.flags[1], 1u);
    }
}

// The merged LCP is 0 where a receiver's strings start.
__global__ void k_merged_starts(const uint32_t* start, uint32_t npe, uint32_t p, const SetSplit* sets,
                                const uint32_t* flags, uint32_t* merged) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= npe || flags[1]) return;
    const uint32_t s = start[r];
    if (s < sets[r / p].end) merged[s] = 0;
}

// Receiver of every position: the last r with bounds[PE][r] <= rank.
__global__ void __launch_bounds__(256) k_bucket_of(const uint32_t* bucket, const uint32_t* rank,
                                                   const uint32_t* bounds, uint32_t p, uint64_t n, uint32_t* out) {
    const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n) return;
    const uint32_t src = bucket[g], li = rank[g];
    const uint32_t* b = bounds + (uint64_t)src * (p + 1);
    uint32_t lo = 0;
    for (uint32_t step = 1u << (31 - __clz(p | 1u)); step; step >>= 1) {
        const uint32_t m = lo + step;
        if (m < p && b[m] <= li) lo = m;
    }
    out[g] = (src / p) * p + lo;
}

// -------------------------------------------------------------------- host --
void layout_project(Carve& c, ProjectLayout& L, uint64_t n, uint32_t nsets, uint32_t p) {
    const uint64_t npe = (uint64_t)nsets * p;
    L.tiles = (std::max<uint64_t>(n, 1) + PJ_TILE - 1) / PJ_TILE;
    const uint64_t cells = L.tiles * npe;
    L.hist = c.take<uint32_t>(cells);
    L.off = c.take<uint32_t>(cells);
    L.scan = c.take<unsigned char>(scan_scratch_bytes(cells));
    L.pb = c.take<uint64_t>(npe + 1);
    L.sets = c.take<SetSplit>(nsets);
    L.bounds = c.take<uint32_t>(npe * (p + 1) + 2);
    L.start = c.take<uint32_t>(npe);
    L.flags = c.sizing ? nullptr : L.bounds + npe * (p + 1);
}

uint64_t project_edge_words(uint64_t n, uint32_t npe) {
    const uint64_t tiles = (std::max<uint64_t>(n, 1) + PJ_TILE - 1) / PJ_TILE;
    return tiles * (2 * (uint64_t)npe + 1);
}

uint64_t project_pin_bytes(uint32_t nsets, uint32_t p) {
    const uint64_t npe = (uint64_t)nsets * p;
    return std::max<uint64_t>((npe + 1) * 8 + nsets * sizeof(SetSplit), (npe * (p + 1) + 2) * 4) + 64;
}

int project_setup(const ProjectLayout& L, uint32_t nsets, uint32_t p, const uint64_t* pb, uint32_t factor, void* pin,
                  cudaStream_t st) {
    const uint64_t npe = (uint64_t)nsets * p;
    uint64_t* hpb = (uint64_t*)pin;
    SetSplit* hs = (SetSplit*)(hpb + npe + 1);
    std::memcpy(hpb, pb, (npe + 1) * 8);
    for (uint32_t s = 0; s < nsets; ++s) {
        uint64_t total = 0;  // the set's samples (getNumberSplitter)
        for (uint32_t q = 0; q < p; ++q) {
            const uint64_t g = (uint64_t)s * p + q;
            total += std::min<uint64_t>((uint64_t)factor * (p - 1), pb[g + 1] - pb[g]);
        }
        hs[s].begin = pb[(uint64_t)s * p];
        hs[s].end = pb[(uint64_t)(s + 1) * p];
        hs[s].nspl = (uint32_t)std::min<uint64_t>(p - 1, total);
        hs[s].dist = (uint32_t)(total / (hs[s].nspl + 1));
    }
    DSSS_CUDA(cudaMemcpyAsync(L.pb, hpb, (npe + 1) * 8, cudaMemcpyHostToDevice, st));
    DSSS_CUDA(cudaMemcpyAsync(L.sets, hs, nsets * sizeof(SetSplit), cudaMemcpyHostToDevice, st));
    DSSS_CUDA(cudaMemsetAsync(L.flags, 0, 2 * sizeof(uint32_t), st));
    return DSSS_OK;
}

int project_local(const ProjectLayout& L, const ArenaDev& a, uint64_t n, uint32_t nsets, uint32_t p,
                  const uint32_t* ord, const uint32_t* lcp, const LenStats* stats, uint32_t* pe, uint32_t* bucket,
                  uint32_t* local_order, uint32_t* rank, uint32_t* dp, uint32_t* edges, unsigned long long* lcp_sum,
                  cudaStream_t st) {
    const uint32_t npe = nsets * p;
    const uint64_t cells = L.tiles * npe;
    if (cells >= (1ull << 32)) return fail(DSSS_ENOTSUP, "local orders: too many tiles x PEs");
    const size_t hsm = (npe + 1 + (size_t)npe * PJ_NW) * sizeof(uint32_t);
    DSSS_LAUNCH("k_pe_hist", st,
                k_pe_hist<<<(unsigned)L.tiles, PJ_NT, hsm, st>>>(ord, n, L.pb, npe, p, L.tiles, pe, bucket, L.hist));
    DSSS_TRY(exclusive_scan_u32(L.hist, L.off, cells, nullptr, L.scan, st));
    static std::atomic<uint64_t> c0{0}, c1{0};
    if (dp) {
        DSSS_TRY(set_smem_once(c0, k_local_scatter<true>, (int)pj_scatter_smem<true>(MAX_SPLIT_BUCKETS)));
        DSSS_LAUNCH("k_ms_scatter_pay", st,  // timed under the multisplits' label
                    k_local_scatter<true><<<(unsigned)L.tiles, PJ_NT, pj_scatter_smem<true>(npe), st>>>(
                        bucket, ord, lcp, a.len, stats, n, npe, L.tiles, L.off, L.pb, local_order, dp, LcpEdges{}, rank,
                        L.flags));
    } else {
        const LcpEdges E{edges, edges + cells, edges + 2 * cells, lcp_sum};
        DSSS_TRY(set_smem_once(c1, k_local_scatter<false>, (int)pj_scatter_smem<false>(MAX_SPLIT_BUCKETS)));
        DSSS_LAUNCH("k_ms_scatter_pay", st,  // timed under the multisplits' label
                    k_local_scatter<false><<<(unsigned)L.tiles, PJ_NT, pj_scatter_smem<false>(npe), st>>>(
                        bucket, ord, lcp, a.len, stats, n, npe, L.tiles, L.off, L.pb, local_order, dp, E, rank,
                        L.flags));
        DSSS_LAUNCH("k_local_lcp_edges", st, k_local_lcp_edges<<<npe, PJ_NT, 0, st>>>(E, L.tiles));
    }
    DSSS_CUDA(cudaGetLastError());
    return DSSS_OK;
}

int project_partition(const ProjectLayout& L, const ArenaDev& a, uint64_t n, uint32_t nsets, uint32_t p,
                      uint32_t factor, int indexed, const unsigned long long* cut, const uint32_t* ord,
                      const uint32_t* lcp, const uint32_t* bucket, const uint32_t* rank, uint32_t* merged,
                      cudaStream_t st) {
    SplitArgs S{a, n, L.tiles, p, factor, indexed, L.sets, L.pb, L.off, ord, lcp, bucket, rank, cut, L.bounds, L.start,
                L.flags};
    const uint32_t npe = nsets * p;
    const size_t sm = (size_t)p * (sizeof(double) + 4 * sizeof(uint32_t));
    DSSS_LAUNCH("k_splitters", st, k_splitters<<<npe, PJ_NT, sm, st>>>(S));
    if (merged)
        DSSS_LAUNCH("k_merged_starts", st,
                    k_merged_starts<<<grid_for(npe, 128), 128, 0, st>>>(L.start, npe, p, L.sets, L.flags, merged));
    DSSS_CUDA(cudaGetLastError());
    return DSSS_OK;
}

int project_read_async(const ProjectLayout& L, uint32_t nsets, uint32_t p, void* pin, cudaStream_t st) {
    const uint64_t npe = (uint64_t)nsets * p;
    DSSS_CUDA(cudaMemcpyAsync(pin, L.bounds, (npe * (p + 1) + 2) * 4, cudaMemcpyDeviceToHost, st));
    return DSSS_OK;
}

int project_read(uint32_t nsets, uint32_t p, const void* pin, uint64_t* intervals, uint64_t* recv_counts,
                 bool* ties) {
    const uint64_t npe = (uint64_t)nsets * p;
    const uint32_t* b = (const uint32_t*)pin;
    if (b[npe * (p + 1)]) return fail(DSSS_EDEVICE, "partition: internal consistency guard tripped");
    *ties = b[npe * (p + 1) + 1] != 0;
    for (uint64_t r = 0; r < npe; ++r) recv_counts[r] = 0;
    // compute_interval_binary (misc.hpp:376-395): differences of the bounds
    for (uint64_t g = 0; g < npe; ++g) {
        const uint32_t* row = b + g * (p + 1);
        uint64_t* recv = recv_counts + (g / p) * p;
        for (uint32_t r = 0; r < p; ++r) {
            const uint64_t v = (uint64_t)row[r + 1] - row[r];
            intervals[g * p + r] = v;
            recv[r] += v;
        }
    }
    return DSSS_OK;
}

int project_buckets(const ProjectLayout& L, uint64_t n, uint32_t p, const uint32_t* bucket, const uint32_t* rank,
                    uint32_t* dest_bucket, cudaStream_t st) {
    DSSS_LAUNCH("k_bucket_of", st,
                k_bucket_of<<<grid_for(n, 256), 256, 0, st>>>(bucket, rank, L.bounds, p, n, dest_bucket));
    return DSSS_OK;
}

}  // namespace dsss
