// C ABI entry points: the full prefix-doubling path and one entry per stage.
//
// The full path (dsss_pd_sort) is laid out for one GPU holding every PE:
//   1. one string sort of all n strings (K3, LCP as by-product);
//   2. stable multisplit by PE of the global order gives each PE's local sorted
//      order (a subsequence of a sorted sequence is sorted), i.e. exactly what
//      radixsort_CI3 produces per PE (prefix_doubling.hpp:228), each string with
//      its distinguishing prefix, which the order's LCPs decide (K1);
//   3. splitters and bounds (K5) from positions and ranks in those orders;
//   4. each receiving PE's merged sequence — what
//      AllToAllStringImplPrefixDoubling + choose_merge deliver
//      (prefix_doubling.hpp:254-281) — is the global order itself, its PEs and
//      ranks the permutation (:282-290), unless equal strings fall on different
//      sides of a splitter: then the stable multisplit of it by receiver.
#include <algorithm>
#include <cstring>
#include <random>
#include <vector>

#include "dp.cuh"
#include "exchange.cuh"
#include "internal.cuh"
#include "merge.cuh"
#include "partition.cuh"
#include "pd.cuh"
#include "project.cuh"
#include "strsort.cuh"
#include "util.cuh"

namespace dsss {

static int check_parts(uint32_t p, const uint64_t* pb, uint64_t n) {
    if (p == 0) return fail(DSSS_EINVAL, "p must be >= 1");
    if (!pb) return fail(DSSS_EINVAL, "part_begin is NULL");
    if (pb[0] != 0 || pb[p] != n) return fail(DSSS_EINVAL, "part_begin must start at 0 and end at n");
    for (uint32_t q = 0; q < p; ++q)
        if (pb[q + 1] < pb[q]) return fail(DSSS_EINVAL, "part_begin must be non-decreasing");
    return DSSS_OK;
}

static ArenaDev view(const dsss_arena* a) { return ArenaDev{a->chars, a->offsets, a->lengths, a->n}; }

static uint32_t factor_of(const dsss_opts* o) { return (o && o->sampling_factor) ? o->sampling_factor : 2; }
static uint32_t sampler_of(const dsss_opts* o) { return o ? o->sampler : DSSS_SAMPLER_NUM_STRINGS; }
static uint32_t smallmax_of(const dsss_opts* o) { return o ? o->small_sort_max : 0; }

__global__ void k_merged_lcp(const uint32_t* out2g, const uint32_t* lcpg, const uint64_t* recv_begin, uint32_t p,
                             uint64_t n, uint32_t* merged) {
    const uint64_t o = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= n) return;
    uint32_t lo = 0, hi = p;  // is o the first string of some PE's merged run?
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (recv_begin[mid] <= o) lo = mid;
        else hi = mid;
    }
    bool first = false;
    for (uint32_t r = lo; r < p && recv_begin[r] <= o; ++r)
        if (recv_begin[r] == o) { first = true; break; }
    if (first) { merged[o] = 0; return; }
    const uint32_t g = out2g[o], gp = out2g[o - 1];
    uint32_t l = 0xFFFFFFFFu;
    for (uint32_t x = gp + 1; x <= g; ++x) l = min(l, lcpg[x]);  // LCP over the skipped run
    merged[o] = l;
}

__global__ void k_zero_starts(uint32_t* a, const uint64_t* pb, uint32_t p) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < p && pb[q] < pb[q + 1]) a[pb[q]] = 0;
}

struct PdLayout {
    ulonglong2* handles;
    LenStats* stats;
    uint32_t *ord, *lcp, *bucket, *err, *nlong;
    uint64_t* recv_begin;
    void* ms;
    SortLayout sort;
    ProjectLayout proj;
    // after the sort, its buffers serve the multisplit of tied calls
    uint32_t* tie[5];
};

// n strings in nsets sets of p PEs each.
static void layout_pd(Carve& c, PdLayout& L, uint64_t n, uint32_t nsets, uint32_t p, uint32_t small_max) {
    uint64_t N = n ? n : 1;
    const uint64_t npe = (uint64_t)nsets * p;
    L.handles = c.take<ulonglong2>(N);
    L.stats = c.take<LenStats>(1);
    L.ord = c.take<uint32_t>(N);
    L.lcp = c.take<uint32_t>(N);
    L.bucket = c.take<uint32_t>(N);
    L.err = c.take<uint32_t>(1);
    L.nlong = c.take<uint32_t>(1);
    L.recv_begin = c.take<uint64_t>(npe + 1);
    L.ms = c.take<unsigned char>(multisplit_scratch_bytes(N, (uint32_t)npe));
    layout_project(c, L.proj, N, nsets, p);
    layout_sort(c, L.sort, N, nsets, small_max);
    L.tie[0] = L.sort.ord[0];
    L.tie[1] = L.sort.ord[1];
    L.tie[2] = (uint32_t*)L.sort.key[0];
    L.tie[3] = c.sizing ? nullptr : (uint32_t*)L.sort.key[0] + N;
    L.tie[4] = (uint32_t*)L.sort.key[1];
}

// Start of every receiver's strings, on the host and (for k_merged_lcp) on
// the device.
static int upload_recv_begin(const PdLayout& L, uint32_t npe, const uint64_t* recv_counts, void* pin,
                             cudaStream_t st) {
    uint64_t* h = (uint64_t*)pin;
    h[0] = 0;
    for (uint32_t r = 0; r < npe; ++r) h[r + 1] = h[r] + recv_counts[r];
    DSSS_CUDA(cudaMemcpyAsync(L.recv_begin, h, (npe + 1) * 8, cudaMemcpyHostToDevice, st));
    return DSSS_OK;
}

uint64_t pd_scratch_bytes(uint64_t n, uint32_t nsets, uint32_t p, const dsss_opts* opts) {
    Carve sz(nullptr);
    PdLayout L;
    layout_pd(sz, L, n, nsets, p, smallmax_of(opts));
    return sz.used;
}

// The fused path over nsets independent string sets of p PEs each (PE q of
// set s = part_begin[s*p + q] .. part_begin[s*p + q + 1]); every set's result
// is the one a call on that set alone gives.  Per-string outputs keep the
// arena's positions (set s's merged sequences fill the positions of its
// strings), intervals and recv_counts are per set, one after the other.
int pd_sort_dev(Ctx* ctx, const dsss_arena* in, uint32_t nsets, uint32_t p, const uint64_t* pb,
                const dsss_opts* opts, dsss_pd_result* out, cudaStream_t st) {
    DSSS_TRY(check_arena(in));
    if (nsets == 0) return fail(DSSS_EINVAL, "nsets must be >= 1");
    if (p == 0) return fail(DSSS_EINVAL, "p must be >= 1");
    if ((uint64_t)nsets * p > MAX_SPLIT_BUCKETS)
        return fail(DSSS_ENOTSUP, "nsets * p > %u PEs per GPU is not supported", MAX_SPLIT_BUCKETS);
    const uint32_t npe = nsets * p;
    DSSS_TRY(check_parts(npe, pb, in->n));
    if (!out || !out->local_order || !out->recv_counts) return fail(DSSS_EINVAL, "result arrays missing");
    if (p > 1 && (!out->dp || !out->intervals || !out->perm_index || !out->perm_pe))
        return fail(DSSS_EINVAL, "result arrays missing");
    const uint64_t n = in->n;
    const uint32_t factor = factor_of(opts), smax = smallmax_of(opts);
    const bool want_local_lcp = opts && (opts->flags & DSSS_FLAG_LOCAL_LCP) && out->local_lcp;
    Carve sz(nullptr);
    PdLayout L;
    layout_pd(sz, L, n, nsets, p, smax);
    DSSS_TRY(ensure_ws(ctx, sz.used));
    // the sort's counters, then the projection's staging area
    const uint64_t pin_sort = 256;
    DSSS_TRY(ensure_pin(ctx, std::max<uint64_t>(4096, pin_sort + project_pin_bytes(nsets, p))));
    Carve c(ctx->ws);
    layout_pd(c, L, n, nsets, p, smax);
    uint32_t* pin = (uint32_t*)ctx->pin;
    void* pinp = (char*)ctx->pin + pin_sort;
    ArenaDev a = view(in);
    if (n == 0) {
        for (uint32_t r = 0; r < npe; ++r) out->recv_counts[r] = 0;
        if (p > 1)
            for (uint64_t k = 0; k < (uint64_t)npe * p; ++k) out->intervals[k] = 0;
        return DSSS_OK;
    }
    std::vector<uint64_t> set_begin(nsets + 1);
    for (uint32_t s = 0; s <= nsets; ++s) set_begin[s] = pb[(uint64_t)s * p];
    if (p > 1) DSSS_TRY(length_stats(a, L.stats, st));
    // 1. one sort per set, all sets in one segmented sort; the global LCPs are
    // the merged ones up to the receivers' starts
    uint32_t* ord = p == 1 ? out->local_order : L.ord;
    uint32_t* lcp = p > 1 && out->merged_lcp ? out->merged_lcp : p == 1 && want_local_lcp ? out->local_lcp : L.lcp;
    {
        StageTimer t("stage:sort", st);
        DSSS_TRY(sort_strings(L.sort, a, n, nsets, set_begin.data(), nullptr, ord, lcp, pin, st, L.handles));
    }
    if (p == 1) {  // prefix_doubling.hpp:236: one PE sorts locally and returns no permutation
        for (uint32_t r = 0; r < npe; ++r) out->recv_counts[r] = 0;
        return DSSS_OK;
    }
    // 2. the PEs' local orders with their distinguishing prefixes; position
    // g's PE and its rank there are the (index, PE) permutation
    uint32_t* pe = out->perm_pe;
    uint32_t* bucket = nsets > 1 ? L.bucket : pe;
    {
        StageTimer t("stage:local", st);
        DSSS_TRY(project_setup(L.proj, nsets, p, pb, factor, pinp, st));
        DSSS_TRY(project_local(L.proj, a, n, nsets, p, ord, lcp, L.stats, pe, bucket, out->local_order,
                               out->perm_index, out->dp, nullptr, nullptr, st));
    }
    // 3. splitters and every PE's bounds; receiving PE (s, r) is bucket s*p + r
    {
        StageTimer t("stage:partition", st);
        DSSS_TRY(project_partition(L.proj, a, n, nsets, p, factor,
                                   sampler_of(opts) == DSSS_SAMPLER_INDEXED_NUM_STRINGS, nullptr, ord, lcp, bucket,
                                   out->perm_index, out->merged_lcp, st));
        DSSS_TRY(project_read_async(L.proj, nsets, p, pinp, st));
    }
    if (want_local_lcp) {
        DSSS_TRY(adjacent_lcp(a, out->local_order, n, out->local_lcp, L.tie[0], L.nlong, st));
        DSSS_LAUNCH("k_zero_starts", st,
                    k_zero_starts<<<grid_for(npe, 128), 128, 0, st>>>(out->local_lcp, L.proj.pb, npe));
    }
    DSSS_CUDA(cudaGetLastError());
    DSSS_CUDA(cudaStreamSynchronize(st));
    bool ties = false;
    DSSS_TRY(project_read(nsets, p, pinp, out->intervals, out->recv_counts, &ties));
    if (!ties) return DSSS_OK;
    // 4. equal strings on different sides of a splitter: the merged sequences
    // are the stable multisplit of the global order by receiver
    StageTimer t_merge("stage:merge", st);
    DSSS_CUDA(cudaMemsetAsync(L.err, 0, sizeof(uint32_t), st));
    DSSS_TRY(upload_recv_begin(L, npe, out->recv_counts, pinp, st));
    DSSS_TRY(project_buckets(L.proj, n, p, bucket, out->perm_index, L.tie[2], st));
    DSSS_CUDA(cudaMemcpyAsync(L.tie[0], out->perm_index, n * 4, cudaMemcpyDeviceToDevice, st));
    DSSS_CUDA(cudaMemcpyAsync(L.tie[1], pe, n * 4, cudaMemcpyDeviceToDevice, st));
    {
        // (index in sender's local order, sender PE, global position)
        const uint32_t* in3[3] = {L.tie[0], L.tie[1], nullptr};
        uint32_t* outs[3] = {out->perm_index, out->perm_pe, L.tie[3]};
        DSSS_TRY(multisplit_payload(L.tie[2], n, npe, 3, in3, outs, nullptr, L.err, L.ms, st));
    }
    if (out->merged_lcp) {
        DSSS_CUDA(cudaMemcpyAsync(L.lcp, out->merged_lcp, n * 4, cudaMemcpyDeviceToDevice, st));
        DSSS_LAUNCH("k_merged_lcp", st,
                    k_merged_lcp<<<grid_for(n, 256), 256, 0, st>>>(L.tie[3], L.lcp, L.recv_begin, npe, n,
                                                                  out->merged_lcp));
    }
    DSSS_CUDA(cudaGetLastError());
    DSSS_CUDA(cudaMemcpyAsync(pin, L.err, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    DSSS_CUDA(cudaStreamSynchronize(st));
    if (pin[0]) return fail(DSSS_EDEVICE, "pd sort: internal consistency guard tripped");
    return DSSS_OK;
}

// ------------------------------------------------------- merge-sort path ----
// DistributedMergeSort::sort on one GPU holding every PE: the global sort, the
// local orders and their LCP arrays, getAvgLcp, the partition with samples cut
// to 200 (avg + 5) bytes, then the receiving PEs' sequences (the global order,
// or its multisplit by receiver when ties cross a splitter) and their strings
// copied out whole.

// Input index, source offset and length (+ 1 for the scan) of every output
// string (the string at global position map[o], or o): the copy then reads its
// string's place sequentially instead of gathering it again.
__global__ void k_ms_source(const uint32_t* ord, const uint32_t* map, ArenaDev a, uint64_t n, uint32_t* source,
                            uint32_t* lengths, uint32_t* len1, uint64_t* src_off) {
    const uint64_t o = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= n) return;
    const uint32_t id = ord[map ? map[o] : (uint32_t)o];
    uint64_t off;
    uint32_t len;
    str_of(a, id, off, len);
    source[o] = id;
    lengths[o] = len;
    len1[o] = len + 1;
    src_off[o] = off;
}

// Whole output strings and their NULs, MS_COPY_LANES lanes per string
// (copy_words16: aligned 16-byte stores, 3.5% faster on B200 than
// copy_words' 8-byte ones, which the knob copy_word = 8 selects; 8 lanes
// measured faster than 4 or 32).
constexpr uint32_t MS_COPY_LANES = 8;
template <uint32_t W>
__global__ void k_ms_copy(const uint8_t* chars, const uint64_t* src_off, const uint32_t* lengths,
                          const uint64_t* out_off, uint64_t n, uint8_t* out) {
    const uint64_t o = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / MS_COPY_LANES;
    const uint32_t lane = threadIdx.x % MS_COPY_LANES;
    if (o >= n) return;
    const uint32_t len = lengths[o];
    uint8_t* dst = out + out_off[o];
    if (W == 16) copy_words16<MS_COPY_LANES>(dst, chars + src_off[o], len, lane);
    else copy_words<MS_COPY_LANES>(dst, chars + src_off[o], len, lane);
    if (lane == 0) dst[len] = 0;
}

static int launch_ms_copy(const uint8_t* chars, const uint64_t* src_off, const uint32_t* lengths,
                          const uint64_t* out_off, uint64_t n, uint8_t* out, cudaStream_t st) {
    const unsigned grid = grid_for(n * MS_COPY_LANES, 256);
    if (tune(TUNE_COPY_WORD) == 16)
        DSSS_LAUNCH("k_ms_copy", st, k_ms_copy<16><<<grid, 256, 0, st>>>(chars, src_off, lengths, out_off, n, out));
    else
        DSSS_LAUNCH("k_ms_copy", st, k_ms_copy<8><<<grid, 256, 0, st>>>(chars, src_off, lengths, out_off, n, out));
    return DSSS_OK;
}

static int ms_sort_dev(Ctx* ctx, const dsss_arena* in, uint32_t p, const uint64_t* pb, const dsss_opts* opts,
                       dsss_ms_result* out, cudaStream_t st) {
    DSSS_TRY(check_arena(in));
    if (p == 0) return fail(DSSS_EINVAL, "p must be >= 1");
    if (p > MAX_SPLIT_BUCKETS) return fail(DSSS_ENOTSUP, "p > %u PEs per GPU is not supported", MAX_SPLIT_BUCKETS);
    DSSS_TRY(check_parts(p, pb, in->n));
    if (!out || !out->local_order || !out->recv_counts || !out->intervals || !out->offsets || !out->lengths ||
        !out->lcp || (in->n && !out->chars))
        return fail(DSSS_EINVAL, "result arrays missing");
    if (opts && opts->sampler != DSSS_SAMPLER_NUM_STRINGS)
        return fail(DSSS_ENOTSUP, "the merge-sort path samples with SampleSplittersNumStringsPolicy only");
    const uint64_t n = in->n;
    const uint32_t factor = 2, smax = smallmax_of(opts);  // computePartition(..., 2): misc.hpp call in :238
    const uint64_t N = n ? n : 1;
    PdLayout L;
    uint32_t *src_tmp, *len1, *pe, *rank, *edges;
    uint64_t* srcoff;
    unsigned long long* total;
    void* scan;
    auto plan = [&](Carve& c) {
        layout_pd(c, L, n, 1, p, smax);
        src_tmp = c.take<uint32_t>(N);
        len1 = c.take<uint32_t>(N);
        pe = c.take<uint32_t>(N);
        rank = c.take<uint32_t>(N);
        edges = c.take<uint32_t>(project_edge_words(N, p));
        srcoff = c.take<uint64_t>(N);
        total = c.take<unsigned long long>(2);
        scan = c.take<unsigned char>(scan_scratch_bytes(N));
    };
    Carve sz(nullptr);
    plan(sz);
    DSSS_TRY(ensure_ws(ctx, sz.used));
    const uint64_t pin_sort = 256;
    DSSS_TRY(ensure_pin(ctx, std::max<uint64_t>(4096, pin_sort + project_pin_bytes(1, p))));
    Carve c(ctx->ws);
    plan(c);
    uint32_t* source = out->source ? out->source : src_tmp;
    out->avg_lcp = 0;
    if (n == 0) {
        for (uint32_t r = 0; r < p; ++r) out->recv_counts[r] = 0;
        for (uint64_t k = 0; k < (uint64_t)p * p; ++k) out->intervals[k] = 0;
        return DSSS_OK;
    }
    ArenaDev a = view(in);
    DSSS_TRY(length_stats(a, L.stats, st));
    uint32_t* pin = (uint32_t*)ctx->pin;
    void* pinp = (char*)ctx->pin + pin_sort;
    LenStats* hstats = (LenStats*)((char*)ctx->pin + 128);
    DSSS_CUDA(cudaMemsetAsync(L.err, 0, sizeof(uint32_t), st));
    DSSS_CUDA(cudaMemsetAsync(total, 0, 2 * sizeof(unsigned long long), st));
    DSSS_CUDA(cudaMemcpyAsync(hstats, L.stats, sizeof(LenStats), cudaMemcpyDeviceToHost, st));
    const uint64_t set_begin[2] = {0, n};
    {
        StageTimer t("stage:sort", st);
        DSSS_TRY(sort_strings(L.sort, a, n, 1, set_begin, nullptr, L.ord, out->lcp, pin, st, L.handles));
    }
    if (!a.h) {  // every string is gathered below
        DSSS_TRY(make_handles(a, L.handles, st));
        a.h = L.handles;
    }
    const uint64_t bytes = hstats->sum + n;  // the sort has synchronised on st
    // local orders per PE and the sum of their LCPs
    StageTimer t_local("stage:local", st);
    DSSS_TRY(project_setup(L.proj, 1, p, pb, factor, pinp, st));
    DSSS_TRY(project_local(L.proj, a, n, 1, p, L.ord, out->lcp, nullptr, pe, pe, out->local_order, rank, nullptr, edges,
                           total, st));
    unsigned long long* hsum = (unsigned long long*)((char*)ctx->pin + 192);
    DSSS_CUDA(cudaMemcpyAsync(hsum, total, 8, cudaMemcpyDeviceToHost, st));
    t_local.end();
    const uint32_t* map = nullptr;
    if (p == 1) {  // lcp_aware_number_string_splitting.hpp:230-232: the local sort is the result
        DSSS_CUDA(cudaStreamSynchronize(st));
        out->intervals[0] = n;
        out->recv_counts[0] = n;
    } else {
        {
            StageTimer t("stage:partition", st);
            DSSS_TRY(project_partition(L.proj, a, n, 1, p, factor, 0, total, L.ord, out->lcp, pe, rank, out->lcp, st));
            DSSS_TRY(project_read_async(L.proj, 1, p, pinp, st));
            DSSS_CUDA(cudaStreamSynchronize(st));
        }
        StageTimer t_merge("stage:merge", st);
        bool ties = false;
        DSSS_TRY(project_read(1, p, pinp, out->intervals, out->recv_counts, &ties));
        if (ties) {
            DSSS_TRY(upload_recv_begin(L, p, out->recv_counts, pinp, st));
            DSSS_TRY(project_buckets(L.proj, n, p, pe, rank, L.tie[2], st));
            const uint32_t* ins[1] = {nullptr};
            uint32_t* outs[1] = {L.tie[3]};
            DSSS_TRY(multisplit_payload(L.tie[2], n, p, 1, ins, outs, nullptr, L.err, L.ms, st));
            DSSS_CUDA(cudaMemcpyAsync(L.lcp, out->lcp, n * 4, cudaMemcpyDeviceToDevice, st));
            DSSS_LAUNCH("k_merged_lcp", st,
                        k_merged_lcp<<<grid_for(n, 256), 256, 0, st>>>(L.tie[3], L.lcp, L.recv_begin, p, n, out->lcp));
            map = L.tie[3];
        }
    }
    out->avg_lcp = *hsum / n;  // getAvgLcp (misc.hpp:68-87)
    if (bytes > out->chars_capacity)
        return fail(DSSS_EINVAL, "chars_capacity %llu is below the %llu output bytes",
                    (unsigned long long)out->chars_capacity, (unsigned long long)bytes);
    // output layout and the strings themselves
    {
        StageTimer t("stage:copy", st);
        DSSS_LAUNCH("k_ms_source", st,
                    k_ms_source<<<grid_for(n, 256), 256, 0, st>>>(L.ord, map, a, n, source, out->lengths, len1,
                                                                 srcoff));
        DSSS_TRY(exclusive_scan_u32_to_u64(len1, out->offsets, n, (uint64_t*)(total + 1), scan, st));
        DSSS_TRY(launch_ms_copy(a.chars, srcoff, out->lengths, out->offsets, n, out->chars, st));
    }
    DSSS_CUDA(cudaMemcpyAsync(pin, L.err, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    DSSS_CUDA(cudaMemcpyAsync(pin + 1, L.proj.flags, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    DSSS_CUDA(cudaStreamSynchronize(st));
    if (pin[0] || pin[1]) return fail(DSSS_EDEVICE, "ms sort: internal consistency guard tripped");
    return DSSS_OK;
}

// ----------------------------------------------------------- hQuicksort ----
// RQuick::sort (sorter/RQuick/RQuick.hpp:834-1104, sortRec :415-627) as the
// hQuicksort executable runs it, on one GPU holding every PE.  Strings never
// move between levels: after one global sort, PE q's sorted data at a level is
// the ascending list of global positions it owns (equal strings are
// byte-identical, so which of them a PE holds is immaterial), the exchange
// relabels owners, and the strings are written once at the end: the PEs'
// sorted data in rank order is the global order.  The lists are never built:
// per-tile owner counts, scanned PE-major, give every list's start and the
// rank of every tile in it, so the pivot and each PE's split are a binary
// search over tiles plus a scan of one tile.

constexpr uint32_t HQ_NT = 256, HQ_IPT = 16, HQ_TILE = HQ_NT * HQ_IPT;
constexpr uint32_t HQ_NONE = 0xFFFFFFFFu;

// The pivot's run: lists are searched for the first position of the run of
// strings equal to the pivot and the first position past it.
// glen: lengths in the global order.
__global__ void k_hq_run_ends(const uint32_t* glen, const uint32_t* lcp, uint64_t n, uint32_t* tail) {
    const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n) return;
    tail[g] = g + 1 < n ? !(glen[g] == glen[g + 1] && lcp[g + 1] == glen[g]) : 1u;
}

// Adds owner o of this lane to the shared histogram, one atomic per owner
// and warp (owners come in long runs).
__device__ __forceinline__ void hq_count(uint32_t* h, uint32_t o, uint32_t pw) {
    const uint32_t peers = __match_any_sync(0xffffffffu, o);
    if (o < pw && (threadIdx.x & 31) == (uint32_t)__ffs(peers) - 1) atomicAdd(&h[o], __popc(peers));
}

// The first level's owners: the PE of the string at each global position,
// PEs past the largest power of two pw folded onto PE q - pw (RQuick.hpp:878-959),
// and the owner counts of every tile, PE-major: tc[q * tiles + t].
__global__ void __launch_bounds__(HQ_NT) k_hq_owner0(const uint32_t* ord, uint64_t n, const uint64_t* pb, uint32_t p,
                                                     uint32_t pw, uint64_t tiles, uint16_t* owner, uint32_t* tc) {
    extern __shared__ uint32_t h[];
    for (uint32_t q = threadIdx.x; q < pw; q += HQ_NT) h[q] = 0;
    __syncthreads();
    const uint64_t t0 = (uint64_t)blockIdx.x * HQ_TILE;
#pragma unroll 4
    for (uint32_t j = 0; j < HQ_IPT; ++j) {
        const uint64_t g = t0 + j * HQ_NT + threadIdx.x;
        uint32_t q = HQ_NONE;
        if (g < n) {
            const uint32_t s = ord[g];
            uint32_t lo = 0, hi = p;  // last q with pb[q] <= s
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (__ldg(&pb[mid]) <= s) lo = mid;
                else hi = mid;
            }
            q = lo >= pw ? lo - pw : lo;
            owner[g] = (uint16_t)q;
        }
        hq_count(h, q, pw);
    }
    __syncthreads();
    for (uint32_t q = threadIdx.x; q < pw; q += HQ_NT) tc[(uint64_t)q * tiles + blockIdx.x] = h[q];
}

// The exchange (RQuick.hpp:496-586): the left half sends its strings from its
// split on, the right half those before it; dest[q] is q's partner, bit 31 set
// for the left half, cut[q] the position of q's split (HQ_NONE: past its
// end).  The new owners' tile counts are those of the next level.
__global__ void __launch_bounds__(HQ_NT) k_hq_move(uint16_t* owner, uint64_t n, uint32_t pw, uint64_t tiles,
                                                   const uint32_t* cut, const uint32_t* dest, uint32_t* tc) {
    extern __shared__ uint32_t h[];
    for (uint32_t q = threadIdx.x; q < pw; q += HQ_NT) h[q] = 0;
    __syncthreads();
    const uint64_t t0 = (uint64_t)blockIdx.x * HQ_TILE;
#pragma unroll 4
    for (uint32_t j = 0; j < HQ_IPT; ++j) {
        const uint64_t g = t0 + j * HQ_NT + threadIdx.x;
        uint32_t o = HQ_NONE;
        if (g < n) {
            o = owner[g];
            if (o < pw) {
                const uint32_t c = cut[o], d = dest[o];
                if ((d >> 31) ? (c != HQ_NONE && g >= c) : (c == HQ_NONE || g < c)) {
                    o = d & 0x7FFFFFFFu;
                    owner[g] = (uint16_t)o;
                }
            }
        }
        hq_count(h, o, pw);
    }
    __syncthreads();
    for (uint32_t q = threadIdx.x; q < pw; q += HQ_NT) tc[(uint64_t)q * tiles + blockIdx.x] = h[q];
}

// Strings per PE from the scanned tile counts (off[pw * tiles] is not held:
// the last PE ends at n).
__global__ void k_hq_counts(const uint32_t* off, uint64_t tiles, uint32_t pw, uint64_t n, uint32_t* cnt) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= pw) return;
    const uint64_t e = q + 1 < pw ? off[(uint64_t)(q + 1) * tiles] : n;
    cnt[q] = (uint32_t)(e - off[(uint64_t)q * tiles]);
}

// One level's parameters of PE q, drawn on the host from its random bits.
struct HqPe {
    uint32_t cnt;   // strings q holds
    uint32_t opt;   // locateSplitter's middle: cnt / 2, + 1 by a bit when cnt is odd
    uint32_t piv;   // first PE of a subcube: index of the pivot in its list, HQ_NONE: the empty pivot
    uint32_t cube;  // subcube size at this level
};

__device__ __forceinline__ uint64_t first_not_below(const uint32_t* v, uint64_t m, uint64_t x) {
    uint64_t lo = 0, hi = m;
    while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if (v[mid] < x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Block sum and exclusive block scan (HQ_NT threads; sh: HQ_NT / 32 + 1 words).
__device__ __forceinline__ uint32_t hq_block_scan(uint32_t v, uint32_t* sh, uint32_t& total) {
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    uint32_t pre = x - v, tot = 0;
    for (uint32_t k = 0; k < HQ_NT / 32; ++k) {
        if (k < w) pre += sh[k];
        tot += sh[k];
    }
    __syncthreads();
    total = tot;
    return pre;
}

// Strings of PE q at positions below x (its list's lower bound of x).
__device__ uint32_t hq_rank(const uint16_t* owner, const uint32_t* off, uint64_t tiles, uint64_t n, uint32_t q,
                            uint32_t cnt, uint64_t x, uint32_t* sh) {
    if (x >= n) return cnt;
    const uint64_t t = x / HQ_TILE, t0 = t * HQ_TILE;
    uint32_t c = 0;
    for (uint32_t j = 0; j < HQ_IPT; ++j) {
        const uint64_t g = t0 + j * HQ_NT + threadIdx.x;
        c += g < x && owner[g] == q;
    }
    uint32_t total;
    hq_block_scan(c, sh, total);
    return off[(uint64_t)q * tiles + t] - off[(uint64_t)q * tiles] + total;
}

// Position of the k-th string (from 0, k < its count) of PE q's list.
__device__ uint32_t hq_select(const uint16_t* owner, const uint32_t* off, uint64_t tiles, uint64_t n, uint32_t q,
                              uint32_t k, uint32_t* sh) {
    const uint32_t* row = off + (uint64_t)q * tiles;
    const uint32_t b = row[0];
    uint64_t lo = 0, hi = tiles;  // the last tile whose list rank is <= k
    while (hi - lo > 1) {
        const uint64_t mid = (lo + hi) >> 1;
        if (row[mid] - b <= k) lo = mid;
        else hi = mid;
    }
    const uint32_t r = k - (row[lo] - b);
    const uint64_t g0 = lo * HQ_TILE + (uint64_t)threadIdx.x * HQ_IPT;
    uint32_t c = 0;
    for (uint32_t j = 0; j < HQ_IPT; ++j) c += g0 + j < n && owner[g0 + j] == q;
    uint32_t total;
    uint32_t pre = hq_block_scan(c, sh, total);
    if (threadIdx.x == 0) sh[HQ_NT / 32] = HQ_NONE;
    __syncthreads();
    if (r >= pre && r < pre + c)
        for (uint32_t j = 0; j < HQ_IPT; ++j)
            if (g0 + j < n && owner[g0 + j] == q) {
                if (pre == r) sh[HQ_NT / 32] = (uint32_t)(g0 + j);
                ++pre;
            }
    __syncthreads();
    const uint32_t v = sh[HQ_NT / 32];
    __syncthreads();
    return v;
}

// locateSplitter (robust, RQuick.hpp:363-385) of PE q = blockIdx.x: the
// subcube's pivot, its run of equal strings, q's lower and upper bound of it,
// the split, and the position where q's split falls.
__global__ void __launch_bounds__(HQ_NT) k_hq_split(const HqPe* prm, const uint16_t* owner, const uint32_t* off,
                                                    uint64_t tiles, const uint32_t* runx, const uint32_t* ord,
                                                    ArenaDev a, uint64_t n, uint32_t pw, uint32_t* cut,
                                                    uint32_t* dest, uint32_t* err) {
    __shared__ uint32_t sh[HQ_NT / 32 + 1];
    const uint32_t q = blockIdx.x;
    const HqPe m = prm[q];
    const uint32_t P = m.cube, b = q & ~(P - 1), half = P >> 1;
    const HqPe r = prm[b];
    uint64_t lo = 0, hi = 0;
    if (r.piv == HQ_NONE) {  // the empty string: every empty string equals it
        uint64_t o;
        uint32_t l;
        str_of(a, ord[0], o, l);
        hi = l == 0 ? first_not_below(runx, n, 1) : 0;
    } else {
        if (r.piv >= r.cnt) {
            if (threadIdx.x == 0) atomicExch(err, 1u);
            return;
        }
        const uint32_t pg = hq_select(owner, off, tiles, n, b, r.piv, sh);
        if (pg >= n) {
            if (threadIdx.x == 0) atomicExch(err, 1u);
            return;
        }
        const uint32_t k = runx[pg];
        lo = first_not_below(runx, n, k);
        hi = first_not_below(runx, n, (uint64_t)k + 1);
    }
    const uint32_t lb = hq_rank(owner, off, tiles, n, q, m.cnt, lo, sh);
    const uint32_t ub = hq_rank(owner, off, tiles, n, q, m.cnt, hi, sh);
    const uint32_t sep = lb < m.opt ? min(m.opt, ub) : lb;
    const uint32_t c = sep < m.cnt ? hq_select(owner, off, tiles, n, q, sep, sh) : HQ_NONE;
    if (threadIdx.x == 0) {
        if (sep < m.cnt && c >= n) atomicExch(err, 1u);
        cut[q] = c;
        dest[q] = (b + (q - b + half) % P) | (q - b < half ? 0x80000000u : 0u);
    }
}

// RandomBitStore (sorter/RQuick/RandomBitStore.hpp:27-52) on PE q's
// std::mt19937_64.
struct HqBits {
    std::mt19937_64 gen;
    uint64_t bits = 0;
    int pos = 64;
    uint32_t next() {
        if (pos == 64) {
            bits = gen();
            pos = 0;
        }
        const uint32_t r = (uint32_t)(bits & 1);
        bits >>= 1;
        ++pos;
        return r;
    }
};

static int hq_sort_dev(Ctx* ctx, const dsss_arena* in, uint32_t p, const uint64_t* pb, uint64_t seed,
                       dsss_hq_result* out, cudaStream_t st) {
    DSSS_TRY(check_arena(in));
    if (p == 0) return fail(DSSS_EINVAL, "p must be >= 1");
    if (p > MAX_SPLIT_BUCKETS) return fail(DSSS_ENOTSUP, "p > %u PEs per GPU is not supported", MAX_SPLIT_BUCKETS);
    DSSS_TRY(check_parts(p, pb, in->n));
    if (!out || !out->counts || !out->offsets || !out->lengths || (in->n && !out->chars))
        return fail(DSSS_EINVAL, "result arrays missing");
    const uint64_t n = in->n;
    uint32_t pw = 1, levels = 0;
    while (pw * 2 <= p) pw *= 2, ++levels;
    out->levels = levels;
    for (uint32_t q = 0; q < p; ++q) out->counts[q] = 0;
    if (n == 0) return DSSS_OK;
    const uint64_t N = n, tiles = (n + HQ_TILE - 1) / HQ_TILE, cells = tiles * pw;
    if (cells >= (1ull << 32)) return fail(DSSS_ENOTSUP, "hq sort: too many tiles x PEs");
    const uint32_t smax = 0;
    auto plan = [&](Carve& c, ulonglong2*& handles, uint32_t*& ord, uint32_t*& lcp, uint16_t*& owner, uint32_t*& tmp,
                    uint32_t*& runx, uint32_t*& srcb, uint32_t*& tc, uint32_t*& off, uint32_t*& cnt, HqPe*& prm,
                    uint32_t*& cut, uint32_t*& dest, uint32_t*& err, uint64_t*& pbd, uint64_t*& total, void*& scan,
                    uint64_t*& srcoff, LenStats*& stats, SortLayout& sl) {
        stats = c.take<LenStats>(1);
        handles = c.take<ulonglong2>(N);
        ord = c.take<uint32_t>(N);
        lcp = c.take<uint32_t>(N);
        owner = c.take<uint16_t>(N);
        tmp = c.take<uint32_t>(N);
        runx = c.take<uint32_t>(N);
        srcb = out->source ? nullptr : c.take<uint32_t>(N);
        srcoff = c.take<uint64_t>(N);
        tc = c.take<uint32_t>(cells);
        off = c.take<uint32_t>(cells);
        cnt = c.take<uint32_t>(MAX_SPLIT_BUCKETS);
        prm = c.take<HqPe>(MAX_SPLIT_BUCKETS);
        cut = c.take<uint32_t>(MAX_SPLIT_BUCKETS);
        dest = c.take<uint32_t>(MAX_SPLIT_BUCKETS);
        err = c.take<uint32_t>(1);
        pbd = c.take<uint64_t>(p + 1);
        total = c.take<uint64_t>(2);
        scan = c.take<unsigned char>(scan_scratch_bytes(N > cells ? N : cells));
        layout_sort(c, sl, N, 1, smax);
    };
    ulonglong2* handles;
    uint32_t *ord, *lcp, *tmp, *runx, *srcb, *tc, *off, *cnt, *cut, *dest, *err;
    uint16_t* owner;
    HqPe* prm;
    uint64_t *pbd, *total, *srcoff;
    void* scan;
    LenStats* stats;
    SortLayout sl;
    Carve sz(nullptr);
    plan(sz, handles, ord, lcp, owner, tmp, runx, srcb, tc, off, cnt, prm, cut, dest, err, pbd, total, scan, srcoff,
         stats, sl);
    DSSS_TRY(ensure_ws(ctx, sz.used));
    const uint64_t pin_bytes = MAX_SPLIT_BUCKETS * (sizeof(uint32_t) + sizeof(HqPe)) + 64;
    DSSS_TRY(ensure_pin(ctx, pin_bytes < 4096 ? 4096 : pin_bytes));
    Carve c(ctx->ws);
    plan(c, handles, ord, lcp, owner, tmp, runx, srcb, tc, off, cnt, prm, cut, dest, err, pbd, total, scan, srcoff,
         stats, sl);
    ArenaDev a = view(in);
    DSSS_TRY(length_stats(a, stats, st));
    DSSS_CUDA(cudaMemsetAsync(err, 0, sizeof(uint32_t), st));
    LenStats* hstats = (LenStats*)((char*)ctx->pin + 128);
    DSSS_CUDA(cudaMemcpyAsync(hstats, stats, sizeof(LenStats), cudaMemcpyDeviceToHost, st));
    const uint64_t set_begin[2] = {0, n};
    {
        StageTimer t("stage:sort", st);
        DSSS_TRY(sort_strings(sl, a, n, 1, set_begin, nullptr, ord, lcp, (uint32_t*)ctx->pin, st, handles));
    }
    if (!a.h) {  // every string is gathered below
        DSSS_TRY(make_handles(a, handles, st));
        a.h = handles;
    }
    // the output layout: the PEs' sorted data in rank order is the global order
    uint32_t* source = out->source ? out->source : srcb;
    {
        StageTimer t("stage:layout", st);
        DSSS_LAUNCH("k_ms_source", st,
                    k_ms_source<<<grid_for(n, 256), 256, 0, st>>>(ord, nullptr, a, n, source, out->lengths, tmp,
                                                                 srcoff));
        DSSS_TRY(exclusive_scan_u32_to_u64(tmp, out->offsets, n, total, scan, st));
        const uint64_t bytes = hstats->sum + n;  // the sort has synchronised on st
        if (bytes > out->chars_capacity)
            return fail(DSSS_EINVAL, "chars_capacity %llu is below the %llu output bytes",
                        (unsigned long long)out->chars_capacity, (unsigned long long)bytes);
    }
    if (levels == 0) {  // one PE: the local sort is the result (RQuick.hpp:855-864)
        out->counts[0] = n;
    } else {
        StageTimer t("stage:levels", st);
        DSSS_CUDA(cudaMemcpyAsync(pbd, pb, (p + 1) * 8, cudaMemcpyHostToDevice, st));
        DSSS_LAUNCH("k_hq_run_ends", st,
                    k_hq_run_ends<<<grid_for(n, 256), 256, 0, st>>>(out->lengths, lcp, n, tmp));
        DSSS_TRY(exclusive_scan_u32(tmp, runx, n, nullptr, scan, st));
        const size_t hsm = pw * sizeof(uint32_t);
        DSSS_LAUNCH("k_hq_owner0", st,
                    k_hq_owner0<<<(unsigned)tiles, HQ_NT, hsm, st>>>(ord, n, pbd, p, pw, tiles, owner, tc));
        std::vector<HqBits> bits(pw);
        for (uint32_t q = 0; q < pw; ++q) bits[q].gen.seed(seed + q);  // HQuicksort.cpp:344-345
        uint32_t* hcnt = (uint32_t*)ctx->pin;
        HqPe* hprm = (HqPe*)((char*)ctx->pin + MAX_SPLIT_BUCKETS * sizeof(uint32_t));
        for (uint32_t P = pw;; P >>= 1) {
            DSSS_TRY(exclusive_scan_u32(tc, off, cells, nullptr, scan, st));
            DSSS_LAUNCH("k_hq_counts", st, k_hq_counts<<<grid_for(pw, 128), 128, 0, st>>>(off, tiles, pw, n, cnt));
            DSSS_CUDA(cudaMemcpyAsync(hcnt, cnt, pw * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
            DSSS_CUDA(cudaStreamSynchronize(st));
            if (P < 2) break;  // the counts after the last level
            // the bits in the reference's order per PE: middleMostElements
            // (:273-314), the first PE's selectMedian
            // (BinTreeMedianSelection.hpp:135-152), locateSplitter (:363-385)
            uint64_t sum = 0;
            for (uint32_t q = 0; q < pw; ++q) {
                const uint32_t k = hcnt[q];
                HqPe& m = hprm[q];
                sum += k;
                m.cnt = k;
                m.cube = P;
                m.piv = HQ_NONE;
                const uint32_t beg = k > 2 ? (k - 2) / 2 + (k % 2 == 1 ? bits[q].next() : 0u) : 0u;
                if (q % P == 0) {
                    const uint32_t nm = k < 2 ? k : 2;
                    if (nm) m.piv = beg + (nm == 2 ? bits[q].next() : 0u);
                }
                m.opt = k / 2 + (k % 2 == 1 ? bits[q].next() : 0u);
            }
            if (sum != n) return fail(DSSS_EDEVICE, "hq sort: owner counts add up to %llu, not %llu",
                                      (unsigned long long)sum, (unsigned long long)n);
            DSSS_CUDA(cudaMemcpyAsync(prm, hprm, pw * sizeof(HqPe), cudaMemcpyHostToDevice, st));
            DSSS_LAUNCH("k_hq_split", st,
                        k_hq_split<<<pw, HQ_NT, 0, st>>>(prm, owner, off, tiles, runx, ord, a, n, pw, cut, dest, err));
            DSSS_LAUNCH("k_hq_move", st,
                        k_hq_move<<<(unsigned)tiles, HQ_NT, hsm, st>>>(owner, n, pw, tiles, cut, dest, tc));
            // the pinned parameters are rewritten only after the next count
            // read-back, which the stream orders after this copy
        }
        uint64_t sum = 0;
        for (uint32_t q = 0; q < pw; ++q) sum += out->counts[q] = hcnt[q];
        if (sum != n) return fail(DSSS_EDEVICE, "hq sort: final counts add up to %llu, not %llu",
                                  (unsigned long long)sum, (unsigned long long)n);
    }
    {
        StageTimer t("stage:copy", st);
        DSSS_TRY(launch_ms_copy(a.chars, srcoff, out->lengths, out->offsets, n, out->chars, st));
    }
    DSSS_CUDA(cudaMemcpyAsync(ctx->pin, err, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    DSSS_CUDA(cudaStreamSynchronize(st));
    if (*(const uint32_t*)ctx->pin) return fail(DSSS_EDEVICE, "hq sort: internal consistency guard tripped");
    return DSSS_OK;
}

}  // namespace dsss

using namespace dsss;

extern "C" {

int dsss_hq_sort(dsss_ctx* ctx, const dsss_arena* in, uint32_t p, const uint64_t* part_begin, uint64_t seed,
                 dsss_hq_result* out, dsss_stream_t stream) {
    if (!ctx) return fail(DSSS_EINVAL, "ctx is NULL");
    ActiveCtx active(ctx);
    DSSS_CUDA(cudaSetDevice(ctx->device));
    return hq_sort_dev(ctx, in, p, part_begin, seed, out, (cudaStream_t)stream);
}

int dsss_ms_sort(dsss_ctx* ctx, const dsss_arena* in, uint32_t p, const uint64_t* part_begin, const dsss_opts* opts,
                 dsss_ms_result* out, dsss_stream_t stream) {
    if (!ctx) return fail(DSSS_EINVAL, "ctx is NULL");
    ActiveCtx active(ctx);
    DSSS_CUDA(cudaSetDevice(ctx->device));
    return ms_sort_dev(ctx, in, p, part_begin, opts, out, (cudaStream_t)stream);
}

int dsss_pd_sort(dsss_ctx* ctx, const dsss_arena* in, uint32_t p, const uint64_t* part_begin, const dsss_opts* opts,
                 dsss_pd_result* out, dsss_stream_t stream) {
    if (!ctx) return fail(DSSS_EINVAL, "ctx is NULL");
    ActiveCtx active(ctx);
    DSSS_CUDA(cudaSetDevice(ctx->device));
    return pd_sort_dev(ctx, in, 1, p, part_begin, opts, out, (cudaStream_t)stream);
}

int dsss_pd_sort_batched(dsss_ctx* ctx, const dsss_arena* in, uint32_t nsets, uint32_t p, const uint64_t* part_begin,
                         const dsss_opts* opts, dsss_pd_result* out, dsss_stream_t stream) {
    if (!ctx) return fail(DSSS_EINVAL, "ctx is NULL");
    ActiveCtx active(ctx);
    DSSS_CUDA(cudaSetDevice(ctx->device));
    return pd_sort_dev(ctx, in, nsets, p, part_begin, opts, out, (cudaStream_t)stream);
}

int dsss_local_sort_lcp(dsss_ctx* ctx, const dsss_arena* in, uint32_t p, const uint64_t* part_begin,
                        const dsss_opts* opts, uint32_t* order, uint32_t* lcp, dsss_stream_t stream) {
    if (!ctx) return fail(DSSS_EINVAL, "ctx is NULL");
    ActiveCtx active(ctx);
    DSSS_TRY(check_arena(in));
    DSSS_TRY(check_parts(p, part_begin, in->n));
    if (in->n && (!order || !lcp)) return fail(DSSS_EINVAL, "order/lcp is NULL");
    DSSS_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t st = (cudaStream_t)stream;
    const uint32_t smax = smallmax_of(opts);
    Carve sz(nullptr);
    SortLayout L;
    sz.take<ulonglong2>(in->n ? in->n : 1);
    layout_sort(sz, L, in->n, p, smax);
    DSSS_TRY(ensure_ws(ctx, sz.used));
    DSSS_TRY(ensure_pin(ctx, 4096));
    Carve c(ctx->ws);
    ulonglong2* h = c.take<ulonglong2>(in->n ? in->n : 1);
    layout_sort(c, L, in->n, p, smax);
    ArenaDev a = view(in);
    return sort_strings(L, a, in->n, p, part_begin, nullptr, order, lcp, (uint32_t*)ctx->pin, st, h);
}

int dsss_dp_prefixes(dsss_ctx* ctx, const dsss_arena* in, uint32_t p, const uint64_t* part_begin,
                     const uint32_t* order, const uint32_t* lcp, uint32_t* dp, uint64_t* round_counts,
                     uint32_t max_rounds, uint32_t* rounds, dsss_stream_t stream) {
    if (!ctx) return fail(DSSS_EINVAL, "ctx is NULL");
    ActiveCtx active(ctx);
    DSSS_TRY(check_arena(in));
    DSSS_TRY(check_parts(p, part_begin, in->n));
    if (in->n && (!order || !lcp || !dp)) return fail(DSSS_EINVAL, "order/lcp/dp is NULL");
    DSSS_CUDA(cudaSetDevice(ctx->device));
    Carve sz(nullptr);
    DpLayout L;
    sz.take<ulonglong2>(in->n ? in->n : 1);
    layout_dp(sz, L, in->n);
    DSSS_TRY(ensure_ws(ctx, sz.used));
    DSSS_TRY(ensure_pin(ctx, 4096));
    Carve c(ctx->ws);
    ulonglong2* h = c.take<ulonglong2>(in->n ? in->n : 1);
    layout_dp(c, L, in->n);
    ArenaDev a = view(in);
    DSSS_TRY(make_handles(a, h, (cudaStream_t)stream));
    a.h = h;
    // The PE split needs no extra handling: every PE's first LCP is 0, so no
    // string is an LCP duplicate of the previous PE's last one.
    return dp_rounds(L, a, in->n, order, lcp, dp, round_counts, max_rounds, rounds, (uint32_t*)ctx->pin,
                     (cudaStream_t)stream);
}

int dsss_dp_round(dsss_ctx* ctx, const dsss_arena* in, const uint32_t* order, const uint32_t* lcp,
                  const uint32_t* candidates, uint64_t m, uint32_t depth, uint32_t* results, uint32_t* next,
                  uint64_t* m_next, dsss_stream_t stream) {
    if (!ctx) return fail(DSSS_EINVAL, "ctx is NULL");
    ActiveCtx active(ctx);
    DSSS_TRY(check_arena(in));
    if (!m_next) return fail(DSSS_EINVAL, "m_next is NULL");
    if (in->n && (!order || !lcp || !results || !next)) return fail(DSSS_EINVAL, "order/lcp/results/next is NULL");
    if (candidates && m > in->n) return fail(DSSS_EINVAL, "more candidates than strings");
    DSSS_CUDA(cudaSetDevice(ctx->device));
    Carve sz(nullptr);
    DpRoundLayout R;
    layout_dp_round(sz, R, in->n);
    DSSS_TRY(ensure_ws(ctx, sz.used));
    DSSS_TRY(ensure_pin(ctx, 4096));
    Carve c(ctx->ws);
    layout_dp_round(c, R, in->n);
    return dp_one_round(R, view(in), in->n, order, lcp, candidates, m, depth, results, next, m_next,
                        (uint32_t*)ctx->pin, (cudaStream_t)stream);
}

int dsss_bucket_scatter(dsss_ctx* ctx, const dsss_arena* in, uint32_t p, const uint64_t* part_begin,
                        const uint32_t* local_order, const uint32_t* lcp, const uint32_t* dp, const uint64_t* intervals,
                        uint8_t* recv_chars, uint64_t recv_capacity, uint64_t* char_total, uint64_t* recv_char_begin,
                        uint32_t* recv_char_start, uint32_t* recv_lcp, uint32_t* recv_index, uint32_t* recv_pe,
                        uint64_t* recv_counts, uint64_t* recv_offsets, dsss_stream_t stream) {
    if (!ctx) return fail(DSSS_EINVAL, "ctx is NULL");
    ActiveCtx active(ctx);
    DSSS_TRY(check_arena(in));
    DSSS_TRY(check_parts(p, part_begin, in->n));
    if (!intervals || !char_total) return fail(DSSS_EINVAL, "intervals/char_total is NULL");
    if (in->n && (!local_order || !lcp || !dp || !recv_lcp || !recv_index || !recv_pe))
        return fail(DSSS_EINVAL, "input or per-string output array is NULL");
    DSSS_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t st = (cudaStream_t)stream;
    Carve sz(nullptr);
    ExchangeLayout L;
    layout_exchange(sz, L, in->n, p);
    DSSS_TRY(ensure_ws(ctx, sz.used));
    DSSS_TRY(ensure_pin(ctx, 4096));
    Carve c(ctx->ws);
    layout_exchange(c, L, in->n, p);
    DSSS_TRY(bucket_scatter(L, view(in), p, part_begin, local_order, lcp, dp, intervals, char_total, recv_chars,
                            recv_capacity, recv_char_begin, recv_lcp, recv_index, recv_pe, recv_counts, recv_offsets,
                            (uint32_t*)ctx->pin, st));
    if (recv_char_start && in->n)
        DSSS_CUDA(cudaMemcpyAsync(recv_char_start, L.cstart, in->n * 4, cudaMemcpyDeviceToDevice, st));
    DSSS_CUDA(cudaStreamSynchronize(st));
    return DSSS_OK;
}

int dsss_lcp_merge(dsss_ctx* ctx, const uint8_t* recv_chars, uint64_t char_bytes, const uint32_t* recv_char_start,
                   const uint32_t* recv_lcp, uint64_t n, uint32_t nrecv, uint32_t p, const uint64_t* recv_counts,
                   const uint64_t* recv_offsets, uint32_t* order, uint32_t* merged_lcp, uint32_t* old_lcp,
                   uint32_t* perm_index, uint32_t* perm_pe, dsss_stream_t stream) {
    if (!ctx) return fail(DSSS_EINVAL, "ctx is NULL");
    ActiveCtx active(ctx);
    if (nrecv == 0 || p == 0 || !recv_counts) return fail(DSSS_EINVAL, "nrecv/p/recv_counts missing");
    if (n && (!recv_chars || !recv_lcp || !order)) return fail(DSSS_EINVAL, "recv_chars/recv_lcp/order is NULL");
    DSSS_CUDA(cudaSetDevice(ctx->device));
    int rc = lcp_merge(ctx, recv_chars, char_bytes, recv_char_start, recv_lcp, n, nrecv, p, recv_counts, recv_offsets,
                       order, merged_lcp, old_lcp, perm_index, perm_pe, (cudaStream_t)stream);
    return rc;
}

int dsss_lcp_merge_strings(dsss_ctx* ctx, const uint8_t* recv_chars, uint64_t char_bytes,
                           const uint32_t* recv_char_start, const uint32_t* recv_lcp, uint64_t n, uint32_t nrecv,
                           uint32_t p, const uint64_t* recv_counts, const uint64_t* recv_offsets, uint32_t* order,
                           uint32_t* merged_lcp, uint8_t* out_chars, uint64_t out_capacity, uint64_t* out_offsets,
                           uint32_t* out_lengths, uint64_t* out_bytes, dsss_stream_t stream) {
    if (!ctx) return fail(DSSS_EINVAL, "ctx is NULL");
    ActiveCtx active(ctx);
    if (nrecv == 0 || p == 0 || !recv_counts || !out_bytes) return fail(DSSS_EINVAL, "nrecv/p/recv_counts/out_bytes missing");
    if (n && (!recv_chars || !recv_lcp || !order || !out_chars || !out_offsets || !out_lengths))
        return fail(DSSS_EINVAL, "input or output arrays are NULL");
    DSSS_CUDA(cudaSetDevice(ctx->device));
    return lcp_merge_strings(ctx, recv_chars, char_bytes, recv_char_start, recv_lcp, n, nrecv, p, recv_counts,
                             recv_offsets, order, merged_lcp, nullptr, nullptr, nullptr, out_chars, out_capacity,
                             out_offsets, out_lengths, out_bytes, (cudaStream_t)stream);
}

int dsss_prefix_hash(const dsss_arena* in, const uint32_t* ids, uint64_t m, uint32_t depth, uint64_t* hash,
                     dsss_stream_t stream) {
    DSSS_TRY(check_arena(in));
    if (m && (!ids || !hash)) return fail(DSSS_EINVAL, "ids/hash is NULL");
    return prefix_hash(view(in), ids, m, depth, hash, (cudaStream_t)stream);
}

int dsss_partition(dsss_ctx* ctx, const dsss_arena* in, uint32_t p, const uint64_t* part_begin,
                   const uint32_t* order, const uint32_t* dp, const dsss_opts* opts, uint64_t* intervals,
                   dsss_stream_t stream) {
    if (!ctx) return fail(DSSS_EINVAL, "ctx is NULL");
    ActiveCtx active(ctx);
    DSSS_TRY(check_arena(in));
    DSSS_TRY(check_parts(p, part_begin, in->n));
    if (!intervals || (in->n && (!order || !dp))) return fail(DSSS_EINVAL, "order/dp/intervals is NULL");
    DSSS_CUDA(cudaSetDevice(ctx->device));
    const uint32_t factor = factor_of(opts);
    Carve sz(nullptr);
    PartitionLayout L;
    layout_partition(sz, L, in->n, p, factor);
    DSSS_TRY(ensure_ws(ctx, sz.used));
    Carve c(ctx->ws);
    layout_partition(c, L, in->n, p, factor);
    return partition_pes(L, ctx, view(in), p, part_begin, order, dp, sampler_of(opts), factor, intervals,
                         (cudaStream_t)stream);
}

int dsss_adjacent_lcp(dsss_ctx* ctx, const dsss_arena* in, const uint32_t* order, uint64_t m, uint32_t* lcp,
                      dsss_stream_t stream) {
    if (!ctx) return fail(DSSS_EINVAL, "ctx is NULL");
    ActiveCtx active(ctx);
    DSSS_TRY(check_arena(in));
    if (m && (!order || !lcp)) return fail(DSSS_EINVAL, "order/lcp is NULL");
    DSSS_CUDA(cudaSetDevice(ctx->device));
    Carve sz(nullptr);
    sz.take<uint32_t>(m + 1);
    sz.take<uint32_t>(1);
    DSSS_TRY(ensure_ws(ctx, sz.used));
    Carve c(ctx->ws);
    uint32_t* longq = c.take<uint32_t>(m + 1);
    uint32_t* nlong = c.take<uint32_t>(1);
    return adjacent_lcp(view(in), order, m, lcp, longq, nlong, (cudaStream_t)stream);
}

// Host-memory variant: device copies of the arena and results live in a
// second context buffer so repeated calls reuse it.
static int pd_sort_host(dsss_ctx* ctx, const dsss_arena* in, uint32_t nsets, uint32_t p, const uint64_t* part_begin,
                        const dsss_opts* opts, dsss_pd_result* out, dsss_stream_t stream) {
    if (!ctx) return fail(DSSS_EINVAL, "ctx is NULL");
    ActiveCtx active(ctx);
    if (!in) return fail(DSSS_EINVAL, "arena is NULL");
    if (nsets == 0 || p == 0) return fail(DSSS_EINVAL, "nsets and p must be >= 1");
    DSSS_TRY(check_parts(nsets * p, part_begin, in->n));
    if (!out) return fail(DSSS_EINVAL, "result is NULL");
    DSSS_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t st = (cudaStream_t)stream;
    const uint64_t n = in->n;
    const bool llcp = opts && (opts->flags & DSSS_FLAG_LOCAL_LCP) && out->local_lcp;
    auto plan = [&](Carve& c, dsss_arena& da, dsss_pd_result& dr) {
        uint8_t* chars = c.take<uint8_t>(in->char_bytes + 64);
        uint64_t* off = c.take<uint64_t>(n ? n : 1);
        uint32_t* len = c.take<uint32_t>(n ? n : 1);
        da = dsss_arena{chars, in->char_bytes, off, len, n};
        dr = *out;
        dr.local_order = c.take<uint32_t>(n ? n : 1);
        dr.local_lcp = llcp ? c.take<uint32_t>(n ? n : 1) : nullptr;
        dr.dp = c.take<uint32_t>(n ? n : 1);
        dr.perm_index = c.take<uint32_t>(n ? n : 1);
        dr.perm_pe = c.take<uint32_t>(n ? n : 1);
        dr.merged_lcp = out->merged_lcp ? c.take<uint32_t>(n ? n : 1) : nullptr;
    };
    Carve sz(nullptr);
    dsss_arena da;
    dsss_pd_result dr;
    plan(sz, da, dr);
    // The io buffer sits in front of the pipeline's own scratch.
    Carve pdsz(nullptr);
    PdLayout PL;
    layout_pd(pdsz, PL, n, nsets, p, smallmax_of(opts));
    const uint64_t io_bytes = (sz.used + 255) & ~255ull;
    DSSS_TRY(ensure_ws(ctx, io_bytes + pdsz.used));
    Carve c(ctx->ws);
    plan(c, da, dr);
    if (in->char_bytes) DSSS_CUDA(cudaMemcpyAsync((void*)da.chars, in->chars, in->char_bytes, cudaMemcpyHostToDevice, st));
    DSSS_CUDA(cudaMemsetAsync((uint8_t*)da.chars + in->char_bytes, 0, 64, st));
    if (n) {
        DSSS_CUDA(cudaMemcpyAsync((void*)da.offsets, in->offsets, n * 8, cudaMemcpyHostToDevice, st));
        DSSS_CUDA(cudaMemcpyAsync((void*)da.lengths, in->lengths, n * 4, cudaMemcpyHostToDevice, st));
    }
    // Run the device path on the scratch behind the io block.
    Ctx sub = *ctx;
    sub.ws = (char*)ctx->ws + io_bytes;
    sub.ws_cap = ctx->ws_cap - io_bytes;
    sub.fixed_ws = true;
    int rc = pd_sort_dev(&sub, &da, nsets, p, part_begin, opts, &dr, st);
    ctx->pin = sub.pin;
    ctx->pin_cap = sub.pin_cap;
    if (rc != DSSS_OK) return rc;
    if (n) {
        DSSS_CUDA(cudaMemcpyAsync(out->local_order, dr.local_order, n * 4, cudaMemcpyDeviceToHost, st));
        if (llcp) DSSS_CUDA(cudaMemcpyAsync(out->local_lcp, dr.local_lcp, n * 4, cudaMemcpyDeviceToHost, st));
        if (p > 1) {
            DSSS_CUDA(cudaMemcpyAsync(out->dp, dr.dp, n * 4, cudaMemcpyDeviceToHost, st));
            DSSS_CUDA(cudaMemcpyAsync(out->perm_index, dr.perm_index, n * 4, cudaMemcpyDeviceToHost, st));
            DSSS_CUDA(cudaMemcpyAsync(out->perm_pe, dr.perm_pe, n * 4, cudaMemcpyDeviceToHost, st));
            if (out->merged_lcp)
                DSSS_CUDA(cudaMemcpyAsync(out->merged_lcp, dr.merged_lcp, n * 4, cudaMemcpyDeviceToHost, st));
        }
    }
    DSSS_CUDA(cudaStreamSynchronize(st));
    return DSSS_OK;
}

int dsss_pd_sort_host(dsss_ctx* ctx, const dsss_arena* in, uint32_t p, const uint64_t* part_begin,
                      const dsss_opts* opts, dsss_pd_result* out, dsss_stream_t stream) {
    return pd_sort_host(ctx, in, 1, p, part_begin, opts, out, stream);
}

int dsss_pd_sort_batched_host(dsss_ctx* ctx, const dsss_arena* in, uint32_t nsets, uint32_t p,
                              const uint64_t* part_begin, const dsss_opts* opts, dsss_pd_result* out,
                              dsss_stream_t stream) {
    return pd_sort_host(ctx, in, nsets, p, part_begin, opts, out, stream);
}

}  // extern "C"
