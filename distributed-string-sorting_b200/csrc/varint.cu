// Varint coding of LCP arrays for the string exchange with compressLcps
// (sendLcps, src/mpi/alltoall.hpp:406-425): Writer::PutVarint
// (src/encoding/integer_compression.hpp:66-140) writes 7 bits per byte, least
// significant first, the high bit set on every byte but the last; ranges
// (one per destination) are encoded back to back (IntegerCompression::
// writeRanges, src/mpi/byte_encoder.hpp:31-53) and decoded the same way
// (readRanges, :63-77).  On the GPU both directions are data-parallel, and
// both touch the values and the bytes twice, once to count per tile and once
// to code, with a scan of the tiles' counts between; the places inside a tile
// come from a scan in its block, and what a tile writes is put together in
// shared memory and leaves it in whole words.  Bound by memory: 16e6 values to
// 19e6 bytes and back, size query included: 0.62 -> 0.17 ms.
#include <vector>

#include "internal.cuh"
#include "varint_bytes.cuh"

namespace dsss {

constexpr uint32_t VI_NT = 256, VI_IPT = 16, VI_TILE = VI_NT * VI_IPT;  // values, or bytes, of a tile

__device__ __forceinline__ uint32_t varint_size(uint32_t v) {
    return v < (1u << 7) ? 1 : v < (1u << 14) ? 2 : v < (1u << 21) ? 3 : v < (1u << 28) ? 4 : 5;
}

// Exclusive sum of v over the block; *total (optional): the sum of all.
__device__ __forceinline__ uint32_t vi_scan(uint32_t v, uint32_t* total) {
    __shared__ uint32_t ws[VI_NT / 32];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    uint32_t before = 0, all = 0;
#pragma unroll
    for (uint32_t q = 0; q < VI_NT / 32; ++q) {
        if (q == w) before = all;
        all += ws[q];
    }
    if (total) *total = all;
    return before + x - v;
}

// Coded bytes of each tile.
__global__ void __launch_bounds__(VI_NT) k_varint_sizes(const uint32_t* v, uint64_t n, uint32_t* sizes) {
    uint32_t x[VI_IPT], s = 0;
#pragma unroll
    for (uint32_t j = 0; j < VI_IPT; ++j) {
        const uint64_t i = (uint64_t)blockIdx.x * VI_TILE + j * VI_NT + threadIdx.x;
        x[j] = i < n ? v[i] : 0u;
    }
#pragma unroll
    for (uint32_t j = 0; j < VI_IPT; ++j)
        if ((uint64_t)blockIdx.x * VI_TILE + j * VI_NT + threadIdx.x < n) s += varint_size(x[j]);
    uint32_t total;
    vi_scan(s, &total);
    if (threadIdx.x == 0) sizes[blockIdx.x] = total;
}

// Codes a tile at out + at[tile].
__global__ void __launch_bounds__(VI_NT) k_varint_write(const uint32_t* v, uint64_t n, const uint64_t* at, uint8_t* out) {
    __shared__ uint32_t sv[VI_TILE + VI_NT];                    // a thread's 16 values, one word apart from the next's
    __shared__ __align__(16) uint8_t sb[5 * VI_TILE + 16];      // as misaligned as the output
    const uint64_t tb = (uint64_t)blockIdx.x * VI_TILE;
    const uint32_t tn = (uint32_t)min((uint64_t)VI_TILE, n - tb);
#pragma unroll
    for (uint32_t j = 0; j < VI_IPT; ++j) {
        const uint32_t i = j * VI_NT + threadIdx.x;
        sv[i + i / VI_IPT] = i < tn ? v[tb + i] : 0u;
    }
    __syncthreads();
    uint32_t x[VI_IPT], s = 0;
#pragma unroll
    for (uint32_t j = 0; j < VI_IPT; ++j) {
        const uint32_t i = threadIdx.x * VI_IPT + j;
        x[j] = sv[i + threadIdx.x];
        if (i < tn) s += varint_size(x[j]);
    }
    uint32_t total;
    uint8_t* dst = out + at[blockIdx.x];
    const uint32_t mis = (uint32_t)((uintptr_t)dst & 15);
    uint32_t o = mis + vi_scan(s, &total);
#pragma unroll
    for (uint32_t j = 0; j < VI_IPT; ++j) {
        if (threadIdx.x * VI_IPT + j >= tn) break;
        uint32_t y = x[j];
        for (; y >= 0x80u; y >>= 7) sb[o++] = (uint8_t)(y | 0x80u);
        sb[o++] = (uint8_t)y;
    }
    __syncthreads();
    uint8_t* d0 = dst - mis;  // aligned; only [mis, mis + total) of it is written
    for (uint32_t k = threadIdx.x * 16; k < mis + total; k += VI_NT * 16) {
        if (k >= mis && k + 16 <= mis + total) {
            *reinterpret_cast<uint4*>(d0 + k) = *reinterpret_cast<const uint4*>(sb + k);
        } else {
            for (uint32_t b = max(k, mis); b < min(k + 16, mis + total); ++b) d0[b] = sb[b];
        }
    }
}

// Byte offsets of the range boundaries (value indices), one warp each: the
// tile's offset and the sizes in the tile up to the boundary.
__global__ void __launch_bounds__(128) k_varint_bounds(const uint32_t* v, uint64_t n, const uint64_t* at, uint64_t total,
                                                       const uint64_t* bound, uint32_t nb, uint64_t* out) {
    const uint32_t r = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (r >= nb) return;
    const uint64_t e = bound[r];
    if (e >= n) {
        if ((threadIdx.x & 31) == 0) out[r] = total;
        return;
    }
    uint32_t s = 0;
    const uint64_t b = e / VI_TILE * VI_TILE;
#pragma unroll 8
    for (uint64_t i = b + (threadIdx.x & 31); i < e; i += 32) s += varint_size(v[i]);
    s = __reduce_add_sync(0xffffffffu, s);
    if ((threadIdx.x & 31) == 0) out[r] = at[e / VI_TILE] + s;
}

// The same with more boundaries than tiles: a block per tile scans its sizes
// once and serves every boundary in it (the last tile also those at n).
__global__ void __launch_bounds__(VI_NT) k_varint_bounds_tiled(const uint32_t* v, uint64_t n, const uint64_t* at,
                                                               uint64_t total, const uint64_t* bound, uint32_t nb,
                                                               uint64_t* out) {
    __shared__ uint32_t pre[VI_TILE];
    const uint64_t tb = (uint64_t)blockIdx.x * VI_TILE;
    uint32_t sz[VI_IPT], s = 0;
#pragma unroll
    for (uint32_t j = 0; j < VI_IPT; ++j) {
        const uint64_t i = tb + threadIdx.x * VI_IPT + j;
        sz[j] = i < n ? varint_size(v[i]) : 0u;
        s += sz[j];
    }
    uint32_t o = vi_scan(s, nullptr);
#pragma unroll
    for (uint32_t j = 0; j < VI_IPT; ++j) {
        pre[threadIdx.x * VI_IPT + j] = o;
        o += sz[j];
    }
    __syncthreads();
    const uint32_t lo = first_at_least(bound, nb, tb);
    const uint32_t hi = blockIdx.x + 1 == gridDim.x ? nb : first_at_least(bound, nb, tb + VI_TILE);
    for (uint32_t r = lo + threadIdx.x; r < hi; r += VI_NT) out[r] = bound[r] < n ? at[blockIdx.x] + pre[bound[r] - tb] : total;
}

// Bit b: byte b of word i (of the thread) is the last one of a value.
__device__ __forceinline__ uint32_t value_ends(const CodedBytes& c, uint64_t i, uint4& w) {
    w = make_uint4(0, 0, 0, 0);
    if (16 * i >= c.end) return 0;
    w = coded_word(c, i);
    const uint32_t x[4] = {w.x, w.y, w.z, w.w};
    uint32_t m = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) m |= (((~x[q] & 0x80808080u) >> 7) * 0x10204080u >> 28) << 4 * q;  // the four flags, first byte lowest
    if (i == 0) m &= 0xFFFFu << c.mis;
    if (16 * i + 16 > c.end) m &= (1u << (c.end - 16 * i)) - 1u;
    return m;
}

// Values that end in each tile; err: the last value is cut off.
__global__ void __launch_bounds__(VI_NT) k_varint_ends(CodedBytes c, uint32_t* counts, uint32_t* err) {
    const uint64_t i = (uint64_t)blockIdx.x * VI_NT + threadIdx.x;
    uint4 w;
    const uint32_t m = value_ends(c, i, w);
    uint32_t total;
    vi_scan(__popc(m), &total);
    if (threadIdx.x == 0) counts[blockIdx.x] = total;
    if (16 * i < c.end && c.end <= 16 * i + 16 && !(m >> ((c.end - 1) & 15) & 1u)) atomicExch(err, 1u);
}

// The values that end in a tile, each put together from its last byte
// backwards.  Nothing is written unless the bytes hold n values.
__global__ void __launch_bounds__(VI_NT) k_varint_read(CodedBytes c, const uint32_t* before, const uint32_t* total,
                                                       uint64_t n, uint32_t* v, uint32_t* err) {
    __shared__ __align__(16) uint8_t sb[VI_TILE + 16];  // 16 bytes of the tile before
    __shared__ uint32_t sv[VI_TILE];
    if (*total != n) return;
    const uint64_t i = (uint64_t)blockIdx.x * VI_NT + threadIdx.x;
    uint4 w;
    const uint32_t ends = value_ends(c, i, w);
    *reinterpret_cast<uint4*>(sb + 16 + 16 * threadIdx.x) = w;
    if (threadIdx.x == 0) *reinterpret_cast<uint4*>(sb) = i ? coded_word(c, i - 1) : make_uint4(0, 0, 0, 0);
    uint32_t cnt;
    uint32_t o = vi_scan(__popc(ends), &cnt);  // its barrier covers sb
    const uint32_t first = blockIdx.x ? 0u : c.mis + 16u;  // first byte of the stream in sb
    bool bad = false;
    for (uint32_t m = ends; m; m &= m - 1) {
        uint32_t b = 16 + 16 * threadIdx.x + __ffs(m) - 1, len = 1;
        uint64_t x = sb[b];
        while (len <= 5 && b > first && (sb[b - 1] & 0x80u)) {
            x = x << 7 | (sb[--b] & 0x7Fu);
            ++len;
        }
        if (len > 5) x = 0;  // more than 5 bytes: not a 32-bit value
        bad = bad || len > 5 || x > 0xFFFFFFFFull;
        sv[o++] = (uint32_t)x;
    }
    if (bad) atomicExch(err, 1u);
    __syncthreads();
    const uint64_t at = before[blockIdx.x];
    for (uint32_t k = threadIdx.x; k < cnt; k += VI_NT)
        if (at + k < n) v[at + k] = sv[k];
}

}  // namespace dsss

using namespace dsss;

extern "C" {

int dsss_varint_encode(dsss_ctx* ctx, const uint32_t* values, uint64_t n, const uint64_t* range_begin,
                       uint32_t nranges, uint8_t* out, uint64_t out_cap, uint64_t* out_bytes, uint64_t* range_bytes,
                       dsss_stream_t stream) {
    if (!ctx) return fail(DSSS_EINVAL, "ctx is NULL");
    ActiveCtx active(ctx);
    if (!out_bytes || (nranges && (!range_begin || !range_bytes))) return fail(DSSS_EINVAL, "output pointers missing");
    if (n && !values) return fail(DSSS_EINVAL, "values is NULL");
    if (nranges && range_begin[0] != 0) return fail(DSSS_EINVAL, "range_begin must start at 0");
    for (uint32_t r = 0; r < nranges; ++r)
        if (range_begin[r] > range_begin[r + 1] || range_begin[r + 1] > n)
            return fail(DSSS_EINVAL, "range_begin must rise from 0 to at most n");
    DSSS_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t st = (cudaStream_t)stream;
    const uint64_t tiles = n ? (n + VI_TILE - 1) / VI_TILE : 1;
    auto plan = [&](Carve& c, uint32_t*& sz, uint64_t*& at, uint64_t*& tot, void*& scan, uint64_t*& bd,
                    uint64_t*& bo) {
        sz = c.take<uint32_t>(tiles);
        at = c.take<uint64_t>(tiles);
        tot = c.take<uint64_t>(1);
        scan = c.take<unsigned char>(scan_scratch_bytes(tiles));
        bd = c.take<uint64_t>(nranges + 1);
        bo = c.take<uint64_t>(nranges + 1);
    };
    uint32_t* sz;
    uint64_t *at, *tot, *bd, *bo;
    void* scan;
    Carve s0(nullptr);
    plan(s0, sz, at, tot, scan, bd, bo);
    DSSS_TRY(ensure_ws(ctx, s0.used));
    DSSS_TRY(ensure_pin(ctx, 8 * (nranges + 2)));
    Carve c(ctx->ws);
    plan(c, sz, at, tot, scan, bd, bo);
    uint64_t* pin = (uint64_t*)ctx->pin;
    uint64_t total = 0;
    if (n) {
        DSSS_LAUNCH("k_varint_sizes", st, k_varint_sizes<<<(unsigned)tiles, VI_NT, 0, st>>>(values, n, sz));
        DSSS_TRY(exclusive_scan_u32_to_u64(sz, at, tiles, tot, scan, st));
        DSSS_CUDA(cudaMemcpyAsync(pin, tot, 8, cudaMemcpyDeviceToHost, st));
        DSSS_CUDA(cudaStreamSynchronize(st));
        total = pin[0];
    }
    *out_bytes = total;
    if (!out) return DSSS_OK;  // size query
    if (total > out_cap) return fail(DSSS_EINVAL, "out_cap %llu below the %llu encoded bytes",
                                     (unsigned long long)out_cap, (unsigned long long)total);
    if (n) DSSS_LAUNCH("k_varint_write", st, k_varint_write<<<(unsigned)tiles, VI_NT, 0, st>>>(values, n, at, out));
    if (nranges) {
        DSSS_CUDA(cudaMemcpyAsync(bd, range_begin, (nranges + 1) * 8, cudaMemcpyHostToDevice, st));
        if (n && nranges >= tiles)
            DSSS_LAUNCH("k_varint_bounds", st,
                        k_varint_bounds_tiled<<<(unsigned)tiles, VI_NT, 0, st>>>(values, n, at, total, bd, nranges + 1, bo));
        else
            DSSS_LAUNCH("k_varint_bounds", st,
                        k_varint_bounds<<<grid_for(nranges + 1, 4), 128, 0, st>>>(values, n, at, total, bd, nranges + 1,
                                                                                 bo));
        DSSS_CUDA(cudaMemcpyAsync(pin, bo, (nranges + 1) * 8, cudaMemcpyDeviceToHost, st));
    }
    DSSS_CUDA(cudaStreamSynchronize(st));
    for (uint32_t r = 0; r < nranges; ++r) range_bytes[r] = pin[r + 1] - pin[r];
    return DSSS_OK;
}

int dsss_varint_decode(dsss_ctx* ctx, const uint8_t* in, uint64_t nbytes, uint32_t* values, uint64_t n,
                       dsss_stream_t stream) {
    if (!ctx) return fail(DSSS_EINVAL, "ctx is NULL");
    ActiveCtx active(ctx);
    if ((nbytes && !in) || (n && !values)) return fail(DSSS_EINVAL, "buffers missing");
    DSSS_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t st = (cudaStream_t)stream;
    if (nbytes == 0) {
        if (n) return fail(DSSS_EINVAL, "no bytes for %llu values", (unsigned long long)n);
        return DSSS_OK;
    }
    if (nbytes >= (1ull << 32)) return fail(DSSS_ENOTSUP, "more than 4 GiB of coded values per call");
    const CodedBytes coded = coded_bytes(in, nbytes);
    const uint64_t tiles = (coded.end + VI_TILE - 1) / VI_TILE;
    auto plan = [&](Carve& c, uint32_t*& cnt, uint32_t*& at, void*& scan, uint32_t*& state) {
        cnt = c.take<uint32_t>(tiles);
        at = c.take<uint32_t>(tiles);
        scan = c.take<unsigned char>(scan_scratch_bytes(tiles));
        state = c.take<uint32_t>(2);  // values, error
    };
    uint32_t *cnt, *at, *state;
    void* scan;
    Carve s0(nullptr);
    plan(s0, cnt, at, scan, state);
    DSSS_TRY(ensure_ws(ctx, s0.used));
    DSSS_TRY(ensure_pin(ctx, 64));
    Carve c(ctx->ws);
    plan(c, cnt, at, scan, state);
    uint32_t* pin = (uint32_t*)ctx->pin;
    DSSS_CUDA(cudaMemsetAsync(state, 0, 8, st));
    DSSS_LAUNCH("k_varint_ends", st, k_varint_ends<<<(unsigned)tiles, VI_NT, 0, st>>>(coded, cnt, state + 1));
    DSSS_TRY(exclusive_scan_u32(cnt, at, tiles, state, scan, st));
    if (n)
        DSSS_LAUNCH("k_varint_read", st,
                    k_varint_read<<<(unsigned)tiles, VI_NT, 0, st>>>(coded, at, state, n, values, state + 1));
    DSSS_CUDA(cudaMemcpyAsync(pin, state, 8, cudaMemcpyDeviceToHost, st));
    DSSS_CUDA(cudaStreamSynchronize(st));
    if (pin[0] != n)
        return fail(DSSS_EINVAL, "the bytes hold %u values, not n = %llu", pin[0], (unsigned long long)n);
    if (pin[1]) return fail(DSSS_EINVAL, "a coded value is cut off, longer than 5 bytes or above 2^32 - 1");
    return DSSS_OK;
}

}  // extern "C"
