// How the varint decoder reads its coded bytes; host code too, so that what it
// touches can be checked without a GPU.
#pragma once
#include <vector_functions.h>
#include <vector_types.h>

#include <cstdint>

namespace dsss {

// The coded bytes [mis, end) of 16-byte words, counted from the aligned word
// that holds the first.
struct CodedBytes {
    const uint4* words;
    uint32_t mis;
    uint64_t end;  // mis + bytes
};

inline CodedBytes coded_bytes(const uint8_t* in, uint64_t nbytes) {
    const uint32_t mis = (uint32_t)((uintptr_t)in & 15);
    return CodedBytes{reinterpret_cast<const uint4*>(in - mis), mis, mis + nbytes};
}

// Word i, zero outside the coded bytes.  The buffer has no padding, so the
// first and the last word are read byte by byte where they are not whole.
__host__ __device__ __forceinline__ uint4 coded_word(const CodedBytes& c, uint64_t i) {
    const uint64_t b = 16 * i;
    if (b >= c.mis && b + 16 <= c.end) {
#ifdef __CUDA_ARCH__
        return __ldg(c.words + i);
#else
        return c.words[i];
#endif
    }
    const uint8_t* p = reinterpret_cast<const uint8_t*>(c.words + i);
    uint32_t x[4] = {0, 0, 0, 0};
#pragma unroll
    for (uint32_t k = 0; k < 16; ++k)
        if (b + k >= c.mis && b + k < c.end) x[k / 4] |= (uint32_t)p[k] << 8 * (k % 4);
    return make_uint4(x[0], x[1], x[2], x[3]);
}

}  // namespace dsss
