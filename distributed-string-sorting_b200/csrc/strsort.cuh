// Segmented MSD string sort with LCP output (K3); see strsort.cu.
#pragma once
#include "internal.cuh"

namespace dsss {

struct SortLayout {
    uint32_t* ord[2];
    unsigned long long* key[2];
    unsigned char* large[2];
    unsigned char* small[4];
    uint32_t* tile0;
    uint32_t* hist;
    uint32_t* bucket;
    uint32_t* cursor;
    uint32_t* counters;
    uint64_t* pb;
    uint32_t dbits, small_max;
    uint64_t cap_large, cap_small[4], cap_tiles;
};

constexpr uint32_t SORT_SMALL_MAX_DEFAULT = 4096;

// Scratch layout for sorting up to n strings in up to p segments.
void layout_sort(Carve& c, SortLayout& L, uint64_t n, uint32_t p, uint32_t small_max);

// Sorts ids (ids_in[i], or i when ids_in is NULL) within the segments
// [pb[q], pb[q+1]) by the bytes of their strings.  ord_out gets the sorted ids,
// lcp_out[i] the LCP with position i-1 (0 at segment starts).  pin: pinned
// host buffer of >= 16 u32 for count read-backs (the call synchronises on st).
// seg_depth (optional, device, p entries): the strings of segment q share
// their first seg_depth[q] bytes (the sort starts there).
// handles (optional, a.n entries, with a.h NULL): built, and put into a.h, once
// the sort goes back to the strings in an order other than the arena's; a sort
// whose first keys tell all strings apart never needs them.
int sort_strings(const SortLayout& L, ArenaDev& a, uint64_t n, uint32_t p, const uint64_t* pb_host,
                 const uint32_t* ids_in, uint32_t* ord_out, uint32_t* lcp_out, uint32_t* pin, cudaStream_t st,
                 ulonglong2* handles = nullptr, const uint32_t* seg_depth = nullptr);

}  // namespace dsss
