// Reads every word of a varint buffer as the decoder does, with the bytes
// around the buffer poisoned (AddressSanitizer): any touch of them ends the
// program.  Prints the bytes' sum per case.
#include <sanitizer/asan_interface.h>

#include <cstdio>
#include <cstdlib>
#include <initializer_list>

#include "varint_bytes.cuh"

static unsigned sum_of(uint4 w) {
    unsigned s = 0;
    for (unsigned x : {w.x, w.y, w.z, w.w})
        for (int k = 0; k < 4; ++k) s += (x >> 8 * k) & 0xFFu;
    return s;
}

int main() {
    constexpr unsigned CAP = 128;
    unsigned char* block = (unsigned char*)std::aligned_alloc(16, CAP);
    // poison has 8-byte grain in front of a byte that may be read, none behind one
    for (unsigned shift = 0; shift < 16; ++shift)
        for (unsigned n = 1; n <= 64; ++n) {
            unsigned want = 0;
            for (unsigned k = 0; k < CAP; ++k) block[k] = (unsigned char)(k + 1);
            for (unsigned k = 0; k < n; ++k) want += block[shift + k];
            ASAN_POISON_MEMORY_REGION(block, shift);
            ASAN_POISON_MEMORY_REGION(block + shift + n, CAP - shift - n);
            const dsss::CodedBytes c = dsss::coded_bytes(block + shift, n);
            unsigned got = 0;
            for (uint64_t i = 0; 16 * i < c.end; ++i) got += sum_of(dsss::coded_word(c, i));
            ASAN_UNPOISON_MEMORY_REGION(block, CAP);
            if (got != want) {
                std::printf("shift %u, %u bytes: %u instead of %u\n", shift, n, got, want);
                return 1;
            }
        }
    std::free(block);
    std::puts("ok");
    return 0;
}
