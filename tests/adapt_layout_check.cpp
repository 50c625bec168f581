// Host check of adaptive_block_kernel's arrays (adapt_arrays_bytes, adapt_rounds; csrc/cpd_model.h):
// for every widest detector of a pass, every narrower one and pass lengths around each limit, a
// row's arrays stay within the pass's bytes, and a row is never left without a round.
// prints: cases <n> outside <arrays larger than the pass's> empty <rows without a round>
//         shorter <widest detectors whose own rows decide fewer rounds than the bytes hold>
#include <cstdio>
#include <initializer_list>

#include "cpd_model.h"

using namespace cpd;

int main()
{
    long n = 0, outside = 0, empty = 0, shorter = 0;
    for (uint32_t rounds : {1u, 2u, 15u, 16u, 17u, 63u, 64u, 65u, 79u, 80u, 128u, 208u, 240u, 255u, 256u, 257u, 131072u})
        for (uint32_t max_B = 1; max_B <= CPD_MAX_BINS; max_B++) {
            const uint32_t bytes = adapt_arrays_bytes(max_B, rounds);
            for (uint32_t B = 1; B <= max_B; B++) {
                const uint32_t r = adapt_rounds(B, bytes);
                n++;
                outside += 16ull * B + (uint64_t)r * adapt_stride(B) > bytes;
                empty += r == 0u;
            }
            const uint32_t own = adapt_rounds(max_B, bytes);
            shorter += own < (rounds < 64u ? rounds : 64u) || own > kAdaptRounds;
        }
    std::printf("cases %ld outside %ld empty %ld shorter %ld\n", n, outside, empty, shorter);
    return 0;
}
