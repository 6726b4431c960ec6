// Copies into page-locked chunks.  Plain C++ for the host; the streaming form is for x86-64 and memcpy does elsewhere (B200s
// come with Arm hosts too).
#pragma once
#include <stddef.h>
#include <stdint.h>
#include <string.h>

#if defined(__x86_64__)
#include <immintrin.h>
#endif

namespace cb200 {

#if defined(__x86_64__)
// Into a chunk that the DMA engine reads next: with streaming stores the bytes go to memory; left modified in the
// caches of the cores that copied them, each line is first fetched from there (4.5 MB: 400 us of DMA instead of 90).
__attribute__((target("avx2"))) static inline void copy_streaming(char *dst, const char *src, size_t n)
{
    while (n && ((uintptr_t)dst & 31)) { *dst++ = *src++; n--; }
    for (; n >= 128; n -= 128, src += 128, dst += 128) {
        const __m256i a = _mm256_loadu_si256((const __m256i *)src), b = _mm256_loadu_si256((const __m256i *)(src + 32));
        const __m256i c = _mm256_loadu_si256((const __m256i *)(src + 64)), d = _mm256_loadu_si256((const __m256i *)(src + 96));
        _mm256_stream_si256((__m256i *)dst, a);
        _mm256_stream_si256((__m256i *)(dst + 32), b);
        _mm256_stream_si256((__m256i *)(dst + 64), c);
        _mm256_stream_si256((__m256i *)(dst + 96), d);
    }
    _mm_sfence();
    memcpy(dst, src, n);
}
#endif

// rows x row_bytes, `spitch` apart in src and packed in dst
static inline void fill_chunk(char *dst, const char *src, size_t spitch, size_t row_bytes, size_t rows)
{
#if defined(__x86_64__)
    static const bool streaming = __builtin_cpu_supports("avx2");
#endif
    if (spitch == row_bytes) { row_bytes *= rows; rows = 1; }
    for (size_t r = 0; r < rows; r++) {
#if defined(__x86_64__)
        if (streaming) {
            copy_streaming(dst + r * row_bytes, src + r * spitch, row_bytes);
            continue;
        }
#endif
        memcpy(dst + r * row_bytes, src + r * spitch, row_bytes);
    }
}

}  // namespace cb200
