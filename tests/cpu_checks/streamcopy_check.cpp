// fill_chunk against byte loops, for sizes and addresses around the streaming loop's blocks.  Built as it is, and with
// NOT_X86 as on a host that is not x86-64 (then without immintrin.h, too).
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <vector>

#ifdef NOT_X86
#undef __x86_64__
#endif
#include "../../comet_b200/csrc/streamcopy.cuh"

int main()
{
#if defined(NOT_X86) && defined(_IMMINTRIN_H_INCLUDED)
    printf("immintrin.h is included\n");
    return 1;
#endif
    std::vector<unsigned char> src(1 << 16), dst(1 << 16);
    for (size_t i = 0; i < src.size(); i++) src[i] = (unsigned char)(i * 131 + (i >> 8));
    for (size_t n : {0, 1, 31, 32, 33, 127, 128, 129, 255, 256, 1000, 4097})
        for (size_t off : {0, 1, 8, 31})
            for (size_t rows : {1, 3})
                for (size_t pitch : {n, n + 8}) {
                    memset(dst.data(), 0xee, dst.size());
                    cb200::fill_chunk((char *)dst.data() + 64 + off, (const char *)src.data() + 3 * off, pitch, n, rows);
                    for (size_t i = 0; i < dst.size(); i++) {
                        const size_t at = i - 64 - off, r = n ? at / n : rows;
                        const unsigned char want = i >= 64 + off && r < rows ? src[3 * off + r * pitch + at % n] : 0xee;
                        if (dst[i] != want) {
                            printf("n %zu offset %zu rows %zu pitch %zu: byte %zu\n", n, off, rows, pitch, i);
                            return 1;
                        }
                    }
                }
    printf("ok\n");
    return 0;
}
