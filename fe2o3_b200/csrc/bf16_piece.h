// Four consecutive bf16 of a row, of which some may lie past its end, for rows at any address (gemm_exact.cu).  Written over
// the loads of a memory, so that a test can run it on the CPU and see every byte that it reads: those of the elements that
// there are and no others, for what lies beside them may belong to somebody else, or to nobody.
#ifndef FE2O3_BF16_PIECE_H
#define FE2O3_BF16_PIECE_H
#include <stdint.h>

#ifdef __CUDACC__
#define FE2O3_PIECE_FN __device__ __forceinline__
#else
#define FE2O3_PIECE_FN inline
#endif

// The piece as it was loaded: two words, or (true) a half, a word and a half, where the row is in the middle of a word.
// They are put together only when they are stored: until then nothing waits for them.
// vec: every row starts on eight bytes, and pieces are whole ones from there.
template <typename Mem>
FE2O3_PIECE_FN bool load_piece(uint32_t (&w)[3], const uint16_t *row, uint32_t first, uint32_t end, bool row_ok, bool vec) {
    if (row_ok && first + 4 <= end) {
        const uint16_t *at = row + first;
        if (vec) {
            Mem::two_words(at, w[0], w[1]);
            return false;
        }
        if (((uintptr_t)at & 2u) == 0) {
            w[0] = Mem::word(at);
            w[1] = Mem::word(at + 2);
            return false;
        }
        w[0] = Mem::half(at);
        w[1] = Mem::word(at + 1);
        w[2] = Mem::half(at + 3);
        return true;
    }
    uint32_t v[4];
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i) v[i] = row_ok && first + i < end ? Mem::half(row + first + i) : 0u;
    w[0] = v[0] | v[1] << 16;
    w[1] = v[2] | v[3] << 16;
    return false;
}

// Its elements, two to a word, the first in the lower half.
FE2O3_PIECE_FN void join_piece(const uint32_t (&w)[3], bool halves, uint32_t &x, uint32_t &y) {
    x = halves ? w[0] | w[1] << 16 : w[0];
    y = halves ? w[1] >> 16 | w[2] << 16 : w[1];
}
#endif
