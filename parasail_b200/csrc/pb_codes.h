/*
 * pb_codes.h -- residue codes against the alphabet, four to a word. Plain
 * C++ too, so that the check can be tested without a GPU.
 */
#ifndef PARASAIL_B200_PB_CODES_H
#define PARASAIL_B200_PB_CODES_H

#include <stdint.h>

#ifdef __CUDACC__
#define PB_CODES_FN __host__ __device__ __forceinline__
#else
#define PB_CODES_FN static inline
#endif

/* The codes of a word that are L (1 to 256) or more: 0x80 in each such byte,
 * 0 in the others. The low seven bits of a byte plus 0x80 - L (0x100 - L for
 * L > 128) reach its top bit exactly where they hold L (L - 128) or more, and
 * no byte carries into the next. */
PB_CODES_FN uint32_t codes_outside(uint32_t codes, int L)
{
    const uint32_t t = (codes & 0x7f7f7f7fu) + 0x01010101u * (uint32_t)(L <= 128 ? 0x80 - L : 0x100 - L);
    return (L <= 128 ? t | codes : t & codes) & 0x80808080u;
}

#endif
