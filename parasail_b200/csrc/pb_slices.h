/*
 * pb_slices.h -- how a batch's CIGARs are split into slices. Plain C++, so
 * that it can be tested without a GPU.
 */
#ifndef PARASAIL_B200_PB_SLICES_H
#define PARASAIL_B200_PB_SLICES_H

#include <stdint.h>

/* Residues of a slice. The elements of a pair take up to 4 bytes for each of
 * its residues before they are packed, so a slice needs 256 MB for them and
 * as much again packed, where a whole batch needed 4 and more bytes per
 * residue beside its sequences and steps (3). 150,000 reads of 200 and their
 * windows are one slice. */
static const int64_t CIGAR_SLICE = (int64_t)1 << 26;

/* The end of the slice that starts at pair k0: at most `limit` residues (ooff:
 * ascending offsets of the pairs' rows + columns), one pair at least. */
static inline int cigar_slice_end(const int64_t *ooff, const int *qlen, const int *tlen, int n, int k0, int64_t limit)
{
    int lo = k0 + 1, hi = n;                   /* pairs before lo are in, from hi on out */
    while (lo < hi) {
        const int k = lo + (hi - lo) / 2;
        if (ooff[k] + qlen[k] + tlen[k] - ooff[k0] <= limit) lo = k + 1;
        else hi = k;
    }
    return lo;
}

#endif
