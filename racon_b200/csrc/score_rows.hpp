// When a consensus layer's score rows may be held in 16 bits. Plain C++ so
// that host tests can compile it.
#pragma once

#ifdef __CUDACC__
#define RB_SCORE_HD __host__ __device__ __forceinline__
#else
#define RB_SCORE_HD inline
#endif

namespace rb {

// Scores are kept slanted: H'[i][j] = H[i][j] - j * gap. A gap along the row
// is then free (H'[i][j] = max(T'[i][j], H'[i][j-1])), so the in-row term is
// a plain running maximum, the diagonal step adds s - gap, the vertical step
// gap, and the empty prefix row is 0. Cells of one column compare as before.
//
// The fast form of a layer's DP stores int16 rows and permutes bytes for the
// substitution scores. It needs a gap not above 0, a match not below the
// mismatch, s - gap in a signed byte, and scores of ndp rows and L columns that
// provably fit, as they are and slanted. H lies above gap x (row + column)
// (the all-gap path, which the maximum includes); and each column is taken by
// one diagonal step, which gives at most the larger of match and mismatch, or
// by a gap, which gives at most 0, so H lies below max(match, mismatch, 0) x
// column. H' therefore lies between gap x row and (max(match, mismatch, 0) -
// gap) x column. Scores are whole numbers: rows that fit hold the same in 16
// bits as in 32.
RB_SCORE_HD bool fast_scores(int match, int mismatch, int gap, int ndp, int L) {
    const int hi = match > mismatch ? match : mismatch;
    const long long column = (long long)(hi > 0 ? hi : 0) - gap;
    return gap <= 0 && match >= mismatch && match - gap <= 127 && mismatch - gap >= -128 &&
           ((long long)ndp + L) * -gap <= 32767 && column * L <= 32767;
}

}  // namespace rb
