// How long a CTA of the cooperative SVD waits for another one, in clock64 cycles.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define MGB_HD __host__ __device__ __forceinline__
#else
#define MGB_HD inline
#endif

namespace mgb {

// Upper estimate of a round of `spc` pairs of columns of M + N elements: an SM
// retires two FP64 operations per clock, which is 14 cycles per element of a
// ComplexF64 pair for the inner products and the rotation (12 .. 14.4 measured
// from 2^18 x 256 to 2^24 x 3, everything included).
MGB_HD int64_t svd_round_cycles(int64_t M, int64_t N, int64_t spc) { return 16 * spc * (M + N); }
// Waiting for a neighbour, which may be a round behind: `floor` (about a second)
// and sixteen rounds.
MGB_HD int64_t svd_wait_round(int64_t floor, int64_t M, int64_t N, int64_t spc) {
    return floor + 16 * svd_round_cycles(M, N, spc);
}
// Waiting at the end of a sweep for `ctas` CTAs, the farthest of which may be as
// many rounds behind.
MGB_HD int64_t svd_wait_sweep(int64_t floor, int64_t M, int64_t N, int64_t spc, int64_t ctas) {
    return floor + (16 + 2 * ctas) * svd_round_cycles(M, N, spc);
}

}  // namespace mgb
