// The emulated GEMM of one contraction in wide tiles (128 x 64), of a fixed
// slice count or one that the device chose.
#include <algorithm>

#include "mgb_oz_gemm.h"

namespace mgb {

template <bool CX>
__global__ void __launch_bounds__(oz_threads(true), 1) k_oz_gemm_wide(const __grid_constant__ OzAnyJob job) {
    const int S = job.a.sel ? *job.a.sel : job.S;
    if (S == 0 || !(job.cand & (1u << S))) return;  // narrow tiles, or the plain form
    switch (S) {
    case 3: oz_gemm_body<3, true, CX, true>(OzChosenJob<3>{&job}); return;
    case 6: oz_gemm_body<6, true, CX, true>(OzChosenJob<6>{&job}); return;
    }
}

template <bool CX>
static int launch_wide_t(const OzAnyJob &job, int64_t units, cudaStream_t s) {
    auto kern = k_oz_gemm_wide<CX>;
    int smem = 0;
    for (int S = 3; S <= 8; ++S)
        if (oz_wide(S)) smem = std::max(smem, oz_smem_bytes(S, true, true));
    static std::atomic<bool> attr_set[OZ_MAX_DEVICES];
    if (int st = set_smem_attr(kern, smem, attr_set)) return st;
    const unsigned grid = (unsigned)std::min<int64_t>(units, sm_count());
    kern<<<grid, oz_threads(true), smem, s>>>(job);
    MGB_CUDA_CHECK(cudaGetLastError());
    return MGB_OK;
}

int oz_launch_wide(bool cx, const OzAnyJob &job, int64_t units, cudaStream_t s) {
    return cx ? launch_wide_t<true>(job, units, s) : launch_wide_t<false>(job, units, s);
}

}  // namespace mgb
