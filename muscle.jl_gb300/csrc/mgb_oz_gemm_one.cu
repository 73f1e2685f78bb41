// The emulated GEMM of one contraction.
#include <algorithm>

#include "mgb_oz_gemm.h"

namespace mgb {

// A single contraction: its job in the parameter space (the tensor maps
// must lie in param, const or global memory for TMA).
template <int S, bool EXACT, bool CX>
__global__ void __launch_bounds__(oz_threads(false), 1) k_oz_gemm(const __grid_constant__ OzJob job) {
    oz_gemm_body<S, EXACT, CX, false>(OzOneJob{&job});
}

template <int S, bool EXACT, bool CX>
static int launch_gemm_t(const OzJob &job, int64_t units, cudaStream_t s) {
    auto kern = k_oz_gemm<S, EXACT, CX>;
    constexpr int smem = oz_smem_bytes(S, EXACT);
    static std::atomic<bool> attr_set[OZ_MAX_DEVICES];
    if (int st = set_smem_attr(kern, smem, attr_set)) return st;
    const unsigned grid = (unsigned)std::min<int64_t>(units, sm_count());
    kern<<<grid, oz_threads(false), smem, s>>>(job);
    MGB_CUDA_CHECK(cudaGetLastError());
    return MGB_OK;
}

int oz_launch_one(int S, bool exact, bool cx, const OzJob &job, int64_t units, cudaStream_t s) {
#define OZ_ONE(SS, EX, CC) launch_gemm_t<SS, EX, CC>(job, units, s)
    OZ_DISPATCH(OZ_ONE)
#undef OZ_ONE
}

}  // namespace mgb
