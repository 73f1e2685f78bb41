// The emulated GEMM of one adaptive contraction: the slice count is read on
// the device.
#include <algorithm>

#include "mgb_oz_gemm.h"

namespace mgb {

// One launch for every slice count: a launch per candidate, of which all but
// one returned at once, cost 3 us each on the device and as much on the host
// (four of them for a tolerance of 1e-13). The body of every count is the one
// of the fixed kernels; registers and shared memory are the largest of them,
// which the one CTA per SM has anyway.
template <bool CX>
__global__ void __launch_bounds__(oz_threads(false), 1) k_oz_gemm_any(const __grid_constant__ OzAnyJob job) {
    const int S = *job.a.sel;
    if (S == 0 || !(job.cand & (1u << S))) return;  // the plain form
    switch (S) {
    case 3: oz_gemm_body<3, true, CX, false>(OzChosenJob<3>{&job}); return;
    case 4: oz_gemm_body<4, true, CX, false>(OzChosenJob<4>{&job}); return;
    case 5: oz_gemm_body<5, true, CX, false>(OzChosenJob<5>{&job}); return;
    case 6: oz_gemm_body<6, true, CX, false>(OzChosenJob<6>{&job}); return;
    case 7: oz_gemm_body<7, true, CX, false>(OzChosenJob<7>{&job}); return;
    case 8: oz_gemm_body<8, true, CX, false>(OzChosenJob<8>{&job}); return;
    }
}
static_assert(sizeof(OzAnyJob) <= 4096, "kernel parameters");

template <bool CX>
static int launch_any_t(const OzAnyJob &job, int64_t units, cudaStream_t s) {
    auto kern = k_oz_gemm_any<CX>;
    int smem = 0;
    for (int S = 3; S <= 8; ++S) smem = std::max(smem, oz_smem_bytes(S, true));
    static std::atomic<bool> attr_set[OZ_MAX_DEVICES];
    if (int st = set_smem_attr(kern, smem, attr_set)) return st;
    const unsigned grid = (unsigned)std::min<int64_t>(units, sm_count());
    kern<<<grid, oz_threads(false), smem, s>>>(job);
    MGB_CUDA_CHECK(cudaGetLastError());
    return MGB_OK;
}

int oz_launch_any(bool cx, const OzAnyJob &job, int64_t units, cudaStream_t s) {
    return cx ? launch_any_t<true>(job, units, s) : launch_any_t<false>(job, units, s);
}

}  // namespace mgb
