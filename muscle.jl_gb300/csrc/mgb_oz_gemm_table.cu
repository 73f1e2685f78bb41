// The emulated GEMM of a group or a served batch: a table of contractions of
// one kernel variant in one persistent launch.
#include <algorithm>

#include "mgb_oz_gemm.h"

namespace mgb {

// A group: every bucket of one kernel variant in one persistent launch.
template <int S, bool EXACT, bool CX>
__global__ void __launch_bounds__(oz_threads(false), 1)
    k_oz_gemm_grouped(const OzJob *__restrict__ jobs, const int64_t *__restrict__ start, int njobs) {
    oz_gemm_body<S, EXACT, CX, false>(OzJobTable{jobs, start, njobs});
}

template <int S, bool EXACT, bool CX>
static int launch_grouped_t(const OzJob *jobs, const int64_t *start, int njobs, int64_t units, cudaStream_t s) {
    auto kern = k_oz_gemm_grouped<S, EXACT, CX>;
    constexpr int smem = oz_smem_bytes(S, EXACT);
    static std::atomic<bool> attr_set[OZ_MAX_DEVICES];
    if (int st = set_smem_attr(kern, smem, attr_set)) return st;
    const unsigned grid = (unsigned)std::min<int64_t>(units, sm_count());
    kern<<<grid, oz_threads(false), smem, s>>>(jobs, start, njobs);
    MGB_CUDA_CHECK(cudaGetLastError());
    return MGB_OK;
}

int oz_launch_table(int S, bool exact, bool cx, const OzJob *jobs, const int64_t *start, int njobs, int64_t units,
                    cudaStream_t s) {
#define OZ_GRP(SS, EX, CC) launch_grouped_t<SS, EX, CC>(jobs, start, njobs, units, s)
    OZ_DISPATCH(OZ_GRP)
#undef OZ_GRP
}

}  // namespace mgb
