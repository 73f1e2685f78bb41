// Emulated forms on the 5th-generation tensor cores (tcgen05, sm_103a).
//
// OZAKI (Float64 / ComplexF64 results)
//   Each row m of A and column n of B gets a power-of-two scale from its
//   largest exponent; the scaled value a in [-1, 1] is cut into S signed
//   W-bit digits by round-to-nearest:  a = sum_i s_i 2^(-W i) + r,
//   |s_1| <= 2^W, |s_i| <= 2^(W-1), |r| <= 2^(-W S - 1).  W = 8 for S <= 6
//   and W = 7 for S >= 7: every digit is an integer that Float16 holds exactly,
//   every digit product is exact, and a float32 accumulator stays exact
//   while the sum of the absolute products it receives is <= 2^24.
//   Products s_i t_j with i + j = d share the scale 2^(-W d) and go to one
//   TMEM accumulator per d ("group"); pairs with i + j > S + 1 are dropped
//   (Ozaki scheme I).  Every KC embedded k (KC = 256 for W = 7, 128 for
//   W = 8) the epilogue warps read every group's float32 partial sums (exact
//   integers), convert them to int and add them, shifted left by
//   W (S + 1 - d), into one exact 96-bit integer per output element
//   (|X| < 2^(log2 K + W (S + 1) + 1) < 2^95 for any K below 2^31). X times
//   the row and column scales is rounded to float64 with integer operations
//   only (x96_ldexp_rn): no float64 arithmetic at all, since GB300's FP64
//   pipe retires about two operations per cycle per SM.
//   Group bound per k: max(d + 1, 4) * 2^(2W-2); KC * bound <= 2^24 for
//   d <= 15 (W = 7) and d <= 7 (W = 8), which covers every group of every
//   supported S (d <= S + 1).
//
// BF16X3 (Float32 / ComplexF32 results)
//   x = hi + mid + lo, three bf16 pieces (exact for normal floats); the six
//   products with piece-index sum <= 2 (0-based) are kept. The tensor core
//   accumulates in float32 with truncation, whose bias grows with the number
//   of accumulations, so the products are grouped by piece-index sum like
//   the digit groups (hi*hi alone, then sums 1 and 2), read out every
//   KC = 256 k and summed in registers with Kahan compensation.
//
// Complex operands are embedded as real GEMMs: A_e[m][2k+p] = part_p(A[m,k]),
// B_e[2n+q][2k+p] holds [[Br, -Bi], [Bi, Br]] so that C_e[m][2n+q] is part q
// of C[m,n] (4 real products per complex product, as zgemm's 4M form).
//
// Pipeline per CTA (128 x BN embedded outputs per tile, BN = 32, or 64 for
// BF16X3; a persistent grid of one CTA per SM, each walking the tiles b,
// b + grid, ... of one contraction or of a group's job table):
//   warp 0       TMA producer: one 3-D box per operand per 32-wide k block
//                loads all S slices at once into a 64B-swizzled stage;
//   warp 1       TMEM allocation, then one thread issues, per 16 k, one
//                tcgen05.mma.cta_group::1.kind::f16 per A slice i with
//                M = 128, N = BN (S - i): B slices 0 .. S-1-i lie back to
//                back in the stage and their accumulators (digit groups
//                i .. S-1) lie back to back in TMEM;
//   warp 10      (OZAKI) a second issuing thread: the two take alternate
//                k blocks;
//   warps 2..9   epilogue: tcgen05.ld 32x32b.x16 per group and column half
//                from the bank the MMAs are not writing, then tcgen05.st of
//                zeros into what was read.
// Long contractions with 3 or 6 slices run in 128 x 64 tiles with one bank and
// one issuer (see oz_gemm_body in mgb_oz_gemm.h).
// Every mbarrier wait is bounded; on timeout the CTA records
// MGB_ERR_DEVICE_TIMEOUT in the device status word, drains its copies and
// MMAs, frees TMEM and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <functional>
#include <map>
#include <tuple>
#include <type_traits>
#include <cstring>
#include <cmath>
#include <mutex>
#include <vector>

#include "mgb_internal.h"
#include "mgb_oz_gemm.h"
#include "mgb_ptx.h"

namespace mgb {

// =============================================================================
// Pre-pass 1: largest biased exponent per row of an operand
// =============================================================================
struct OpGeom {
    ModeGroup gr, gk, gl;  // rows, contracted, batch
    const void *const *ptrs;  // per-batch-entry base pointers (grouped execution) or null
    int t;                 // tensor index inside the groups (0 = A, 1 = B)
    int64_t R, K;
    int rows_fast;         // operand's unit-stride mode is a row mode
    int scan_lk;           // exponent scan: log2 of a block's warps along k
    int kvec;              // 16-byte vectors along k are aligned, if the base is
};

__device__ __forceinline__ int bexp(double v) { return (__double2hiint(v) >> 20) & 0x7FF; }
__device__ __forceinline__ int bexp_of(double v) { return bexp(v); }
__device__ __forceinline__ int bexp_of(double2 v) { return max(bexp(v.x), bexp(v.y)); }
// Float32 operands of a Float64 / ComplexF64 contraction (promote_eltype),
// widened exactly
__device__ __forceinline__ int bexp_of(float v) { return bexp((double)v); }
__device__ __forceinline__ int bexp_of(float2 v) { return max(bexp((double)v.x), bexp((double)v.y)); }

// 2^(2 d) as a float (0 below 2^-126)
__device__ __forceinline__ float pow4f(int d) { return d >= -63 ? __int_as_float((127 + 2 * d) << 23) : 0.f; }
// |x|^2 4^-(t - 1023), from the exponent and the top of the mantissa, for an
// element whose biased exponent is at most t (zero, subnormal and non-finite
// elements give 0: negligible, or flagged through the exponent table)
__device__ __forceinline__ float sq_tile(double x, int t) {
    const uint32_t h = (uint32_t)__double2hiint(x);
    const int be = (int)((h >> 20) & 0x7FF);
    const float f = __uint_as_float(0x3F800000u | (__funnelshift_l((uint32_t)__double2loint(x), h, 3) & 0x7FFFFFu));
    return (be == 0 || be == 0x7FF) ? 0.f : f * f * pow4f(be - t);
}
__device__ __forceinline__ float sq_tile(double2 x, int t) { return sq_tile(x.x, t) + sq_tile(x.y, t); }
__device__ __forceinline__ float sq_tile(float x, int t) { return sq_tile((double)x, t); }
__device__ __forceinline__ float sq_tile(float2 x, int t) { return sq_tile((double)x.x, t) + sq_tile((double)x.y, t); }

// Exponent scan. A warp takes 32 rows x 32 k with one lane per k (rows_fast:
// per row) and four or eight loads in flight, so that one of the two reductions stays
// in registers and the other is one warp instruction (redux) per row (per k).
// A block is 2^(3 - lk) row tiles by 2^lk k tiles of its eight warps (wide in
// k, for the row maxima meet in shared memory before they go to the table).
// The integer ALU bounds it: 69 instructions per Float64 element with shuffles
// and shared-memory column sums, about 25 now.
constexpr int OZ_SCAN_WARPS = 8;
struct ScaleSmem {
    int64_t roff[32 * OZ_SCAN_WARPS], koff[32 * OZ_SCAN_WARPS];
    int red[OZ_SCAN_WARPS][33];
};
__host__ __device__ inline int64_t oz_scan_tiles(int64_t R, int64_t K, int lk) {
    const int64_t rb = 32ll << (3 - lk), kb = 32ll << lk;
    return ((R + rb - 1) / rb) * ((K + kb - 1) / kb);
}
// Warps along k: as many as K fills
static int oz_scan_lk(int64_t K) { return K > 128 ? 3 : K > 64 ? 2 : K > 32 ? 1 : 0; }

// `part` (nullable, adaptive plans): per 32-row tile and k, the tile's largest
// exponent t and the sum of |x|^2 4^-(t - 1023) over its rows, at
// part[(l * ceil(R / 32) + tile) * K + k]. `emax` (nullable): the largest
// exponent of the whole operand.
template <typename T>
__device__ __forceinline__ void oz_scale_tile(const T *__restrict__ X, const OpGeom &g, int32_t *exps,
                                              int32_t *emax, int2 *part, int64_t blk, int64_t l, ScaleSmem &sm) {
    const int lk = g.scan_lk, wk = 1 << lk;
    const int64_t tiles_k = (g.K + (32 << lk) - 1) / (32 << lk);
    const int64_t tr = blk / tiles_k, tk = blk - tr * tiles_k;
    const int64_t R0 = tr * (32 << (3 - lk)), K0 = tk * (32 << lk);
    const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
    if (tid < (32 << (3 - lk))) sm.roff[tid] = (R0 + tid < g.R) ? group_offset(g.gr, g.t, R0 + tid) : 0;
    if (tid < (32 << lk)) sm.koff[tid] = (K0 + tid < g.K) ? group_offset(g.gk, g.t, K0 + tid) : 0;
    const T *Xl = g.ptrs ? (const T *)g.ptrs[l] : X + group_offset(g.gl, g.t, l);
    __syncthreads();
    const int rt = warp >> lk, kt = warp & (wk - 1);  // this warp's tile in the block
    const int64_t r0 = R0 + 32 * rt, k0 = K0 + 32 * kt;
    const int64_t *roff = sm.roff + 32 * rt, *koff = sm.koff + 32 * kt;
    const int nr = (int)min((int64_t)32, g.R - r0), nk = (int)min((int64_t)32, g.K - k0);  // may be <= 0
    int rmax = 0;  // largest exponent of row `lane`
    if (nr > 0 && nk > 0) {
        int t = 0;      // column `lane`: largest exponent
        float q = 0.f;  // and sum of |x|^2 4^-(t - 1023)
        constexpr int U = sizeof(T) == 16 ? 4 : 8;  // loads in flight per lane
        if (g.rows_fast) {
            const T *x = Xl + roff[lane];
#pragma unroll 1
            for (int j0 = 0; j0 < nk; j0 += U) {
                T v[U];
#pragma unroll
                for (int j = 0; j < U; ++j) {
                    memset(&v[j], 0, sizeof(T));
                    if (lane < nr && j0 + j < nk) v[j] = __ldg(x + koff[j0 + j]);
                }
#pragma unroll
                for (int j = 0; j < U; ++j) {
                    const int be = bexp_of(v[j]);
                    rmax = max(rmax, be);
                    if (part) {
                        // the sum over the lanes as an integer: terms are below 8,
                        // so 32 of them stay below 2^32 in units of 2^-23
                        const int tm = __reduce_max_sync(0xffffffffu, be);
                        const uint32_t u = __reduce_add_sync(0xffffffffu, __float2uint_rn(sq_tile(v[j], tm) * 8388608.f));
                        if (lane == j0 + j) {
                            t = tm;
                            q = (float)u * 1.1920928955078125e-7f;
                        }
                    }
                }
            }
        } else {
            const T *x = Xl + koff[lane];
#pragma unroll 1
            for (int j0 = 0; j0 < nr; j0 += U) {
                T v[U];
                int tn = t;
#pragma unroll
                for (int j = 0; j < U; ++j) {
                    memset(&v[j], 0, sizeof(T));
                    if (lane < nk && j0 + j < nr) v[j] = __ldg(x + roff[j0 + j]);
                }
#pragma unroll
                for (int j = 0; j < U; ++j) {
                    const int be = bexp_of(v[j]);
                    tn = max(tn, be);
                    const int m = __reduce_max_sync(0xffffffffu, be);
                    if (lane == j0 + j) rmax = m;
                }
                if (part) {
                    q *= pow4f(t - tn);
#pragma unroll
                    for (int j = 0; j < U; ++j) q += sq_tile(v[j], tn);
                    t = tn;
                }
            }
        }
        if (part && lane < nk) {
            const int64_t R32 = (g.R + 31) / 32;
            part[(l * R32 + r0 / 32) * g.K + k0 + lane] = make_int2(t, __float_as_int(q));
        }
    }
    sm.red[warp][lane] = rmax;
    __syncthreads();
    if (kt == 0 && nr > 0) {
        for (int w = 1; w < wk; ++w) rmax = max(rmax, sm.red[warp + w][lane]);
        if (lane < nr && rmax > 0) atomicMax(exps + l * g.R + r0 + lane, rmax);
        if (emax) {
            const int m = __reduce_max_sync(0xffffffffu, rmax);
            if (lane == 0 && m > 0) atomicMax(emax, m);
        }
    }
}

// Both operands of one contraction (or of one bucket of a group), as the
// pre-pass launches see them. Blocks [0, tiles) of a launch work on op[0],
// the rest on op[1]: one launch per phase instead of one per operand, since a
// small contraction's pre-pass is launches and little else (`only` >= 0: the
// launch covers that operand alone, when their element types differ).
struct PreOperand {
    OpGeom g;
    const void *X;
    int32_t *exps;      // [L][R] (Ozaki)
    int2 *part;         // the exponent scan's partials (adaptive) or null
    uint32_t *out;      // slice planes
    int64_t rows_e;
    int64_t tiles;      // blocks per batch entry of this launch
};
struct OzStats;
struct PrePair {
    PreOperand op[2];
    int32_t *emax;        // [2] largest exponents (adaptive) or null
    int64_t kw;
    const int32_t *sel;   // adaptive choice or null
    int32_t S;            // slice count when `sel` is null
    int32_t ncnt;
    int32_t *cnt;         // counters of split tiles, cleared by the slicing, or null
};
static_assert(sizeof(PrePair) + 16 <= 4096, "kernel parameters");
// The operand of this block, and the block's tile of it.
__device__ __forceinline__ int pre_operand(const PrePair &a, int only, int64_t &blk) {
    blk = blockIdx.x;
    if (only >= 0) return only;
    if (blk < a.op[0].tiles) return 0;
    blk -= a.op[0].tiles;
    return 1;
}

template <typename T>
__global__ void __launch_bounds__(256, 4) k_oz_scale(const __grid_constant__ PrePair a, int only) {
    __shared__ ScaleSmem sm;
    int64_t blk;
    const int o = pre_operand(a, only, blk);
    const PreOperand &p = a.op[o];
    oz_scale_tile<T>((const T *)p.X, p.g, p.exps, a.emax ? a.emax + o : nullptr, p.part, blk, blockIdx.y, sm);
}

// =============================================================================
// Adaptive slice count: operand statistics and the choice
// =============================================================================
// Error model of the OZAKI form with S digits of W bits (u = 2^-(W S)), for
// row scales 2^e_i of A and column scales 2^f_j of B:
//   * each scaled element is represented to within u/2 (round-to-nearest
//     digits), an error of variance u^2/12 per real part: over C this sums to
//     u^2/12 sum_ij (4^e_i |b_j|^2 + 4^f_j |a_i|^2) = u^2/12 (P_A Q_B + P_B Q_A)
//     with P = sum of the squared scales and Q = squared Frobenius norm;
//   * the dropped digit pairs (i + j = S, 0-based) are S - 1 products of
//     digits of at most 2^(W-1) at weight 2^-(W (S+2)): variance at most
//     (S - 1) u^2 / 144 per k per real product, (S - 1) u^2/144 K P_A P_B;
//   * without cancellation, ||C||^2 = sum_k q_A[k] q_B[k] with q_A[k] the
//     squared norm of A's column k and q_B[k] of B's row k.
// Complex products count twice (re and im parts) in the first term and four
// times in the second. A numpy emulation of the digit scheme gave estimate /
// actual error between 1.0 (Gaussian data) and 5 (log-uniform magnitudes over
// 2^-60..2^60) for every slice count. Everything is measured relative to the
// operand's largest exponent, so the sums stay in float range.
struct OzStats {
    int32_t sel;        // chosen slice count, 0 = plain
    int32_t nonfinite;  // an operand holds Inf / NaN
    int32_t emax[2];    // largest biased exponent of A and B
    float est[9];       // estimated error per candidate slice count
    uint32_t blocks;    // blocks of k_oz_stat that are done
    int32_t pad[2];
    // sums over k and batch entries (cleared with the header every call):
    // P_A sum q_B + P_B sum q_A, sum q_A q_B, K P_A P_B
    double acc[3];
    double pad2;
};
static_assert(sizeof(OzStats) == 96, "stats header");



// Statistics of one operand from the exponent scan's partials, once the
// operand's largest exponent is known. Blocks [0, ceil(K / 256)) of batch
// entry l write q[l][k], the squared norm of column k relative to 4^(be_max
// + 1 - 1023); the blocks after them add the rows' squared scales
// 4^(be_i - be_max) to P[l] and flag non-finite rows.
struct StatSmem {
    float red[32];
};
__device__ __forceinline__ void oz_stat_block(const int2 *__restrict__ part, const int32_t *__restrict__ exps,
                                              OzStats *st, int t, float *q, float *P, int64_t R, int64_t K,
                                              int64_t blk, int64_t l, StatSmem &sm) {
    const int be_max = st->emax[t];
    const int64_t nq = (K + 255) / 256, R32 = (R + 31) / 32;
    if (blk < nq) {
        const int64_t k = blk * 256 + threadIdx.x;
        if (k < K) {
            const int2 *p = part + l * R32 * K + k;
            float acc = 0.f;
            for (int64_t tr = 0; tr < R32; ++tr) {
                const int2 v = __ldg(p + tr * K);
                const float x = __int_as_float(v.y);
                if (x != 0.f) acc += x * pow4f(v.x - be_max - 1);
            }
            q[l * K + k] = acc;
        }
        return;
    }
    const int64_t i = (blk - nq) * 256 + threadIdx.x;
    float w = 0.f;
    if (i < R) {
        const int be = exps[l * R + i];
        if (be == 0x7FF) st->nonfinite = 1;
        else if (be > 0) w = pow4f(be - be_max);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) w += __shfl_xor_sync(0xffffffffu, w, d);
    if (threadIdx.x % 32 == 0) sm.red[threadIdx.x / 32] = w;
    __syncthreads();
    if (threadIdx.x == 0) {
        float s2 = 0.f;
        for (int y = 0; y < (int)blockDim.x / 32; ++y) s2 += sm.red[y];
        if (s2 != 0.f) atomicAdd(P + l, s2);
    }
}
__host__ __device__ inline int64_t oz_stat_blocks(int64_t R, int64_t K) { return (K + 255) / 256 + (R + 255) / 256; }

// The sums behind the estimate, spread over the GPU: block b of batch entry
// l (flattened as l * blocks + b) covers OZ_EST_K values of k and adds its
// part of P_A sum q_B + P_B sum q_A and of sum q_A q_B into the header in
// double; the entry's first block adds K P_A P_B.
constexpr int OZ_EST_K = 2048;
__host__ __device__ inline int64_t oz_est_blocks(int64_t K) { return (K + OZ_EST_K - 1) / OZ_EST_K; }
__device__ __forceinline__ void oz_est_block(OzStats *st, const float *__restrict__ qa, const float *__restrict__ qb,
                                             const float *__restrict__ pa, const float *__restrict__ pb, int64_t K,
                                             int64_t blk, int64_t l, double (&red)[2][8]) {
    double sa = 0.0, sb = 0.0, d = 0.0;
    const int64_t k1 = min(K, (blk + 1) * OZ_EST_K);
    for (int64_t k = blk * OZ_EST_K + threadIdx.x; k < k1; k += blockDim.x) {
        const float x = __ldg(qa + l * K + k), y = __ldg(qb + l * K + k);
        sa += x;
        sb += y;
        d += (double)x * y;
    }
    const double Pa = pa[l], Pb = pb[l];
    double tr = Pa * sb + Pb * sa;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        tr += __shfl_xor_sync(0xffffffffu, tr, o);
        d += __shfl_xor_sync(0xffffffffu, d, o);
    }
    const int lane = threadIdx.x % 32, w = threadIdx.x / 32;
    if (lane == 0) {
        red[0][w] = tr;
        red[1][w] = d;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        tr = d = 0.0;
        for (int i = 0; i < (int)blockDim.x / 32; ++i) {
            tr += red[0][i];
            d += red[1][i];
        }
        if (tr != 0.0) atomicAdd(&st->acc[0], tr);
        if (d != 0.0) atomicAdd(&st->acc[1], d);
        if (blk == 0 && Pa * Pb != 0.0) atomicAdd(&st->acc[2], (double)K * Pa * Pb);
    }
}
// One warp: the error estimate of every candidate slice count (bit S of
// `cand`, lane S) from the sums, and the choice, the smallest count within
// `tol`, else 0 (plain).
__device__ __forceinline__ void oz_choose_warp(OzStats *st, double trunc, double den, double drop, uint32_t cand,
                                               double tol, double margin, int cx) {
    const int S = threadIdx.x % 32;
    const bool is = S >= 1 && S <= 8 && (cand & (1u << S));
    double e = 0.0;
    if (is) {
        const double f1 = cx ? 2.0 : 1.0, f2 = cx ? 4.0 : 1.0;
        const int W = S <= 6 ? 8 : 7;
        const double u = __longlong_as_double((long long)(1023 - W * S) << 52);
        const double num = u * u * (f1 / 12.0 * trunc + f2 * (S - 1) / 144.0 * drop);
        if (num == 0.0) e = 0.0;                 // an operand is zero: every form is exact
        else if (den == 0.0) e = INFINITY;       // no overlap the estimate can rest on
        else e = sqrt(num / den) * margin;
    }
    const bool fin = __ldcg(&st->nonfinite) == 0;
    const uint32_t ok = __ballot_sync(0xffffffffu, is && e <= tol && fin);
    if (S <= 8) st->est[S] = is ? (float)e : 0.f;
    if (S == 0) st->sel = ok ? __ffs(ok) - 1 : 0;
}

// Statistics, estimate and choice of one contraction in one launch. Blocks
// [0, ceil(K / 32)) of batch entry l sum the scan's partials of both operands
// over their row tiles (a warp takes every eighth one, so that few k still
// fill the GPU) and add the entry's sum of q_A, of q_B and of q_A q_B; the
// blocks after them add the rows' squared scales to P and flag non-finite
// rows; the block that finishes last chooses.
constexpr int OZ_STAT_K = 32;
struct StatArgs {
    const int2 *part[2];
    const int32_t *exps[2];
    int64_t R[2], K, L;
    OzStats *st;
    float *P[2];   // [L]
    // [L] sums of q: doubles, or floats for K = 1, whose one q per entry is the
    // sum (the area holds one float per entry and k)
    void *Q[2];
    double tol, margin;
    uint32_t cand;
    int32_t cx;
};
__host__ __device__ inline int64_t oz_stat_grid(int64_t R0, int64_t R1, int64_t K) {
    return (K + OZ_STAT_K - 1) / OZ_STAT_K + (R0 + 255) / 256 + (R1 + 255) / 256;
}
__global__ void __launch_bounds__(256) k_oz_stat(const __grid_constant__ StatArgs a) {
    __shared__ float red[2][8][33];
    __shared__ double dred[2][8];
    __shared__ int last;
    const int64_t nq = (a.K + OZ_STAT_K - 1) / OZ_STAT_K, l = blockIdx.y;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    int64_t blk = blockIdx.x;
    if (blk < nq) {
        const int64_t k = blk * OZ_STAT_K + lane;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int64_t R32 = (a.R[t] + 31) / 32;
            const int be_max = a.st->emax[t];
            const int2 *p = a.part[t] + l * R32 * a.K + k;
            float acc = 0.f;
            if (k < a.K)
#pragma unroll 4
                for (int64_t tr = warp; tr < R32; tr += 8) {
                    const int2 v = __ldg(p + tr * a.K);
                    const float x = __int_as_float(v.y);
                    if (x != 0.f) acc += x * pow4f(v.x - be_max - 1);
                }
            red[t][warp][lane] = acc;
        }
        __syncthreads();
        if (warp < 3) {  // the sums of q_A, of q_B, of q_A q_B
            float q[2] = {0.f, 0.f};
#pragma unroll
            for (int y = 0; y < 8; ++y) {
                q[0] += red[0][y][lane];
                q[1] += red[1][y][lane];
            }
            double v = warp == 0 ? (double)q[0] : warp == 1 ? (double)q[1] : (double)q[0] * q[1];
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
            if (lane == 0) {
                if (warp == 2) {
                    if (v != 0.0) atomicAdd(&a.st->acc[1], v);
                } else if (a.K == 1) {
                    ((float *)a.Q[warp])[l] = (float)v;
                } else if (v != 0.0) {
                    atomicAdd((double *)a.Q[warp] + l, v);
                }
            }
        }
    } else {
        blk -= nq;
        const int64_t nr0 = (a.R[0] + 255) / 256;
        const int t = blk >= nr0;
        const int64_t i = (t ? blk - nr0 : blk) * 256 + threadIdx.x;
        float w = 0.f;
        if (i < a.R[t]) {
            const int be = a.exps[t][l * a.R[t] + i];
            if (be == 0x7FF) a.st->nonfinite = 1;
            else if (be > 0) w = pow4f(be - a.st->emax[t]);
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) w += __shfl_xor_sync(0xffffffffu, w, d);
        if (lane == 0) red[0][0][warp] = w;
        __syncthreads();
        if (threadIdx.x == 0) {
            float s2 = 0.f;
            for (int y = 0; y < 8; ++y) s2 += red[0][0][y];
            if (s2 != 0.f) atomicAdd(a.P[t] + l, s2);
        }
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(&a.st->blocks, 1u) + 1u == gridDim.x * gridDim.y;
        __threadfence();
    }
    __syncthreads();
    if (!last) return;
    auto sum_q = [&](int t, int64_t i) {
        return a.K == 1 ? (double)__ldcg((const float *)a.Q[t] + i) : __ldcg((const double *)a.Q[t] + i);
    };
    double tr = 0.0, drop = 0.0;
    for (int64_t i = threadIdx.x; i < a.L; i += blockDim.x) {
        const double Pa = __ldcg(a.P[0] + i), Pb = __ldcg(a.P[1] + i);
        tr += Pa * sum_q(1, i) + Pb * sum_q(0, i);
        drop += (double)a.K * Pa * Pb;
    }
    if (a.L > 1) {
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            tr += __shfl_xor_sync(0xffffffffu, tr, d);
            drop += __shfl_xor_sync(0xffffffffu, drop, d);
        }
        if (lane == 0) {
            dred[0][warp] = tr;
            dred[1][warp] = drop;
        }
        __syncthreads();
        tr = drop = 0.0;
        for (int y = 0; y < 8; ++y) {
            tr += dred[0][y];
            drop += dred[1][y];
        }
    }
    if (warp != 0) return;
    tr = __shfl_sync(0xffffffffu, tr, 0);
    drop = __shfl_sync(0xffffffffu, drop, 0);
    oz_choose_warp(a.st, tr, __ldcg(&a.st->acc[1]), drop, a.cand, a.tol, a.margin, a.cx);
}

// =============================================================================
// Pre-pass 2: slices (OZAKI digits or BF16X3 pieces), permutation fused
// =============================================================================
// Output words (2 x 16 bits) of slice plane s: out[((l*S + s) * rows_e + row) * kw + word].
//   MODE_REAL : row = r,        word w holds k = 2w, 2w+1
//   MODE_CA   : row = r,        word k holds (re, im)           (A side)
//   MODE_CB   : rows 2r, 2r+1,  word k holds (re, -im), (im, re) (B side)
enum { MODE_REAL = 0, MODE_CA = 1, MODE_CB = 2 };

// Signed digits of Q = x 2^(62 - e) truncated to 62 bits, most significant
// first, rounded to nearest (balanced): with B = half a unit of the last digit
// plus 2^(W-1) at every digit position after the first, digit s >= 1 is the
// W-bit window of Q + B at its position minus 2^(W-1), and the leading digit
// is everything above its position (signed). |d_0| <= 2^W, |d_s| <= 2^(W-1),
// and the remainder below the last digit lies in [-1/2, 1/2) units of it: the
// rounding of taking the digits one at a time, with one 64-bit add for all of
// them. 2^62 more makes the leading digit's window d_0 + 2^W, not negative.
__host__ __device__ constexpr uint64_t oz_digit_bias(int S, int W) {
    uint64_t b = (1ull << 62) + (1ull << (62 - W * S - 1));
    for (int s = 1; s < S; ++s) b += 1ull << (62 - W * (s + 1) + W - 1);
    return b;
}
// Q + B for a value of a row whose largest biased exponent is rowc - 1 (rowc
// 10000: a row with Inf or NaN, all of whose digits are zero). The mantissa,
// left-justified by 10, moves right by the distance to the row's exponent plus
// one (subnormal elements have the exponent of the smallest normal one).
__device__ __forceinline__ uint64_t oz_biased(double x, int rowc, uint64_t bias) {
    const uint32_t lo = (uint32_t)__double2loint(x), hi = (uint32_t)__double2hiint(x);
    const int be = (int)((hi >> 20) & 0x7FF);
    const uint32_t mh = (hi & 0xFFFFFu) | (be ? 0x100000u : 0u);
    const uint64_t m = ((uint64_t)__funnelshift_l(lo, mh, 10) << 32) | (lo << 10);
    const uint64_t M = m >> min(rowc - max(be, 1), 63);
    const uint64_t neg = (uint64_t)((int64_t)(int32_t)hi >> 63);
    return (M ^ neg) + (bias | (hi >> 31));  // the bias is even: -M = ~M + 1
}
// Digit s of two biased values as two Float16 (exact: integers up to 256),
// the first in the low half. The windows become the low bits of 1024 + u, from
// which 1024 and the window's offset are subtracted, both at once. For W = 8
// the windows after the first are bytes of the values shifted left by 2 (which
// is what the caller passes for s > 0), so a byte permute gathers both: 3
// instructions per digit pair.
template <int W, int s>
__device__ __forceinline__ uint32_t oz_digit_pair(uint64_t u0, uint64_t u1) {
    uint32_t w;
    constexpr uint32_t off = s == 0 ? 1u << W : 1u << (W - 1);
    if constexpr (s == 0) {
        constexpr int sh = 62 - W - 32;
        w = ((uint32_t)(u0 >> 32) >> sh) | (((uint32_t)(u1 >> 32) >> sh) << 16);
    } else if constexpr (W == 8) {
        constexpr int b = 7 - s;  // byte of the shifted value
        constexpr uint32_t c = b % 4;
        const uint32_t x0 = (uint32_t)(b >= 4 ? u0 >> 32 : u0), x1 = (uint32_t)(b >= 4 ? u1 >> 32 : u1);
        w = __byte_perm(x0, x1, c | (c << 4) | ((4 + c) << 8) | ((4 + c) << 12)) & 0x00FF00FFu;
    } else {
        constexpr int sh = 62 - W * (s + 1);
        w = __byte_perm((uint32_t)(u0 >> sh), (uint32_t)(u1 >> sh), 0x5410) & 0x007F007Fu;
    }
    w |= 0x64006400u;
    const uint32_t k = 0x64006400u + off * 0x00010001u;
    const __half2 d = __hsub2(*reinterpret_cast<const __half2 *>(&w), *reinterpret_cast<const __half2 *>(&k));
    return *reinterpret_cast<const uint32_t *>(&d);
}
// Three bf16 pieces of two floats: x = hi + mid + lo (to ~2^-24 relative).
__device__ __forceinline__ void bf3_pairs(float x0, float x1, uint32_t (&p)[3]) {
#pragma unroll
    for (int s = 0; s < 3; ++s) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(x0, x1);
        p[s] = *reinterpret_cast<const uint32_t *>(&h);
        x0 -= __uint_as_float(p[s] << 16);
        x1 -= __uint_as_float(p[s] & 0xFFFF0000u);
    }
}

template <typename T>
struct OzIn;
template <>
struct OzIn<double> {
    static constexpr bool cx = false;
    __device__ static double re(double v) { return v; }
    __device__ static double im(double) { return 0.0; }
};
template <>
struct OzIn<double2> {
    static constexpr bool cx = true;
    __device__ static double re(double2 v) { return v.x; }
    __device__ static double im(double2 v) { return v.y; }
};
template <>
struct OzIn<float> {
    static constexpr bool cx = false;
    __device__ static float re(float v) { return v; }
    __device__ static float im(float) { return 0.f; }
};
template <>
struct OzIn<float2> {
    static constexpr bool cx = true;
    __device__ static float re(float2 v) { return v.x; }
    __device__ static float im(float2 v) { return v.y; }
};

// A slicer tile: 32 rows by 128 embedded columns (128 k, or 64 complex ones),
// staged in shared memory in 16-byte chunks. A row's chunks are permuted so
// that a thread's own (8 embedded columns, CPT consecutive chunks) and a
// column of rows both spread over the banks.
// Four blocks per SM (64 registers, a few spilled for complex operands): 3.07 ms
// for the pre-pass of a 4.8 GB Float64 operand, 3.22 with three (80 registers)
constexpr int OZ_SLICE_OCC = 4;
__host__ __device__ constexpr int oz_slice_kt(bool cx) { return cx ? 64 : 128; }  // k per tile
template <typename T, bool CX>
struct SliceTile {
    static constexpr int KT = oz_slice_kt(CX);
    static constexpr int PITCH = KT * (int)sizeof(T);           // bytes per row
    static constexpr int EPT = CX ? 4 : 8;                      // elements per thread and row
    static constexpr int CPT = EPT * (int)sizeof(T) / 16;       // their 16-byte chunks
    static constexpr int VE = 16 / (int)sizeof(T);              // elements per chunk
    __device__ static int at(int r, int c) { return r * PITCH + ((c & ~7) | ((c ^ ((c >> 3) & (CPT - 1)) ^ r) & 7)) * 16; }
};
template <typename T, bool CX>
struct SliceSmem {
    alignas(16) unsigned char tile[32 * SliceTile<T, CX>::PITCH];
    int64_t roff[32], koff[SliceTile<T, CX>::KT];
    int rowc[32];
};
static int64_t oz_slice_tiles(bool cx, int64_t R, int64_t K) {
    return ((R + 31) / 32) * ((K + oz_slice_kt(cx) - 1) / oz_slice_kt(cx));
}
// 16-byte vectors of an operand along k: k's fastest mode is contiguous, and
// every vector of it starts on a 16-byte boundary when the base does.
static int oz_kvec(const ModeGroup &gr, const ModeGroup &gk, const ModeGroup &gl, int t, int dtype) {
    const int64_t ve = 16 / elem_bytes(dtype);
    if (gk.n == 0 || gk.str[t][0] != 1 || gk.ext[0] % ve) return 0;
    for (int i = 1; i < gk.n; ++i)
        if (gk.str[t][i] % ve) return 0;
    for (int i = 0; i < gr.n; ++i)
        if (gr.str[t][i] % ve) return 0;
    for (int i = 0; i < gl.n; ++i)
        if (gl.str[t][i] % ve) return 0;
    return 1;
}

// BYTES from global to shared memory; zeros when !in
template <int BYTES>
__device__ __forceinline__ void cp_async_zfill(uint32_t dst, const void *src, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(BYTES), "r"(in ? BYTES : 0)
                 : "memory");
}

// The thread's 8 embedded columns of one row (four pairs) as S planes of 16
// bytes: digits or pieces of consecutive k (MODE_REAL), of (re, im)
// (MODE_CA), or for the two rows (re, -im) and (im, re) (MODE_CB).
template <int MODE>
__device__ __forceinline__ void oz_store_plane(uint32_t *o, int64_t kw, const uint32_t (&w)[4]) {
    if constexpr (MODE == MODE_CB) {
        *reinterpret_cast<uint4 *>(o) =
            make_uint4(w[0] ^ 0x80000000u, w[1] ^ 0x80000000u, w[2] ^ 0x80000000u, w[3] ^ 0x80000000u);
        *reinterpret_cast<uint4 *>(o + kw) =
            make_uint4(__byte_perm(w[0], 0, 0x1032), __byte_perm(w[1], 0, 0x1032), __byte_perm(w[2], 0, 0x1032),
                       __byte_perm(w[3], 0, 0x1032));
    } else {
        *reinterpret_cast<uint4 *>(o) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}
template <int S, typename X, int MODE>
__device__ __forceinline__ void oz_write_digits(const X (&x)[8], int rowc, uint32_t *o, int64_t plane, int64_t kw) {
    constexpr int W = oz_digit_bits(S);
    constexpr uint64_t bias = oz_digit_bias(S, W);
    uint64_t u[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) u[i] = oz_biased((double)x[i], rowc, bias);
    oz_static_for<S>([&](auto sc) {
        constexpr int s = decltype(sc)::value;
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = oz_digit_pair<W, s>(u[2 * i], u[2 * i + 1]);
        oz_store_plane<MODE>(o, kw, w);
        o += plane;
        if constexpr (s == 0 && W == 8) {
#pragma unroll
            for (int i = 0; i < 8; ++i) u[i] <<= 2;
        }
    });
}

// One 32-row tile of an operand: staged through shared memory (coalesced
// reads whichever mode is contiguous, asynchronous, 16 bytes at a time where
// k runs contiguously on 16-byte boundaries), then written as digit (or
// piece) planes [L][S][rows_e][kw] with K contiguous, 16 bytes per thread and
// plane. BF3: float inputs split into bf16 pieces, otherwise Ozaki digits.
// HBM bounds it now: the pre-pass of a 4.8 GB Float64 operand takes 3.07 ms
// (scan and slices; 2.5 at the copy rate) and took 6.65 with a shift, a mask
// and a float add per digit and 4-byte stores (134 instructions per element).
template <typename T, int MODE, bool BF3>
__device__ __forceinline__ void oz_slice_tile(const T *__restrict__ X, const OpGeom &g,
                                              const int32_t *__restrict__ exps, int S,
                                              uint32_t *__restrict__ out, int64_t rows_e, int64_t kw, int64_t blk,
                                              int64_t l, SliceSmem<T, MODE != MODE_REAL> &sm) {
    using ST = SliceTile<T, MODE != MODE_REAL>;
    constexpr int KT = ST::KT, ES = (int)sizeof(T);
    const int64_t tiles_k = (g.K + KT - 1) / KT;
    const int64_t tr = blk / tiles_k, tk = blk - tr * tiles_k;
    const int64_t r0 = tr * 32, k0 = tk * KT;
    const int tid = threadIdx.x;
    if (tid < 32) {
        sm.roff[tid] = (r0 + tid < g.R) ? group_offset(g.gr, g.t, r0 + tid) : 0;
        if (!BF3) {
            const int be = (r0 + tid < g.R) ? exps[l * g.R + r0 + tid] : 0;
            sm.rowc[tid] = be == 0x7FF ? 10000 : be + 1;
        }
    }
    if (tid >= 128 && tid - 128 < KT) sm.koff[tid - 128] = (k0 + tid - 128 < g.K) ? group_offset(g.gk, g.t, k0 + tid - 128) : 0;
    const T *Xl = g.ptrs ? (const T *)g.ptrs[l] : X + group_offset(g.gl, g.t, l);
    __syncthreads();
    const int nr = (int)min((int64_t)32, g.R - r0), nk = (int)min((int64_t)KT, g.K - k0);
    const uint32_t tile = smem_u32(sm.tile);
    if (g.rows_fast) {
        const int r = tid % 32;
        const T *x = Xl + sm.roff[r];
#pragma unroll 8
        for (int k = tid / 32; k < KT; k += 8)
            cp_async_zfill<ES>(tile + ST::at(r, k * ES / 16) + (k * ES) % 16, x + sm.koff[k], r < nr && k < nk);
    } else if (ES < 16 && g.kvec && ((uintptr_t)Xl & 15) == 0) {
        constexpr int NC = KT / ST::VE;
        const int c = tid % NC;
        const T *x = Xl + sm.koff[c * ST::VE];
#pragma unroll
        for (int r = tid / NC; r < 32; r += 256 / NC)
            cp_async_zfill<16>(tile + ST::at(r, c), x + sm.roff[r], r < nr && c * ST::VE < nk);
    } else {
        const int k = tid % KT;
        const T *x = Xl + sm.koff[k];
#pragma unroll 8
        for (int r = tid / KT; r < 32; r += 256 / KT)
            cp_async_zfill<ES>(tile + ST::at(r, k * ES / 16) + (k * ES) % 16, x + sm.roff[r], r < nr && k < nk);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const int64_t plane = rows_e * kw;
    uint32_t *outl = out + l * (int64_t)S * plane;
    const int col = tid % 16;
    const int64_t word = (tk * 128 + 8 * col) / 2;
    if (word >= kw) return;  // kw is a multiple of 4 words: 16 bytes fit or none
#pragma unroll 1
    for (int r = tid / 16; r < nr; r += 16) {
        // 8 embedded columns: components in order
        using F = decltype(OzIn<T>::re(T()));
        F x[8];
        uint4 raw[ST::CPT];
#pragma unroll
        for (int j = 0; j < ST::CPT; ++j)
            raw[j] = *reinterpret_cast<const uint4 *>(sm.tile + ST::at(r, col * ST::CPT + j));
        if constexpr (MODE == MODE_REAL || OzIn<T>::cx) {
            static_assert(sizeof(x) == sizeof(raw), "a thread's chunks");
            memcpy(x, raw, sizeof(x));
        } else {  // a real operand of a complex contraction: zero imaginary parts
            F re[4];
            static_assert(sizeof(re) == sizeof(raw), "a thread's chunks");
            memcpy(re, raw, sizeof(re));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                x[2 * i] = re[i];
                x[2 * i + 1] = F(0);
            }
        }
        uint32_t *o = outl + (MODE == MODE_CB ? 2 : 1) * (r0 + r) * kw + word;
        if constexpr (BF3) {
            uint32_t p[4][3];
#pragma unroll
            for (int i = 0; i < 4; ++i) bf3_pairs((float)x[2 * i], (float)x[2 * i + 1], p[i]);
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                const uint32_t w[4] = {p[0][s], p[1][s], p[2][s], p[3][s]};
                oz_store_plane<MODE>(o + s * plane, kw, w);
            }
        } else {
            const int rowc = sm.rowc[r];
            switch (S) {
            case 3: oz_write_digits<3, F, MODE>(x, rowc, o, plane, kw); break;
            case 4: oz_write_digits<4, F, MODE>(x, rowc, o, plane, kw); break;
            case 5: oz_write_digits<5, F, MODE>(x, rowc, o, plane, kw); break;
            case 6: oz_write_digits<6, F, MODE>(x, rowc, o, plane, kw); break;
            case 7: oz_write_digits<7, F, MODE>(x, rowc, o, plane, kw); break;
            case 8: oz_write_digits<8, F, MODE>(x, rowc, o, plane, kw); break;
            default: break;  // plans hold 3..8
            }
        }
    }
}

// The first block of an operand's slicing clears the `n` counters of the
// contraction's split tiles (null for one of its two operands), which the
// GEMM after it counts with.
__device__ __forceinline__ void oz_clear_counters(int32_t *cnt, int n) {
    if (cnt)
        for (int i = threadIdx.x; i < n; i += blockDim.x) cnt[i] = 0;
}

// Slices of both operands (see PrePair). With an adaptive choice the slice
// count is read from it, and the launch does nothing when it is 0 (plain).
template <typename T, bool CX, bool BF3>
__global__ void __launch_bounds__(256, OZ_SLICE_OCC) k_oz_slice(const __grid_constant__ PrePair a, int only) {
    int S = a.S;
    if (a.sel) {
        S = *a.sel;
        if (S == 0) return;
    }
    if (blockIdx.x == 0 && blockIdx.y == 0) oz_clear_counters(a.cnt, a.ncnt);
    __shared__ SliceSmem<T, CX> sm;
    int64_t blk;
    if (pre_operand(a, only, blk) == 0) {
        const PreOperand &p = a.op[0];
        oz_slice_tile<T, CX ? MODE_CA : MODE_REAL, BF3>((const T *)p.X, p.g, p.exps, S, p.out, p.rows_e, a.kw, blk,
                                                        blockIdx.y, sm);
    } else {
        const PreOperand &p = a.op[1];
        oz_slice_tile<T, CX ? MODE_CB : MODE_REAL, BF3>((const T *)p.X, p.g, p.exps, S, p.out, p.rows_e, a.kw, blk,
                                                        blockIdx.y, sm);
    }
}

// =============================================================================
// Self-test of the bounded waits: one CTA waits on an mbarrier that nothing
// completes, with the production wait routine, and must come back with
// MGB_ERR_DEVICE_TIMEOUT in the status word.
// =============================================================================
__global__ void k_wait_selftest(int32_t *status) {
    __shared__ __align__(8) uint64_t bar;
    __shared__ int abort_flag;
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bar), 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) (void)mbar_wait(smem_u32(&bar), 0, &abort_flag, status);
    __syncthreads();
}

int selftest_wait_timeout(cudaStream_t s) {
    int32_t *status = device_status_ptr();
    if (!status) return fail(MGB_ERR_CUDA, "device status word unavailable");
    k_wait_selftest<<<1, 32, 0, s>>>(status);
    MGB_CUDA_CHECK(cudaGetLastError());
    return MGB_OK;
}

// =============================================================================
// Host side
// =============================================================================
static uint64_t align256(uint64_t x) { return (x + 255) & ~uint64_t(255); }

// |X| <= k_e * 2^(2W) * 2^(W(S-1)) * (1 + small) must stay below 2^95.
static bool oz_fits(int64_t k_e, int S) {
    const int W = oz_digit_bits(S);
    return std::log2((double)std::max<int64_t>(k_e, 1)) + 2 * W + W * (S - 1) + 1 < 94;
}

// Candidate slice counts of an adaptive plan: those whose exact accumulator
// holds K and whose digits could reach the tolerance at all (2^-(W S) within
// 64 tol; the estimate is at least about u for any data).
static uint32_t oz_candidates(int64_t k_e, double tol) {
    uint32_t m = 0;
    for (int S = 3; S <= 8; ++S)
        if (oz_fits(k_e, S) && std::ldexp(1.0, -oz_digit_bits(S) * S) <= 64.0 * tol) m |= 1u << S;
    return m;
}

// A plan's tensor-core tiles are 128 rows of A by oz_bn embedded columns of
// B (complex B embeds two columns per column). When A has few rows and B many
// columns, most of each 128-row tile is empty; C^T = B^T A^T puts the long
// side on the rows. The exact forms give the same digits and the same exact
// sums either way (the kept digit pairs and the adaptive error estimate are
// symmetric in A and B), so only the tile count decides.
void ozaki_orient(ContractionPlan &p) {
    if (p.form == MGB_FORM_PLAIN || p.swapped) return;
    const bool exact = p.form == MGB_FORM_OZAKI, cx = is_complex(p.compute_dtype);
    const int64_t bn = oz_bn(exact ? p.slices : 3, exact);
    auto tiles = [&](int64_t rows, int64_t cols) {
        return ((rows + OZ_BM - 1) / OZ_BM) * (((cx ? 2 : 1) * cols + bn - 1) / bn);
    };
    if (tiles(p.N, p.M) >= tiles(p.M, p.N)) return;
    std::swap(p.a, p.b);
    std::swap(p.gm, p.gn);
    for (ModeGroup *g : {&p.gm, &p.gn, &p.gk, &p.gl})
        for (int i = 0; i < kMaxRank; ++i) std::swap(g->str[0][i], g->str[1][i]);
    std::swap(p.M, p.N);
    std::swap(p.convert_a, p.convert_b);
    std::swap(p.pa, p.pb);
    p.swapped = true;
}

// ---- splitting K ---------------------------------------------------------------
// The tiles of one contraction rarely fill a whole number of waves of the
// persistent grid, and a long contraction of few rows and columns has fewer
// tiles than SMs. The tiles of the last, unfilled wave are therefore cut along
// K into `splits` units each, at most OZ_SPLIT_WAVES waves of them, by the
// number of units for which that wave is shortest under these times (us),
// measured on 1 .. 256 tiles of 4 .. 512 k blocks: a k block 0.6 (0.52 with
// idle SMs, 0.68 without, at S = 6; 1.1 at S = 8) or 0.4 (BF16x3), publishing
// the sums 2, reading those of one unit 0.4, a second wave of units 8 (its
// readout waits for the first's sums to leave). One when none is shorter by
// OZ_SPLIT_GAIN. E.g. one tile of 512 k blocks at S = 6: 279 us whole, 33 in
// 32 units; 100 tiles of 128: 88 whole, 78 in 3 units; 75 tiles of 8: 16.4
// whole, 17.9 in 2 units. The bits of an exact result do not depend on the
// cut.
constexpr int OZ_SPLIT_WAVES = 2;
constexpr double OZ_SPLIT_FIXED = 2.0, OZ_SPLIT_EACH = 0.4, OZ_SPLIT_WAVE = 8.0, OZ_SPLIT_GAIN = 1.0;
constexpr double oz_kb_us(bool exact, bool wide) { return wide ? 1.21 : exact ? 0.6 : 0.4; }
// Wide or narrow tiles (see oz_gemm_body): the faster under these times (us,
// S = 6, every SM busy): a k block 0.69 narrow and 1.21 wide, a launch 8 and
// 25 (the wide readout's code, and the first chunk's MMAs, which nothing
// overlaps), a wave of wide tiles 4 more; wide ones only if they save
// OZ_WIDE_GAIN. Measured wide / narrow for 128 x 64 tiles x k blocks, us:
// 152 x 128 184 / 182, 304 x 64 188 / 170, 608 x 32 192 / 165, 608 x 128
// 662 / 700, 2432 x 64 1340 / 1396, 72 x 4096 (cut in two) 2600 / 3240,
// 8192 x 256 16870 / 18620. With 3 slices wide tiles win a little earlier (152 x
// 128 94 / 98).
// The rule sees shapes only.
constexpr uint32_t kWideCounts = 1u << 3 | 1u << 6;  // as a mask
static_assert(oz_wide(3) && oz_wide(6) && !oz_wide(4) && !oz_wide(5) && !oz_wide(7) && !oz_wide(8), "kWideCounts");
constexpr double OZ_KB_NARROW = 0.69, OZ_LAUNCH_NARROW = 8.0, OZ_LAUNCH_WIDE = 25.0, OZ_WAVE_WIDE = 4.0, OZ_WIDE_GAIN = 0.97;
static uint64_t oz_part_bytes(bool exact, bool wide) {
    return (uint64_t)OZ_BM * oz_bn(exact ? 8 : 3, exact, wide) * (exact ? 12 : 8);
}
// BF16X3 sums round, so their bits depend on where a sum is cut, and that must
// not depend on how the contraction is run: alone, as a member of a group or a
// served batch, with the workspace for parts or without. So the parts of a sum
// (k blocks in each, a multiple of the readout's chunk; 0: one sum) follow from
// one batch entry's tiles and K, by the times above on OZ_SUM_SMS SMs, and a
// tile adds them in the order of k whether its parts are units of their own
// (oz_part_last) or it runs whole. Entries of a wave or more of tiles gain
// little from a cut and have one sum.
constexpr int64_t OZ_SUM_SMS = 152;
static int32_t oz_sum_blocks(const ContractionPlan &p) {
    const int64_t bn = oz_bn(3, false), chunk = oz_chunk(3, false);
    const int64_t tiles = ((p.m_e + OZ_BM - 1) / OZ_BM) * ((p.n_e + bn - 1) / bn), nkb = (p.k_e + OZ_BK - 1) / OZ_BK;
    if (tiles == 0 || tiles >= OZ_SUM_SMS || nkb <= chunk || nkb >= INT32_MAX / 2) return 0;
    const double kb = oz_kb_us(false, false);
    double best = nkb * kb - OZ_SPLIT_GAIN;
    int64_t kbs = 0;
    for (int64_t most = 2; most <= OZ_SPLIT_WAVES * OZ_SUM_SMS / tiles; ++most) {
        const int64_t c = ((nkb + most - 1) / most + chunk - 1) / chunk * chunk, s = (nkb + c - 1) / c;
        const int64_t waves = (tiles * s + OZ_SUM_SMS - 1) / OZ_SUM_SMS;
        const double t = waves * c * kb + (waves - 1) * OZ_SPLIT_WAVE + OZ_SPLIT_FIXED + OZ_SPLIT_EACH * s;
        if (t < best) {
            best = t;
            kbs = s > 1 ? c : 0;
        }
    }
    return (int32_t)kbs;
}
// The plan's tiling with narrow or wide tiles; `units` of its split tiles (0:
// none is split) and the GEMM's time in us under the rule's model.
static OzTiling oz_tiling(const ContractionPlan &p, bool wide, int64_t &units, double &us) {
    const bool exact = p.form == MGB_FORM_OZAKI;
    const int64_t bn = oz_bn(p.slices, exact, wide), sms = sm_count();
    const int64_t tiles = ((p.m_e + OZ_BM - 1) / OZ_BM) * ((p.n_e + bn - 1) / bn) * p.L;
    const int64_t nkb = (p.k_e + OZ_BK - 1) / OZ_BK, tail = tiles % sms;
    const double kb = oz_kb_us(exact, wide);
    OzTiling r;
    r.full = tiles;
    units = 0;
    const double full_kb = exact && !wide ? OZ_KB_NARROW : kb;
    const int64_t whole = tiles / sms;
    us = (wide ? OZ_LAUNCH_WIDE + OZ_WAVE_WIDE * (whole + (tail > 0)) : OZ_LAUNCH_NARROW) + full_kb * (double)(whole * nkb);
    if (tail == 0) return r;
    double best = nkb * kb - OZ_SPLIT_GAIN, last = full_kb * nkb;
    if (!exact) {  // cut into the parts of the sum, or not at all
        if (p.sum_kb == 0) return r;
        const int64_t s = (nkb + p.sum_kb - 1) / p.sum_kb, waves = (tail * s + sms - 1) / sms;
        if (waves > 2 * OZ_SPLIT_WAVES ||
            waves * p.sum_kb * kb + (waves - 1) * OZ_SPLIT_WAVE + OZ_SPLIT_FIXED + OZ_SPLIT_EACH * s >= best)
            return r;
        r.full = tiles - tail;
        r.splits = (int32_t)s;
        r.kbs = p.sum_kb;
        units = tail * s;
        return r;
    }
    for (int64_t s = 2; s <= OZ_SPLIT_WAVES * sms / tail && s <= nkb && nkb < INT32_MAX / 2; ++s) {
        const int64_t kbs = (nkb + s - 1) / s, waves = (tail * s + sms - 1) / sms;
        if ((s - 1) * kbs >= nkb) continue;  // an empty last unit
        const double over = (waves - 1) * OZ_SPLIT_WAVE + OZ_SPLIT_FIXED + OZ_SPLIT_EACH * s;
        const double t = waves * kbs * kb + over;
        if (t < best) {
            best = t;
            last = waves * kbs * full_kb + over;
            r.full = tiles - tail;
            r.splits = (int32_t)s;
            r.kbs = (int32_t)kbs;
        }
    }
    units = r.splits > 1 ? tail * r.splits : 0;
    us += last;
    return r;
}

void ozaki_setup(ContractionPlan &p) {
    bool cx = is_complex(p.compute_dtype);
    if (p.adaptive) {
        const int64_t k_e = cx ? 2 * p.K : p.K;
        p.cand_mask = oz_candidates(k_e, p.tol);
        // the workspace holds the slices of the largest count that fits K, so
        // that a later tolerance never needs more
        p.slices = 0;
        for (int S = 8; S >= 3 && !p.slices; --S)
            if (oz_fits(k_e, S)) p.slices = S;
        if (!p.slices) p.slices = 3;  // K too long for any count: ozaki_setup reports it below
    }
    int S = p.slices;
    p.m_e = p.M;
    p.n_e = cx ? 2 * p.N : p.N;
    p.k_e = cx ? 2 * p.K : p.K;
    p.kpad = (p.k_e + 7) / 8 * 8;
    p.oz_w = oz_digit_bits(S);
    p.oz_kc = p.form == MGB_FORM_OZAKI ? 32 * oz_chunk_blocks(S) : OZ_KC;
    uint64_t off = 0;
    p.ws_a = off;
    off = align256(off + (uint64_t)p.L * S * p.m_e * p.kpad * 2);
    p.ws_b = off;
    off = align256(off + (uint64_t)p.L * S * p.n_e * p.kpad * 2);
    if (p.form == MGB_FORM_OZAKI) {
        p.ws_scale_a = off;
        off = align256(off + (uint64_t)p.L * p.M * 4);
        p.ws_scale_b = off;
        off = align256(off + (uint64_t)p.L * p.N * 4);
        p.oz_R = oz_fits(p.k_e, S) ? 0 : -1;  // -1: K too long for the exact accumulator
        if (p.adaptive) {
            // OzStats, P_A[L], P_B[L], q_A[L][K], q_B[L][K] (cleared every
            // call), then the exponent scan's partials of A and B
            // ([L][ceil(R / 32)][K] pairs, every one written every call)
            p.ws_stat = off;
            off = align256(off + sizeof(OzStats) + 2 * (uint64_t)p.L * 4);
            off = align256(off + 2 * (uint64_t)p.L * p.K * 4);
            off = align256(off + (uint64_t)p.L * ((p.M + 31) / 32) * p.K * 8);
            off = align256(off + (uint64_t)p.L * ((p.N + 31) / 32) * p.K * 8);
        }
    }
    p.ws_min = off;
    // tilings, and room for the split tiles of those that may run
    const bool exact = p.form == MGB_FORM_OZAKI;
    int64_t units[2] = {0, 0};
    double us[2];
    p.sum_kb = exact ? 0 : oz_sum_blocks(p);
    p.tile[0] = oz_tiling(p, false, units[0], us[0]);
    p.wide = false;
    if (exact && (p.adaptive || oz_wide(S))) {
        p.tile[1] = oz_tiling(p, true, units[1], us[1]);
        p.wide = us[1] < us[0] * OZ_WIDE_GAIN;
    }
    uint64_t cnt = 0, part = 0;
    for (int w = 0; w < (p.wide ? 2 : 1); ++w)
        if (units[w]) {
            cnt = std::max(cnt, (uint64_t)(units[w] / p.tile[w].splits) * OZ_EPI_WARPS * 4);
            part = std::max(part, (uint64_t)units[w] * oz_part_bytes(exact, w));
        }
    if (part) {
        p.ws_cnt = off;
        off = align256(off + cnt);
        p.ws_part = off;
        off = align256(off + part);
    }
    p.ws_bytes = off;
}

// Counters of the split tiles (one per tile and epilogue warp).
static int split_counters(const ContractionPlan &p) {
    if (p.ws_bytes == p.ws_min) return 0;
    return (int)((p.ws_part - p.ws_cnt) / 4);  // with the padding between the two areas
}

// Statistics area of an adaptive plan inside the workspace.
struct OzStatArea {
    OzStats *st;
    float *pa, *pb, *qa, *qb;
    int2 *parta, *partb;
};
static OzStatArea stat_area(const ContractionPlan &p, void *ws) {
    OzStatArea a;
    uint8_t *w = (uint8_t *)ws + p.ws_stat;
    a.st = (OzStats *)w;
    a.pa = (float *)(w + sizeof(OzStats));
    a.pb = a.pa + p.L;
    uint64_t off = align256(p.ws_stat + sizeof(OzStats) + 2 * (uint64_t)p.L * 4);
    a.qa = (float *)((uint8_t *)ws + off);
    a.qb = a.qa + p.L * p.K;
    off = align256(off + 2 * (uint64_t)p.L * p.K * 4);
    a.parta = (int2 *)((uint8_t *)ws + off);
    off = align256(off + (uint64_t)p.L * ((p.M + 31) / 32) * p.K * 8);
    a.partb = (int2 *)((uint8_t *)ws + off);
    return a;
}
// Fluctuations of a Frobenius norm over few outputs: a margin on the estimate
// that vanishes for large results.
static double choice_margin(const ContractionPlan &p) {
    return 1.0 + 2.0 / std::sqrt((double)std::max<int64_t>(p.M * p.N * p.L, 1));
}
static uint64_t stat_bytes(const ContractionPlan &p) {
    return align256(align256(sizeof(OzStats) + 2 * (uint64_t)p.L * 4) + 2 * (uint64_t)p.L * p.K * 4);
}

PFN_encodeTiled_t tensor_map_encoder() {
    static PFN_encodeTiled_t fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                             &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_encodeTiled_t)p;
    });
    return fn;
}

static int make_map(CUtensorMap *tm, void *base, int64_t k_e, int64_t rows, int64_t planes,
                    int64_t kpad, int box_rows, int S) {
    PFN_encodeTiled_t enc = tensor_map_encoder();
    if (!enc) return fail(MGB_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
    cuuint64_t dims[3] = {(cuuint64_t)k_e, (cuuint64_t)rows, (cuuint64_t)planes};
    cuuint64_t strides[2] = {(cuuint64_t)kpad * 2, (cuuint64_t)(kpad * 2 * rows)};
    cuuint32_t box[3] = {OZ_BK, (cuuint32_t)box_rows, (cuuint32_t)S};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, base, dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        return fail(MGB_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
    return MGB_OK;
}

static int unit_row_fast(const ModeGroup &gr, const ModeGroup &gk, int t) {
    int64_t sr = gr.n > 0 ? std::llabs(gr.str[t][0]) : INT64_MAX;
    int64_t sk = gk.n > 0 ? std::llabs(gk.str[t][0]) : INT64_MAX;
    return sr <= sk ? 1 : 0;
}

// Calls f with a null pointer of the operand's element type.
template <typename F>
static int by_type(int dtype, F &&f) {
    switch (dtype) {
    case MGB_F64: return f((double *)nullptr);
    case MGB_C64: return f((double2 *)nullptr);
    case MGB_F32: return f((float *)nullptr);
    default: return f((float2 *)nullptr);
    }
}
template <typename P>
using TypeOf = typename std::remove_pointer<P>::type;

// Launches f(type tag, operand) for both operands at once (operand -1) when
// their element types agree, else one by one.
template <typename F>
static int by_operand(const ContractionPlan &p, F &&f) {
    if (p.a.dtype == p.b.dtype) return by_type(p.a.dtype, [&](auto tag) { return f(tag, -1); });
    if (int st = by_type(p.a.dtype, [&](auto tag) { return f(tag, 0); })) return st;
    return by_type(p.b.dtype, [&](auto tag) { return f(tag, 1); });
}

// Pre-pass of the emulated forms into the workspace: exponents, for adaptive
// plans the statistics and the choice (OZAKI), and slices of A and B. One
// launch per phase.
int ozaki_prepass(const ContractionPlan &p, const void *A, const void *B, void *ws, bool split, cudaStream_t s) {
    if (((uintptr_t)ws & 255) != 0) return fail(MGB_ERR_WORKSPACE, "workspace must be 256-byte aligned");
    const bool exact = p.form == MGB_FORM_OZAKI;
    const bool cx = is_complex(p.compute_dtype);
    uint8_t *w = (uint8_t *)ws;
    OzStatArea area = {};
    if (exact && p.adaptive) area = stat_area(p, ws);

    PrePair pre;
    for (int o = 0; o < 2; ++o) {
        PreOperand &q = pre.op[o];
        q.g.gr = o ? p.gn : p.gm;
        q.g.gk = p.gk;
        q.g.gl = p.gl;
        q.g.ptrs = o ? p.pb : p.pa;
        q.g.t = o;
        q.g.R = o ? p.N : p.M;
        q.g.K = p.K;
        q.g.rows_fast = unit_row_fast(q.g.gr, p.gk, o);
        q.X = o ? B : A;
        q.exps = exact ? (int32_t *)(w + (o ? p.ws_scale_b : p.ws_scale_a)) : nullptr;
        q.part = o ? area.partb : area.parta;
        q.out = (uint32_t *)(w + (o ? p.ws_b : p.ws_a));
        q.rows_e = o ? p.n_e : p.m_e;
        q.g.scan_lk = oz_scan_lk(p.K);
        q.g.kvec = oz_kvec(q.g.gr, p.gk, p.gl, o, o ? p.b.dtype : p.a.dtype);
    }
    auto set_tiles = [&](bool scan) -> int {
        for (PreOperand &q : pre.op)
            q.tiles = scan ? oz_scan_tiles(q.g.R, p.K, q.g.scan_lk) : oz_slice_tiles(cx, q.g.R, p.K);
        if (pre.op[0].tiles + pre.op[1].tiles > INT32_MAX)
            return fail(MGB_ERR_UNSUPPORTED, "operand too large for the pre-pass grid");
        return MGB_OK;
    };
    pre.emax = area.st ? area.st->emax : nullptr;
    pre.kw = p.kpad / 2;
    pre.sel = area.st ? &area.st->sel : nullptr;
    pre.S = exact ? p.slices : 3;
    pre.ncnt = split ? split_counters(p) : 0;
    pre.cnt = pre.ncnt ? (int32_t *)(w + p.ws_cnt) : nullptr;
    auto grid = [&](int o) {
        return dim3((unsigned)(o < 0 ? pre.op[0].tiles + pre.op[1].tiles : pre.op[o].tiles), (unsigned)p.L);
    };
    if (exact) {
        // exponents, statistics header and sums: one contiguous area
        uint64_t end = p.ws_scale_b + (uint64_t)p.L * p.N * 4;
        if (p.adaptive)
            end = p.K > 1 ? (uint64_t)((uint8_t *)area.qa - w) + 2 * (uint64_t)p.L * sizeof(double)
                          : (uint64_t)((uint8_t *)(area.pb + p.L) - w);
        MGB_CUDA_CHECK(cudaMemsetAsync(w + p.ws_scale_a, 0, end - p.ws_scale_a, s));
        if (int st = set_tiles(true)) return st;
        int st = by_operand(p, [&](auto tag, int o) -> int {
            k_oz_scale<TypeOf<decltype(tag)>><<<grid(o), 256, 0, s>>>(pre, o);
            MGB_CUDA_CHECK(cudaGetLastError());
            return MGB_OK;
        });
        if (st) return st;
        if (p.adaptive) {
            StatArgs a;
            a.part[0] = area.parta;
            a.part[1] = area.partb;
            a.exps[0] = pre.op[0].exps;
            a.exps[1] = pre.op[1].exps;
            a.R[0] = p.M;
            a.R[1] = p.N;
            a.K = p.K;
            a.L = p.L;
            a.st = area.st;
            a.P[0] = area.pa;
            a.P[1] = area.pb;
            a.Q[0] = area.qa;
            a.Q[1] = p.K > 1 ? (void *)((double *)area.qa + p.L) : (void *)(area.qa + p.L);
            a.tol = p.tol;
            a.margin = choice_margin(p);
            a.cand = p.cand_mask;
            a.cx = cx ? 1 : 0;
            const int64_t blocks = oz_stat_grid(p.M, p.N, p.K);
            if (blocks * p.L > INT32_MAX) return fail(MGB_ERR_UNSUPPORTED, "operand too large for the statistics grid");
            k_oz_stat<<<dim3((unsigned)blocks, (unsigned)p.L), 256, 0, s>>>(a);
            MGB_CUDA_CHECK(cudaGetLastError());
        }
    }
    if (int st = set_tiles(false)) return st;
    return by_operand(p, [&](auto tag, int o) -> int {
        using T = TypeOf<decltype(tag)>;
        if (exact) {
            if (cx) k_oz_slice<T, true, false><<<grid(o), 256, 0, s>>>(pre, o);
            else if constexpr (!OzIn<T>::cx) k_oz_slice<T, false, false><<<grid(o), 256, 0, s>>>(pre, o);
        } else if constexpr (std::is_same<T, float>::value || std::is_same<T, float2>::value) {
            if (cx) k_oz_slice<T, true, true><<<grid(o), 256, 0, s>>>(pre, o);
            else if constexpr (!OzIn<T>::cx) k_oz_slice<T, false, true><<<grid(o), 256, 0, s>>>(pre, o);
        }
        MGB_CUDA_CHECK(cudaGetLastError());
        return MGB_OK;
    });
}

// The GEMM's view of a plan whose slices lie in `ws`. `split`: the workspace
// has room for the sums of split tiles (ws_bytes, not only ws_min).
static int ozaki_shape(const ContractionPlan &p, void *C, void *ws, bool split, bool wide, OzJobShape &job) {
    const bool exact = p.form == MGB_FORM_OZAKI;
    uint8_t *w = (uint8_t *)ws;
    int32_t *status = device_status_ptr();
    if (!status) return fail(MGB_ERR_CUDA, "device status word unavailable");
    const int bn = oz_bn(p.slices, exact, wide);
    const OzTiling &tile = p.tile[wide ? 1 : 0];
    OzGemmArgs &a = job.a;
    a.M = p.M;
    a.Ne = p.n_e;
    a.N = p.N;
    a.nkb = (int32_t)((p.k_e + OZ_BK - 1) / OZ_BK);
    a.expA = exact ? (int32_t *)(w + p.ws_scale_a) : nullptr;
    a.expB = exact ? (int32_t *)(w + p.ws_scale_b) : nullptr;
    a.C = C;
    a.cptr = p.pc;
    a.gm = p.gm;
    a.gn = p.gn;
    a.gl = p.gl;
    a.status = status;
    a.sel = nullptr;
    if (a.gm.n == 0) { a.gm.n = 1; a.gm.ext[0] = 1; for (int t = 0; t < 3; ++t) a.gm.str[t][0] = 0; }
    if (a.gn.n == 0) { a.gn.n = 1; a.gn.ext[0] = 1; for (int t = 0; t < 3; ++t) a.gn.str[t][0] = 0; }
    job.tiles_n = (int32_t)((p.n_e + bn - 1) / bn);
    job.tiles_m = (int32_t)((p.M + OZ_BM - 1) / OZ_BM);
    job.L = (int32_t)p.L;
    if ((p.n_e + bn - 1) / bn > INT32_MAX || (p.M + OZ_BM - 1) / OZ_BM > INT32_MAX || p.L > INT32_MAX)
        return fail(MGB_ERR_UNSUPPORTED, "contraction too large for the tile grid");
    a.full = (int64_t)job.tiles_n * job.tiles_m * job.L;
    a.splits = 1;
    a.kbs = a.nkb;
    a.fold = p.sum_kb / oz_chunk(3, false);
    if (split && tile.splits > 1) {
        a.full = tile.full;
        a.splits = tile.splits;
        a.kbs = tile.kbs;
        a.cnt = (int32_t *)(w + p.ws_cnt);
        a.part = (uint32_t *)(w + p.ws_part);
    }
    return MGB_OK;
}
// The slice tensor maps and the band for S slices.
static int ozaki_maps(const ContractionPlan &p, void *ws, int S, bool wide, CUtensorMap *ta, CUtensorMap *tb,
                      int32_t &band) {
    uint8_t *w = (uint8_t *)ws;
    int st;
    if ((st = make_map(ta, w + p.ws_a, p.k_e, p.m_e, p.L * S, p.kpad, OZ_BM, S))) return st;
    if ((st = make_map(tb, w + p.ws_b, p.k_e, p.n_e, p.L * S, p.kpad, oz_bn(S, p.form == MGB_FORM_OZAKI, wide), S)))
        return st;
    band = p.band;
    if (band <= 0) {
        band = OZ_GROUP_M;
        while (band > 1 && (int64_t)band * OZ_BM * p.kpad * S * 2 > OZ_BAND_BYTES) --band;
    }
    return MGB_OK;
}
// A job of slice count S (0: the plan's), run only when `sel` (nullable) holds S.
// In narrow tiles.
static int ozaki_job(const ContractionPlan &p, void *C, void *ws, bool split, OzJob &job, int S = 0,
                     const int32_t *sel = nullptr) {
    std::memset(&job, 0, sizeof(job));
    if (int st = ozaki_shape(p, C, ws, split, false, job)) return st;
    job.a.sel = sel;
    return ozaki_maps(p, ws, S ? S : p.slices, false, &job.tmA, &job.tmB, job.band);
}

// The units of a launch of several jobs. Each job's cut is the best for it alone;
// beside others that fill the GPU it mostly adds work: publishing a unit's sums
// and adding them up takes 2.4 us: a burst of 600 served ComplexF64 requests of
// one tile and 64 k blocks took 2945 us, each cut for itself, and takes 2384 so
// (200 Float64 ones of 256 k blocks 2798, 2270). All cuts are thinned out by a
// factor f = 1, 2, 4, .. (BF16X3: kept or dropped, its parts are fixed) to the
// shortest launch, in k blocks per SM: the units and their overhead, and half of the
// longest unit for the uneven end, but no less than that unit.
static void ozaki_recut(std::vector<OzJob> &jobs, bool exact) {
    if (jobs.size() < 2) return;
    const double over = (OZ_SPLIT_FIXED + OZ_SPLIT_EACH) / oz_kb_us(exact, false), sms = sm_count();
    struct Cut {
        int32_t splits, kbs;
    };
    auto thin = [](const OzJob &j, int f) {
        Cut c{1, j.a.nkb};
        const int32_t s = (j.a.splits + f - 1) / f;
        if (s > 1) {
            c.kbs = f == 1 ? j.a.kbs : (j.a.nkb + s - 1) / s;
            c.splits = (j.a.nkb + c.kbs - 1) / c.kbs;
        }
        return c;
    };
    int most = 1;
    for (const OzJob &j : jobs) most = std::max(most, j.a.splits);
    if (most == 1) return;
    int best_f = 1;
    double best = 0.0;
    for (int f = 1;; f = exact ? 2 * f : most) {
        double sum = 0.0, longest = 0.0;
        for (const OzJob &j : jobs) {
            const int64_t tiles = (int64_t)j.tiles_n * j.tiles_m * j.L;
            const Cut c = thin(j, f);
            sum += (double)tiles * j.a.nkb;
            if (c.splits > 1) sum += over * (double)(tiles - j.a.full) * c.splits;
            longest = std::max(longest, c.splits > 1 && j.a.full == 0 ? c.kbs + over : (double)j.a.nkb);
        }
        const double t = std::max(longest, sum / sms + 0.5 * longest);
        if (f == 1 || t < best) {
            best = t;
            best_f = f;
        }
        if (f >= most) break;
    }
    if (best_f == 1) return;
    for (OzJob &j : jobs) {
        const Cut c = thin(j, best_f);
        if (c.splits == 1) j.a.full = (int64_t)j.tiles_n * j.tiles_m * j.L;
        j.a.splits = c.splits;
        j.a.kbs = c.kbs;
    }
}

// The job of every slice count in `cand`, of which `sel` (nullable) names the
// one to run; without it cand is one count.
static int ozaki_any_job(const ContractionPlan &p, void *C, void *ws, bool split, bool wide, uint32_t cand,
                         const int32_t *sel, OzAnyJob &job) {
    std::memset(&job, 0, sizeof(job));
    if (int st = ozaki_shape(p, C, ws, split, wide, job)) return st;
    job.a.sel = sel;
    job.cand = cand;
    for (int S = 3; S <= 8; ++S)
        if (cand & (1u << S)) {
            job.S = S;
            if (int st = ozaki_maps(p, ws, S, wide, &job.tm[S - 3][0], &job.tm[S - 3][1], job.band[S - 3])) return st;
        }
    return MGB_OK;
}

int ozaki_gemm(const ContractionPlan &p, const void *A, const void *B, void *C, void *ws, bool split, cudaStream_t s) {
    const bool cx = is_complex(p.compute_dtype);
    OzAnyJob job;
    if (!p.adaptive) {
        if (p.wide) {
            if (int st = ozaki_any_job(p, C, ws, split, true, 1u << p.slices, nullptr, job)) return st;
            return oz_launch_wide(cx, job, job.units(), s);
        }
        OzJob one;
        if (int st = ozaki_job(p, C, ws, split, one)) return st;
        return oz_launch_one(p.slices, p.form == MGB_FORM_OZAKI, cx, one, one.units(), s);
    }
    // The kernels read the chosen count: one launch, or one for the counts
    // that wide tiles hold and one for the others. With none chosen the plain
    // form runs.
    const int32_t *sel = &stat_area(p, ws).st->sel;
    uint32_t narrow = p.cand_mask;
    if (p.wide && (p.cand_mask & kWideCounts)) {
        if (int st = ozaki_any_job(p, C, ws, split, true, p.cand_mask & kWideCounts, sel, job)) return st;
        if (int st = oz_launch_wide(cx, job, job.units(), s)) return st;
        narrow &= ~kWideCounts;
    }
    if (narrow) {
        if (int st = ozaki_any_job(p, C, ws, split, false, narrow, sel, job)) return st;
        if (int st = oz_launch_any(cx, job, job.units(), s)) return st;
    }
    return launch_plain_gemm(p, A, B, C, s, sel);
}

int launch_ozaki(const ContractionPlan &p, const void *A, const void *B, void *C, void *ws,
                 bool split, cudaStream_t s, cudaEvent_t mid) {
    int st = ozaki_prepass(p, A, B, ws, split, s);
    if (st) return st;
    if (mid) MGB_CUDA_CHECK(cudaEventRecord(mid, s));
    return ozaki_gemm(p, A, B, C, ws, split, s);
}

int ozaki_adaptive_report(const ContractionPlan &p, const void *ws, cudaStream_t s, mgb_adaptive_report *out) {
    if (!p.adaptive) return fail(MGB_ERR_ARGUMENT, "adaptive report: the plan has a fixed slice count");
    if (!ws) return fail(MGB_ERR_ARGUMENT, "adaptive report: null workspace");
    OzStats h;
    MGB_CUDA_CHECK(cudaMemcpyAsync(&h, stat_area(p, const_cast<void *>(ws)).st, sizeof(h), cudaMemcpyDeviceToHost, s));
    MGB_CUDA_CHECK(cudaStreamSynchronize(s));
    std::memset(out, 0, sizeof(*out));
    out->slices = h.sel;
    out->nonfinite = h.nonfinite;
    for (int S = 0; S <= 8; ++S) out->estimate[S] = (p.cand_mask & (1u << S)) ? (double)h.est[S] : 0.0;
    out->tolerance = p.tol;
    return MGB_OK;
}

int ozaki_set_tolerance(ContractionPlan &p, double tol) {
    if (!p.adaptive) return fail(MGB_ERR_ARGUMENT, "tolerance: the plan has a fixed slice count");
    if (!(tol > 0.0)) return fail(MGB_ERR_ARGUMENT, "tolerance must be positive");
    p.tol = tol;
    p.cand_mask = oz_candidates(is_complex(p.compute_dtype) ? 2 * p.K : p.K, tol);
    return MGB_OK;
}

// ---- one persistent GEMM launch for several plans of one kernel variant ----
struct OzGrouped {
    int S = 0;
    bool exact = false, cx = false;
    int njobs = 0;
    int64_t tiles = 0;
    OzJob *jobs = nullptr;     // device
    int64_t *start = nullptr;  // device [njobs + 1]
};

int ozaki_grouped_create(const std::vector<const ContractionPlan *> &plans, const std::vector<void *> &ws, int S,
                         bool exact, bool cx, OzGrouped **out) {
    *out = nullptr;
    if (plans.empty()) return fail(MGB_ERR_ARGUMENT, "grouped GEMM: no plans");
    auto *g = new OzGrouped();
    g->S = S;
    g->exact = exact;
    g->cx = cx;
    std::vector<OzJob> host(plans.size());
    std::vector<int64_t> start(plans.size() + 1, 0);
    for (size_t i = 0; i < plans.size(); ++i) {
        const ContractionPlan &p = *plans[i];
        const bool variant_ok = (p.form == MGB_FORM_OZAKI) == exact && is_complex(p.compute_dtype) == cx &&
                                (p.adaptive ? exact && (p.cand_mask & (1u << S)) != 0 : p.slices == S);
        if (!variant_ok) {
            delete g;
            return fail(MGB_ERR_ARGUMENT, "grouped GEMM: plans of different kernel variants");
        }
        // an adaptive plan's job works only when its device choice is S
        const int st = p.adaptive ? ozaki_job(p, nullptr, ws[i], true, host[i], S, &stat_area(p, ws[i]).st->sel)
                                  : ozaki_job(p, nullptr, ws[i], true, host[i]);
        if (st) {
            delete g;
            return st;
        }
    }
    ozaki_recut(host, exact);
    for (size_t i = 0; i < plans.size(); ++i) start[i + 1] = start[i] + host[i].units();
    g->njobs = (int)plans.size();
    g->tiles = start.back();
    cudaError_t e = cudaMalloc((void **)&g->jobs, host.size() * sizeof(OzJob));
    if (e == cudaSuccess) e = cudaMalloc((void **)&g->start, start.size() * sizeof(int64_t));
    if (e == cudaSuccess) e = cudaMemcpy(g->jobs, host.data(), host.size() * sizeof(OzJob), cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaMemcpy(g->start, start.data(), start.size() * sizeof(int64_t), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        ozaki_grouped_destroy(g);
        return cuda_fail(e, "grouped GEMM job table");
    }
    *out = g;
    return MGB_OK;
}

int ozaki_grouped_launch(const OzGrouped *g, cudaStream_t s) {
    if (g->tiles == 0) return MGB_OK;
    return oz_launch_table(g->S, g->exact, g->cx, g->jobs, g->start, g->njobs, g->tiles, s);
}

void ozaki_grouped_destroy(OzGrouped *g) {
    if (!g) return;
    if (g->jobs) cudaFree(g->jobs);
    if (g->start) cudaFree(g->start);
    delete g;
}


// =============================================================================
// Batched execution of many different contractions (the serving form): one
// launch per pre-pass phase over a table of operands, one multi-job chooser,
// and one persistent tensor-core launch per kernel variant over a table of
// (contraction, slice count) jobs.
// =============================================================================
enum { PRE_ZERO = 0, PRE_SCALE = 1, PRE_STAT = 2, PRE_SLICE = 3, PRE_PHASES = 4 };

// One operand of one contraction.
struct PreJob {
    OpGeom g;
    const void *X;
    int32_t dtype;      // the operand's element type
    int32_t mode;       // MODE_REAL / MODE_CA / MODE_CB
    int32_t bf3;        // BF16X3 pieces instead of Ozaki digits
    int32_t S;          // slice count when `sel` is null
    int32_t t;          // 0 = A, 1 = B
    int32_t L;
    int32_t *exps;      // [L][R] (Ozaki)
    int32_t *emax;      // largest exponent of the operand (adaptive) or null
    uint32_t *out;      // slice planes
    int64_t rows_e, kw;
    const int32_t *sel; // adaptive choice of the contraction, or null
    OzStats *st;        // its statistics (adaptive) or null
    float *q, *P;       // this operand's per-k norms and squared scales
    int2 *part;         // the exponent scan's partials of this operand (adaptive) or null
    int32_t *cnt;       // counters of split tiles, cleared by the slicing (A's job) or null
    int32_t ncnt;
    void *zero[2];      // regions cleared by PRE_ZERO (exponents; statistics for t == 0)
    int64_t zero_words[2];
    int64_t tiles[PRE_PHASES];  // blocks of every phase
};

// One adaptive contraction for the multi-job chooser.
struct ChooseJob {
    OzStats *st;
    const float *qa, *qb, *pa, *pb;
    int64_t K, L;
    uint32_t cand;
    int32_t cx;
    double tol, margin;
};

// Clearing and statistics over a table of operand jobs (the scan and the
// slicing have typed launches of their own).
__global__ void __launch_bounds__(256) k_oz_pre_multi(const PreJob *__restrict__ jobs,
                                                         const int64_t *__restrict__ start, int njobs, int phase) {
    __shared__ StatSmem sm;
    const int64_t b = blockIdx.x;
    int lo = 0, hi = njobs - 1;  // the last job whose first block is <= b
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (start[mid] <= b) lo = mid;
        else hi = mid - 1;
    }
    const PreJob &J = jobs[lo];
    const int64_t local = b - start[lo];
    if (phase == PRE_ZERO) {
        for (int r = 0; r < 2; ++r) {  // this job's blocks clear both regions
            int32_t *z = (int32_t *)J.zero[r];
            const int64_t n = J.zero_words[r], nb = J.tiles[PRE_ZERO];
            for (int64_t w = local * blockDim.x + threadIdx.x; w < n; w += nb * blockDim.x) z[w] = 0;
        }
        return;
    }
    const int64_t per_l = J.tiles[phase] / max(J.L, 1);
    const int64_t l = local / per_l, blk = local - l * per_l;
    oz_stat_block(J.part, J.exps, J.st, J.t, J.q, J.P, J.g.R, J.g.K, blk, l, sm);
}

// The last job of a table whose first block is <= b.
__device__ __forceinline__ int multi_job(const int64_t *__restrict__ start, int njobs, int64_t b) {
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (start[mid] <= b) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Exponent scan over a table of operand jobs of one element type: the same
// tile routine, shared memory and occupancy as the single-plan scan, for
// many operands in one launch (no launch per operand, one tail for all).
template <typename T>
__global__ void __launch_bounds__(256, 4) k_oz_scale_multi(const PreJob *__restrict__ jobs,
                                                        const int64_t *__restrict__ start, int njobs) {
    __shared__ ScaleSmem sm;
    const int j = multi_job(start, njobs, blockIdx.x);
    const PreJob &J = jobs[j];
    const int64_t local = blockIdx.x - start[j];
    const int64_t per_l = J.tiles[PRE_SCALE] / max(J.L, 1);
    const int64_t l = local / per_l;
    oz_scale_tile<T>((const T *)J.X, J.g, J.exps, J.emax, J.part, local - l * per_l, l, sm);
}

// Slicing over a table of operand jobs of one element type, embedding and
// form, as the single-plan slicer does it.
template <typename T, int MODE, bool BF3>
__global__ void __launch_bounds__(256, OZ_SLICE_OCC) k_oz_slice_multi(const PreJob *__restrict__ jobs,
                                                        const int64_t *__restrict__ start, int njobs) {
    __shared__ SliceSmem<T, MODE != MODE_REAL> sm;
    const int j = multi_job(start, njobs, blockIdx.x);
    const PreJob &J = jobs[j];
    int S = J.S;
    if (J.sel) {
        S = *J.sel;
        if (S == 0) return;  // the plain form will run this contraction
    }
    const int64_t local = blockIdx.x - start[j];
    if (local == 0) oz_clear_counters(J.cnt, J.ncnt);
    const int64_t per_l = J.tiles[PRE_SLICE] / max(J.L, 1);
    const int64_t l = local / per_l;
    oz_slice_tile<T, MODE, BF3>((const T *)J.X, J.g, J.exps, S, J.out, J.rows_e, J.kw, local - l * per_l, l, sm);
}

// dst[i] = *src[i]: every item's slice count after the choice
__global__ void k_gather_sel(const int32_t *const *__restrict__ src, int32_t *__restrict__ dst, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = *src[i];
}

// The estimate's sums of every adaptive contraction of a batch: job j owns
// blocks [start[j], start[j + 1]) (oz_est_blocks(K) per batch entry).
__global__ void __launch_bounds__(256) k_oz_est_multi(const ChooseJob *__restrict__ jobs,
                                                      const int64_t *__restrict__ start, int njobs) {
    __shared__ double red[2][8];
    const int64_t b = blockIdx.x;
    int lo = 0, hi = njobs - 1;  // the last job whose first block is <= b
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (start[mid] <= b) lo = mid;
        else hi = mid - 1;
    }
    const ChooseJob &c = jobs[lo];
    const int64_t local = b - start[lo], nb = oz_est_blocks(c.K), l = local / nb;
    oz_est_block(c.st, c.qa, c.qb, c.pa, c.pb, c.K, local - l * nb, l, red);
}
// One warp per adaptive contraction: its estimate and choice.
__global__ void k_oz_choose_multi(const ChooseJob *__restrict__ jobs, int njobs) {
    const int j = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
    if (j >= njobs) return;
    const ChooseJob &c = jobs[j];
    oz_choose_warp(c.st, c.st->acc[0], c.st->acc[1], c.st->acc[2], c.cand, c.tol, c.margin, c.cx);
}

struct OzBatchBuffers {
    // device tables and their pinned staging, grown on demand
    uint8_t *dev = nullptr, *host = nullptr;
    size_t cap = 0;
    cudaEvent_t staged = nullptr;  // the last upload has left the staging area
};

OzBatchBuffers *ozaki_batch_buffers_create() { return new OzBatchBuffers(); }

void ozaki_batch_buffers_destroy(OzBatchBuffers *b) {
    if (!b) return;
    if (b->staged) cudaEventSynchronize(b->staged), cudaEventDestroy(b->staged);
    if (b->dev) cudaFree(b->dev);
    if (b->host) cudaFreeHost(b->host);
    delete b;
}

static int batch_reserve(OzBatchBuffers *b, size_t bytes) {
    if (b->staged) MGB_CUDA_CHECK(cudaEventSynchronize(b->staged));  // the previous upload read the staging
    if (bytes <= b->cap) return MGB_OK;
    size_t cap = std::max(bytes, 2 * b->cap);
    if (b->dev) cudaFree(b->dev);
    if (b->host) cudaFreeHost(b->host);
    b->dev = b->host = nullptr;
    b->cap = 0;
    MGB_CUDA_CHECK(cudaMalloc((void **)&b->dev, cap));
    MGB_CUDA_CHECK(cudaMallocHost((void **)&b->host, cap));
    b->cap = cap;
    if (!b->staged) MGB_CUDA_CHECK(cudaEventCreateWithFlags(&b->staged, cudaEventDisableTiming));
    return MGB_OK;
}

static void fill_prejob(PreJob &J, const ContractionPlan &p, int t, const void *X, void *ws, bool split) {
    std::memset(&J, 0, sizeof(J));
    const bool cx = is_complex(p.compute_dtype), exact = p.form == MGB_FORM_OZAKI;
    uint8_t *w = (uint8_t *)ws;
    // one operand, or (X null) the plan's per-batch-entry pointer table
    J.g.ptrs = X ? nullptr : (t == 0 ? p.pa : p.pb);
    J.g.gr = t == 0 ? p.gm : p.gn;
    J.g.gk = p.gk;
    J.g.gl = p.gl;
    J.g.t = t;
    J.g.R = t == 0 ? p.M : p.N;
    J.g.K = p.K;
    J.g.rows_fast = unit_row_fast(J.g.gr, p.gk, t);
    J.g.scan_lk = oz_scan_lk(p.K);
    J.g.kvec = oz_kvec(J.g.gr, p.gk, p.gl, t, t == 0 ? p.a.dtype : p.b.dtype);
    J.X = X;
    J.dtype = t == 0 ? p.a.dtype : p.b.dtype;
    J.mode = cx ? (t == 0 ? MODE_CA : MODE_CB) : MODE_REAL;
    J.bf3 = exact ? 0 : 1;
    J.S = exact ? p.slices : 3;
    J.t = t;
    J.L = (int32_t)p.L;
    J.exps = exact ? (int32_t *)(w + (t == 0 ? p.ws_scale_a : p.ws_scale_b)) : nullptr;
    J.out = (uint32_t *)(w + (t == 0 ? p.ws_a : p.ws_b));
    J.rows_e = t == 0 ? p.m_e : p.n_e;
    J.kw = p.kpad / 2;
    if (t == 0 && split && split_counters(p)) {
        J.cnt = (int32_t *)(w + p.ws_cnt);
        J.ncnt = split_counters(p);
    }
    const int64_t R = J.g.R, K = p.K, L = p.L;
    int64_t zw = 0;
    if (exact) {
        J.zero[0] = J.exps;
        J.zero_words[0] = L * R;
        zw += L * R;
        if (p.adaptive) {
            OzStatArea a = stat_area(p, ws);
            J.sel = &a.st->sel;
            J.st = a.st;
            J.emax = &a.st->emax[t];
            J.q = t == 0 ? a.qa : a.qb;
            J.P = t == 0 ? a.pa : a.pb;
            J.part = t == 0 ? a.parta : a.partb;
            if (t == 0) {
                J.zero[1] = a.st;
                J.zero_words[1] = (int64_t)(stat_bytes(p) / 4);
                zw += J.zero_words[1];
            }
        }
    }
    J.tiles[PRE_ZERO] = zw ? std::min<int64_t>((zw + 1023) / 1024, 64) : 0;
    J.tiles[PRE_SCALE] = exact ? oz_scan_tiles(R, K, J.g.scan_lk) * L : 0;
    J.tiles[PRE_STAT] = (exact && p.adaptive) ? oz_stat_blocks(R, K) * L : 0;
    J.tiles[PRE_SLICE] = oz_slice_tiles(cx, R, K) * L;
}

// The chooser's job for an adaptive plan whose statistics lie in `ws`.
static ChooseJob choose_job(const ContractionPlan &p, void *ws) {
    OzStatArea a = stat_area(p, ws);
    ChooseJob c;
    c.st = a.st;
    c.qa = a.qa;
    c.qb = a.qb;
    c.pa = a.pa;
    c.pb = a.pb;
    c.K = p.K;
    c.L = p.L;
    c.cand = p.cand_mask;
    c.cx = is_complex(p.compute_dtype) ? 1 : 0;
    c.tol = p.tol;
    c.margin = choice_margin(p);
    return c;
}

// Pre-pass tables of emulated items: two operand jobs per item (operands
// given by pointer, or, when null, by the plan's pointer tables), one
// chooser job per adaptive item.
static int pre_tables(const std::vector<OzBatchItem> &items, std::vector<PreJob> &pre, std::vector<ChooseJob> &choose) {
    pre.assign(2 * items.size(), PreJob{});
    choose.clear();
    for (size_t i = 0; i < items.size(); ++i) {
        const OzBatchItem &it = items[i];
        const ContractionPlan &p = *it.p;
        if (p.form == MGB_FORM_PLAIN) return fail(MGB_ERR_ARGUMENT, "batch: plain-form plans are not batched");
        if (((uintptr_t)it.ws & 255) != 0) return fail(MGB_ERR_WORKSPACE, "batch: workspace must be 256-byte aligned");
        fill_prejob(pre[2 * i], p, 0, p.swapped ? it.B : it.A, it.ws, it.split);
        fill_prejob(pre[2 * i + 1], p, 1, p.swapped ? it.A : it.B, it.ws, it.split);
        if (p.adaptive) choose.push_back(choose_job(p, it.ws));
    }
    // operand jobs of one (form, element type, embedding) lie together: the
    // scan and the slicer run one launch per such segment
    std::stable_sort(pre.begin(), pre.end(), [](const PreJob &u, const PreJob &v) {
        return std::make_tuple(u.bf3, u.dtype, u.mode) < std::make_tuple(v.bf3, v.dtype, v.mode);
    });
    return MGB_OK;
}

// Byte offsets of the pre-pass tables in one device area: [pre jobs]
// [block starts of each phase][chooser jobs][their estimate blocks' starts].
struct PreSegment {
    int first = 0, count = 0;  // operand jobs [first, first + count)
    int32_t bf3 = 0, dtype = 0, mode = 0;
    size_t o_scale = 0, o_slice = 0;  // their block starts of the scan and the slicer
    int64_t scale_blocks = 0, slice_blocks = 0;
};
struct PreLayout {
    size_t o_pre = 0, o_pst = 0, o_ch = 0, o_cs = 0, end = 0;
    int64_t blocks[PRE_PHASES] = {};
    int64_t est_blocks = 0;
    std::vector<PreSegment> seg;  // runs of jobs with one (form, element type, embedding)
};
static size_t al256(size_t x) { return (x + 255) & ~size_t(255); }
static PreLayout pre_layout(const std::vector<PreJob> &pre, const std::vector<ChooseJob> &choose, size_t base) {
    PreLayout L;
    size_t off = base;
    L.o_pre = off;
    off = al256(off + pre.size() * sizeof(PreJob));
    L.o_pst = off;
    off = al256(off + PRE_PHASES * (pre.size() + 1) * sizeof(int64_t));
    L.o_ch = off;
    off = al256(off + choose.size() * sizeof(ChooseJob));
    L.o_cs = off;
    off = al256(off + (choose.size() + 1) * sizeof(int64_t));
    for (size_t j = 0; j < pre.size();) {
        PreSegment g;
        g.first = (int)j;
        g.bf3 = pre[j].bf3;
        g.dtype = pre[j].dtype;
        g.mode = pre[j].mode;
        while (j < pre.size() && pre[j].bf3 == g.bf3 && pre[j].dtype == g.dtype && pre[j].mode == g.mode) ++j;
        g.count = (int)j - g.first;
        g.o_scale = off;
        off = al256(off + (g.count + 1) * sizeof(int64_t));
        g.o_slice = off;
        off = al256(off + (g.count + 1) * sizeof(int64_t));
        L.seg.push_back(g);
    }
    L.end = off;
    return L;
}
// Writes the tables at their offsets of host area `h` and fills the block counts.
static void pre_write(PreLayout &L, const std::vector<PreJob> &pre, const std::vector<ChooseJob> &choose, uint8_t *h) {
    std::memcpy(h + L.o_pre, pre.data(), pre.size() * sizeof(PreJob));
    int64_t *pst = (int64_t *)(h + L.o_pst);
    for (int ph = 0; ph < PRE_PHASES; ++ph) {
        int64_t *st = pst + ph * (pre.size() + 1);
        st[0] = 0;
        for (size_t j = 0; j < pre.size(); ++j) st[j + 1] = st[j] + pre[j].tiles[ph];
        L.blocks[ph] = st[pre.size()];
    }
    for (PreSegment &g : L.seg) {
        int64_t *a = (int64_t *)(h + g.o_scale), *b = (int64_t *)(h + g.o_slice);
        a[0] = b[0] = 0;
        for (int j = 0; j < g.count; ++j) {
            a[j + 1] = a[j] + pre[g.first + j].tiles[PRE_SCALE];
            b[j + 1] = b[j] + pre[g.first + j].tiles[PRE_SLICE];
        }
        g.scale_blocks = a[g.count];
        g.slice_blocks = b[g.count];
    }
    std::memcpy(h + L.o_ch, choose.data(), choose.size() * sizeof(ChooseJob));
    int64_t *cst = (int64_t *)(h + L.o_cs);
    cst[0] = 0;
    for (size_t j = 0; j < choose.size(); ++j) cst[j + 1] = cst[j] + oz_est_blocks(choose[j].K) * choose[j].L;
    L.est_blocks = cst[choose.size()];
}
// One typed launch of phase `ph` (scan or slicing) over segment `g`.
static int seg_launch(const PreSegment &g, int ph, const PreJob *dpre, const uint8_t *d, cudaStream_t s) {
    const int64_t blocks = ph == PRE_SCALE ? g.scale_blocks : g.slice_blocks;
    if (blocks == 0) return MGB_OK;
    if (blocks > INT32_MAX) return fail(MGB_ERR_UNSUPPORTED, "batch: pre-pass grid too large");
    const PreJob *jobs = dpre + g.first;
    const int64_t *st = (const int64_t *)(d + (ph == PRE_SCALE ? g.o_scale : g.o_slice));
    const unsigned nb = (unsigned)blocks;
    if (ph == PRE_SCALE) {
        switch (g.dtype) {
        case MGB_F64: k_oz_scale_multi<double><<<nb, 256, 0, s>>>(jobs, st, g.count); break;
        case MGB_C64: k_oz_scale_multi<double2><<<nb, 256, 0, s>>>(jobs, st, g.count); break;
        case MGB_F32: k_oz_scale_multi<float><<<nb, 256, 0, s>>>(jobs, st, g.count); break;
        default: k_oz_scale_multi<float2><<<nb, 256, 0, s>>>(jobs, st, g.count); break;
        }
    } else {
#define MGB_SLICE_MULTI(T, MODE, BF3) k_oz_slice_multi<T, MODE, BF3><<<nb, 256, 0, s>>>(jobs, st, g.count)
        auto by_mode = [&](auto tag, bool bf3) {
            using T = typename std::remove_pointer<decltype(tag)>::type;
            if (bf3) {
                if constexpr (std::is_same<T, float>::value || std::is_same<T, float2>::value) {
                    if (g.mode == MODE_CA) MGB_SLICE_MULTI(T, MODE_CA, true);
                    else if (g.mode == MODE_CB) MGB_SLICE_MULTI(T, MODE_CB, true);
                    else if constexpr (!OzIn<T>::cx) MGB_SLICE_MULTI(T, MODE_REAL, true);
                }
            } else {
                if (g.mode == MODE_CA) MGB_SLICE_MULTI(T, MODE_CA, false);
                else if (g.mode == MODE_CB) MGB_SLICE_MULTI(T, MODE_CB, false);
                else if constexpr (!OzIn<T>::cx) MGB_SLICE_MULTI(T, MODE_REAL, false);
            }
        };
#undef MGB_SLICE_MULTI
        switch (g.dtype) {
        case MGB_F64: by_mode((double *)nullptr, g.bf3 != 0); break;
        case MGB_C64: by_mode((double2 *)nullptr, g.bf3 != 0); break;
        case MGB_F32: by_mode((float *)nullptr, g.bf3 != 0); break;
        default: by_mode((float2 *)nullptr, g.bf3 != 0); break;
        }
    }
    MGB_CUDA_CHECK(cudaGetLastError());
    return MGB_OK;
}

// Every pre-pass phase over the tables at device area `d`: clearing and the
// statistics as one launch each, the scan and the slicing as one typed
// launch per segment, the estimate and the choice before the slicing.
static int pre_launch(const PreLayout &L, size_t npre, size_t nch, const uint8_t *d, cudaStream_t s) {
    const PreJob *dpre = (const PreJob *)(d + L.o_pre);
    for (int ph = 0; ph < PRE_PHASES; ++ph) {
        if (ph == PRE_SLICE && nch > 0) {
            if (L.est_blocks > INT32_MAX) return fail(MGB_ERR_UNSUPPORTED, "batch: estimate grid too large");
            if (L.est_blocks > 0) {
                k_oz_est_multi<<<(unsigned)L.est_blocks, 256, 0, s>>>((const ChooseJob *)(d + L.o_ch),
                                                                      (const int64_t *)(d + L.o_cs), (int)nch);
                MGB_CUDA_CHECK(cudaGetLastError());
            }
            k_oz_choose_multi<<<((int)nch + 3) / 4, 128, 0, s>>>((const ChooseJob *)(d + L.o_ch), (int)nch);
            MGB_CUDA_CHECK(cudaGetLastError());
        }
        if (ph == PRE_SCALE || ph == PRE_SLICE) {
            for (const PreSegment &g : L.seg)
                if (int st = seg_launch(g, ph, dpre, d, s)) return st;
            continue;
        }
        if (L.blocks[ph] == 0) continue;
        if (L.blocks[ph] > INT32_MAX) return fail(MGB_ERR_UNSUPPORTED, "batch: pre-pass grid too large");
        k_oz_pre_multi<<<(unsigned)L.blocks[ph], 256, 0, s>>>(dpre, (const int64_t *)(d + L.o_pst) + ph * (npre + 1),
                                                              (int)npre, ph);
        MGB_CUDA_CHECK(cudaGetLastError());
    }
    return MGB_OK;
}

// The plain-form candidate of an adaptive plan (runs only when the device
// chose no slice count), after its pre-pass into `ws`.
int ozaki_plain_fallback(const ContractionPlan &p, const void *A, const void *B, void *C, void *ws, cudaStream_t s) {
    if (!p.adaptive) return MGB_OK;
    return launch_plain_gemm(p, A, B, C, s, &stat_area(p, ws).st->sel);
}

int ozaki_batch_launch(const std::vector<OzBatchItem> &items, OzBatchBuffers *buf, cudaStream_t s,
                       int32_t *sel_dev_out, const std::function<int()> &after_prepass,
                       const std::function<int(int S, bool exact, bool cx)> &after_variant) {
    const int n = (int)items.size();
    if (n == 0) return MGB_OK;
    int32_t *status = device_status_ptr();
    if (!status) return fail(MGB_ERR_CUDA, "device status word unavailable");
    // ---- host tables
    std::vector<PreJob> pre;
    std::vector<ChooseJob> choose;
    if (int st = pre_tables(items, pre, choose)) return st;
    // GEMM jobs per variant: key (S, exact, cx) ordered cheapest first
    std::map<std::tuple<int, int, int>, std::vector<OzJob>> gem;
    for (int i = 0; i < n; ++i) {
        const OzBatchItem &it = items[i];
        const ContractionPlan &p = *it.p;
        const bool exact = p.form == MGB_FORM_OZAKI, cx = is_complex(p.compute_dtype);
        if (p.adaptive) {
            OzStatArea a = stat_area(p, it.ws);
            for (int S = 3; S <= 8; ++S) {
                if (!(p.cand_mask & (1u << S))) continue;
                OzJob job;
                if (int st = ozaki_job(p, it.C, it.ws, it.split, job, S, &a.st->sel)) return st;
                gem[std::make_tuple(S, 1, cx ? 1 : 0)].push_back(job);
            }
        } else {
            OzJob job;
            if (int st = ozaki_job(p, it.C, it.ws, it.split, job)) return st;
            gem[std::make_tuple(exact ? p.slices : 3, exact ? 1 : 0, cx ? 1 : 0)].push_back(job);
        }
    }
    // longest tiles first in every variant's launch: each CTA ends its walk
    // on short tiles, which even out the CTAs' finishing times
    for (auto &kv : gem) {
        ozaki_recut(kv.second, std::get<1>(kv.first) != 0);
        std::stable_sort(kv.second.begin(), kv.second.end(),
                         [](const OzJob &u, const OzJob &v) { return u.a.nkb > v.a.nkb; });
    }
    // ---- one staging area: [pre-pass tables][per item: fixed slice count,
    //      address of its slice count][per variant: jobs, starts]
    auto al = al256;
    PreLayout PL = pre_layout(pre, choose, 0);
    size_t off = PL.end;
    // per item: the address of its slice count (adaptive: the choice; else
    // the fixed count stored here)
    const size_t o_fix = off;
    off = al(off + n * sizeof(int32_t));
    const size_t o_sp = off;
    off = al(off + n * sizeof(void *));
    std::vector<size_t> o_gj, o_gs;
    for (auto &kv : gem) {
        o_gj.push_back(off);
        off = al(off + kv.second.size() * sizeof(OzJob));
        o_gs.push_back(off);
        off = al(off + (kv.second.size() + 1) * sizeof(int64_t));
    }
    if (int st = batch_reserve(buf, off)) return st;
    uint8_t *h = buf->host, *d = buf->dev;
    pre_write(PL, pre, choose, h);
    for (int i = 0; i < n; ++i) {
        const ContractionPlan &p = *items[i].p;
        ((int32_t *)(h + o_fix))[i] = p.form == MGB_FORM_OZAKI ? p.slices : 3;
        ((const int32_t **)(h + o_sp))[i] =
            p.adaptive ? &stat_area(p, items[i].ws).st->sel : (const int32_t *)(d + o_fix) + i;
    }
    size_t vi = 0;
    std::vector<int64_t> vtiles;
    for (auto &kv : gem) {
        std::memcpy(h + o_gj[vi], kv.second.data(), kv.second.size() * sizeof(OzJob));
        int64_t *st = (int64_t *)(h + o_gs[vi]);
        st[0] = 0;
        for (size_t j = 0; j < kv.second.size(); ++j)
            st[j + 1] = st[j] + kv.second[j].units();
        vtiles.push_back(st[kv.second.size()]);
        ++vi;
    }
    MGB_CUDA_CHECK(cudaMemcpyAsync(d, h, off, cudaMemcpyHostToDevice, s));
    MGB_CUDA_CHECK(cudaEventRecord(buf->staged, s));
    // ---- pre-pass phases
    if (int st = pre_launch(PL, pre.size(), choose.size(), d, s)) return st;
    // every item's slice count (its fixed count, or the device's choice; 0 = plain)
    if (sel_dev_out) {
        k_gather_sel<<<(n + 255) / 256, 256, 0, s>>>((const int32_t *const *)(d + o_sp), sel_dev_out, n);
        MGB_CUDA_CHECK(cudaGetLastError());
    }
    if (after_prepass)
        if (int st = after_prepass()) return st;
    // ---- one persistent launch per kernel variant
    vi = 0;
    for (auto &kv : gem) {
        const int S = std::get<0>(kv.first);
        const bool exact = std::get<1>(kv.first) != 0, cx = std::get<2>(kv.first) != 0;
        if (vtiles[vi] > 0)
            if (int st = oz_launch_table(S, exact, cx, (const OzJob *)(d + o_gj[vi]), (const int64_t *)(d + o_gs[vi]),
                                        (int)kv.second.size(), vtiles[vi], s))
                return st;
        if (after_variant)
            if (int st = after_variant(S, exact, cx)) return st;
        ++vi;
    }
    return MGB_OK;
}
}  // namespace mgb
