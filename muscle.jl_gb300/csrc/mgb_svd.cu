// Thin singular value decomposition on the device, for the factorisation step
// of simple_update (src/Operations/simple_update.jl:56-60), whose host path is
// LinearAlgebra.svd in tensor_svd_thin (src/Operations/tensor_svd.jl:98-125)
// and whose CUDA path is cuTensorNet (:34).
//
// One-sided Jacobi (Hestenes) rotations: the columns of W (A, or A^H when A
// is wide, so that W has at least as many rows as columns) are rotated in
// pairs until every pair is orthogonal to within `tol` relative to their
// norms; V accumulates the rotations. Each sweep visits every pair once, in
// n - 1 rounds of disjoint pairs (the circle method). The singular values are
// the final column norms, with high relative accuracy. They are then sorted
// in descending order, the columns normalised into singular vectors, and the
// left vectors of exactly zero singular values completed to an orthonormal
// set (Gram-Schmidt on unit vectors). Sweeps are bounded (kMaxSweeps), so the
// kernel always ends; the sweep count is reported.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstddef>

#include "mgb_internal.h"
#include "mgb_ptx.h"
#include "mgb_svd_wait.h"

namespace mgb {

constexpr int kSvdThreads = 256;
constexpr int kSvdWarps = kSvdThreads / 32;
constexpr int kMaxSweeps = 60;
constexpr int64_t kSvdMaxCols = 1024;  // min(m, n)

__device__ __forceinline__ double sconj(double x) { return x; }
__device__ __forceinline__ double2 sconj(double2 x) { return make_double2(x.x, -x.y); }
__device__ __forceinline__ double abs2(double x) { return x * x; }
__device__ __forceinline__ double abs2(double2 x) { return x.x * x.x + x.y * x.y; }
__device__ __forceinline__ double smul(double a, double b) { return a * b; }
__device__ __forceinline__ double2 smul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double sadd(double a, double b) { return a + b; }
__device__ __forceinline__ double2 sadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double sscale(double a, double c) { return a * c; }
__device__ __forceinline__ double2 sscale(double2 a, double c) { return make_double2(a.x * c, a.y * c); }
__device__ __forceinline__ double zero_of(double) { return 0.0; }
__device__ __forceinline__ double2 zero_of(double2) { return make_double2(0.0, 0.0); }
__device__ __forceinline__ double one_of(double) { return 1.0; }
__device__ __forceinline__ double2 one_of(double2) { return make_double2(1.0, 0.0); }
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}
__device__ __forceinline__ double2 warp_sum(double2 v) { return make_double2(warp_sum(v.x), warp_sum(v.y)); }
// Position `i` of round `r` in the circle method over nn (even) players:
// player 0 stays, the others rotate.
__device__ __forceinline__ int circle(int i, int r, int nn) { return i == 0 ? 0 : (i - 1 + r) % (nn - 1) + 1; }

// ---- waiting between the CTAs of one cooperative launch ----------------------
constexpr int kSvdMaxCtas = 512;
struct SvdSync {
    int32_t info;                            // sweeps used
    uint32_t abort;                          // a bounded wait gave up
    uint32_t pad[62];
    uint32_t sweep[kMaxSweeps];              // CTAs that ended sweep s, and 2^16 x those that rotated
    uint32_t pad2[4];
    struct alignas(32) {
        uint32_t rounds;                     // rounds that CTA c has completed
    } cta[kSvdMaxCtas];
    double sv[kSvdMaxCols];                  // column norms
    int32_t col_of_rank[kSvdMaxCols];        // columns by descending norm
    double norm2;                            // squared norm of the kept ones
};

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(uint32_t *p, uint32_t v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Bounded wait for (*p & mask) >= v; false when it gave up (after `limit`
// clock64 cycles) or another CTA did.
__device__ __forceinline__ bool svd_wait(const uint32_t *p, uint32_t mask, uint32_t v, long long limit, SvdSync *sy,
                                         int32_t *status) {
    if ((ld_acquire(p) & mask) >= v) return true;
    const long long t0 = clock64();
    for (uint32_t n = 1;; ++n) {
        if ((ld_acquire(p) & mask) >= v) return true;
        if ((n & 255) == 0) {
            if (ld_acquire(&sy->abort)) return false;
            if (clock64() - t0 > limit) {
                st_release(&sy->abort, 1u);
                atomicCAS(status, 0, (int32_t)MGB_ERR_DEVICE_TIMEOUT);
                return false;
            }
        }
    }
}

// ---- scalars of a rotation ----------------------------------------------------
// One FP64 instruction takes a scheduler 54 cycles to issue and 66 to answer
// here, whatever the number of active lanes, and the rotation is a serial
// chain: so it starts from float estimates (MUFU), works on exponents with
// integers, and spends 25 FP64 instructions (3.1 k cycles with rsqrt(),
// sqrt() and divisions, 1.6 k now).
__device__ __forceinline__ float f32_rsqrt(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float f32_rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float f32_sqrt(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ int dexp(double x) { return (__double2hiint(x) >> 20) & 0x7FF; }
// x 2^d; 0 when the result would be subnormal (x finite, no overflow)
__device__ __forceinline__ double dscale(double x, int d) {
    const int e = dexp(x), h = __double2hiint(x) + (d << 20);
    return (e == 0 || e + d <= 0) ? 0.0 : __hiloint2double(h, __double2loint(x));
}
__device__ __forceinline__ double2 dscale(double2 x, int d) { return make_double2(dscale(x.x, d), dscale(x.y, d)); }
__device__ __forceinline__ int dexp_max(double g) { return dexp(g); }
__device__ __forceinline__ int dexp_max(double2 g) { return max(dexp(g.x), dexp(g.y)); }
// x 2^-e as a float, for a normal positive x whose exponent is near e (truncated; 0 below 2^-100)
__device__ __forceinline__ float d2f(double x, int e) {
    const int h = __double2hiint(x), k = ((h >> 20) & 0x7FF) - 1023 - e;
    const uint32_t m = ((uint32_t)(h & 0xFFFFF) << 3) | ((uint32_t)__double2loint(x) >> 29);
    return k < -100 ? 0.f : __uint_as_float(((uint32_t)(k + 127) << 23) | m);
}
// f 2^e exactly, for a normal positive f
__device__ __forceinline__ double f2d(float f, int e) {
    const uint32_t b = __float_as_uint(f);
    return __hiloint2double((int)((b >> 3) + 0x38000000u) + (e << 20), (int)(b << 29));
}
// 1 / sqrt(x) from an estimate y0 with a relative error near 2^-21: one
// third-order Newton (Halley) step, y0 + y0 e (1/2 + 3/8 e) with e = 1 - x y0^2
__device__ __forceinline__ double rsqrt_step(double x, double y0) {
    const double e = fma(-x * y0, y0, 1.0);
    return fma(y0 * e, fma(e, 0.375, 0.5), y0);
}

__device__ __forceinline__ bool nonzero(double x) { return x != 0.0; }
__device__ __forceinline__ bool nonzero(double2 x) { return x.x != 0.0 || x.y != 0.0; }

// The rotation of a pair with squared norms a, b and inner product g =
// w_p^H w_q: [w_p, w_q] <- [w_p, w_q] J, J = [[c, s e], [-s conj(e), c]],
// e = g / |g|, makes w_p^H w_q vanish: t = s / c is the smaller root of
// t^2 + d t - 1 with d = (b - a) / |g|. False when the pair is orthogonal
// already (|g|^2 <= tol2 a b). t has a relative error near 1e-13 (a float
// estimate and one Newton step); c = 1 / sqrt(1 + t^2) makes J unitary for any
// t. This one for norms and inner products anywhere in the range of doubles, and
// however far apart: g, a and b in the product, and the difference are each
// scaled by the power of two that brings them near 1 and the powers kept as
// integers; subnormal ones are multiplied by 2^512 first.
template <typename T>
__device__ __forceinline__ bool rotation_far(double a, double b, T g, double tol2, double &c, T &se, T &sec) {
    int ea = dexp(a), eb = dexp(b), eg = dexp_max(g), be = max(max(ea, eb), eg);
    if (be == 0x7FF || !nonzero(g)) return false;
    if (be < 1500) {
        constexpr double up = 1.3407807929942597e154;  // 2^512
        a *= up;
        b *= up;
        g = sscale(g, up);
        ea = dexp(a), eb = dexp(b), eg = dexp_max(g), be = max(max(ea, eb), eg);
    }
    if (eg == 0) return false;
    g = dscale(g, 1023 - eg);
    const double g2 = abs2(g);  // 1 .. 8
    const int ab = ea + eb - 2 * eg;  // the exponent of a b / |g|^2
    if (ea != 0 && eb != 0 &&
        (ab > 300 || !(g2 > dscale(tol2 * (dscale(a, 1023 - ea) * dscale(b, 1023 - eb)), ab))))
        return false;
    const int ge = dexp(g2), k = (ge - 1023) >> 1;
    const double ig = rsqrt_step(g2, f2d(f32_rsqrt(d2f(g2, 2 * k)), -k));
    double d = (dscale(b, 1023 - be) - dscale(a, 1023 - be)) * ig;  // times 2^(be - eg)
    // beyond 2^30, t is 1 / d to double precision: of d's mantissa, then scaled
    const int e0 = dexp(d), de = e0 - 1023 + be - eg;
    const bool far = e0 != 0 && de > 30;
    d = dscale(d, far ? 1023 - e0 : be - eg);
    const double ad = fabs(d);
    const float df = d2f(ad, 0);
    const float tf = far ? f32_rcp(df) : 2.f * f32_rcp(df + f32_sqrt(fmaf(df, df, 4.f)));
    const float rf = far ? tf : f32_rcp(fmaf(2.f, tf, df));
    const float cf = far ? 1.f : f32_rsqrt(fmaf(tf, tf, 1.f));
    const double t0 = f2d(tf, 0);
    double t = fma(-fma(t0, far ? ad : t0 + ad, -1.0), f2d(rf, 0), t0);
    t = copysign(far ? dscale(t, -de) : t, d);
    c = rsqrt_step(fma(t, t, 1.0), f2d(cf, 0));
    se = sscale(g, c * t * ig);
    sec = sscale(sconj(se), -1.0);
    return true;
}
// The usual case: everything normal and within 2^400 of the largest, by whose
// power of two all is scaled, so that squares stay in range.
template <typename T>
__device__ __forceinline__ bool rotation(double a, double b, T g, double tol2, double &c, T &se, T &sec) {
    const int ea = dexp(a), eb = dexp(b), eg = dexp_max(g), be = max(max(ea, eb), eg), le = min(min(ea, eb), eg);
    if (be == 0x7FF || le < 60 || be - le > 400) return rotation_far<T>(a, b, g, tol2, c, se, sec);
    const int sh = 1023 - be;
    a = dscale(a, sh);
    b = dscale(b, sh);
    g = dscale(g, sh);
    const double g2 = abs2(g);
    if (!(g2 > tol2 * (a * b))) return false;
    const int k = (dexp(g2) - 1023) >> 1;
    const double ig = rsqrt_step(g2, f2d(f32_rsqrt(d2f(g2, 2 * k)), -k));
    const double d = (b - a) * ig, ad = fabs(d);
    // beyond 2^30, t is 1 / d to double precision
    const int de = dexp(d) - 1023;
    const bool far = de > 30;
    const float df = d2f(ad, far ? de : 0);
    const float tf = far ? f32_rcp(df) : 2.f * f32_rcp(df + f32_sqrt(fmaf(df, df, 4.f)));
    const float rf = far ? tf : f32_rcp(fmaf(2.f, tf, df));
    const float cf = far ? 1.f : f32_rsqrt(fmaf(tf, tf, 1.f));
    const double t0 = f2d(tf, far ? -de : 0);
    const double t = copysign(fma(-fma(t0, t0 + ad, -1.0), f2d(rf, far ? -de : 0), t0), d);
    c = rsqrt_step(fma(t, t, 1.0), f2d(cf, 0));
    se = sscale(g, c * t * ig);
    sec = sscale(sconj(se), -1.0);
    return true;
}

// Sums of four values over the warp: every lane gets all four. Two halving
// steps leave each lane one of the four values, three more sum it over the
// lanes that hold the same one: 6 FP64 additions instead of 20.
__device__ __forceinline__ void warp_sum4(double (&v)[4], int lane) {
    const bool h = lane & 16, q = lane & 8;
    const double s0 = h ? v[0] : v[2], s1 = h ? v[1] : v[3];
    double k0 = (h ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, s0, 16);
    double k1 = (h ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, s1, 16);
    double k = (q ? k1 : k0) + __shfl_xor_sync(0xffffffffu, q ? k0 : k1, 8);
#pragma unroll
    for (int d = 4; d > 0; d >>= 1) k += __shfl_xor_sync(0xffffffffu, k, d);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = __shfl_sync(0xffffffffu, k, 8 * i);
}

__device__ __forceinline__ void dot_push(double (&s)[4], double x, double y) {
    s[0] = fma(x, x, s[0]);
    s[1] = fma(y, y, s[1]);
    s[2] = fma(x, y, s[2]);
}
__device__ __forceinline__ void dot_push(double (&s)[4], double2 x, double2 y) {  // conj(x) y
    s[0] = fma(x.x, x.x, fma(x.y, x.y, s[0]));
    s[1] = fma(y.x, y.x, fma(y.y, y.y, s[1]));
    s[2] = fma(x.x, y.x, fma(x.y, y.y, s[2]));
    s[3] = fma(x.x, y.y, fma(-x.y, y.x, s[3]));
}
__device__ __forceinline__ double dot_g(const double (&s)[4], double) { return s[2]; }
__device__ __forceinline__ double2 dot_g(const double (&s)[4], double2) { return make_double2(s[2], s[3]); }
__device__ __forceinline__ double ldcg(const double *p) { return __ldcg(p); }
__device__ __forceinline__ double2 ldcg(const double2 *p) { return __ldcg(p); }

// W: M x N (column-major, M >= N), V: N x N, one cooperative launch.
//
// FP64 work bounds large matrices: an SM retires two FP64 operations per
// clock, so one SM needs 120 ms for a 128 x 128 ComplexF64 matrix and 904 ms
// for 256 x 256 (22 ms here). The pairs of a
// round are independent, so each CTA owns `spc` consecutive pair slots of the
// circle. From one round to the next, a slot's upper column comes from the
// slot after it and its lower column from the slot before it (slot 0 keeps
// column 0 and hands its lower column round), so a CTA waits for its two
// neighbours' round counters only, never for the whole grid; the columns go
// through L2, where every one has exactly one owner in a round. The CTAs meet
// once a sweep, to agree whether any of them rotated.
//
// A slot's columns stay in registers between the inner products and the
// rotation (R elements per thread; longer columns are read again), the four
// sums of a pair take one pass, and one warp computes the rotation.
template <typename T, int R>
__global__ void __launch_bounds__(kSvdThreads) k_svd_jacobi(T *__restrict__ W, int M, int N, T *__restrict__ V,
                                                            double tol2, int spc, SvdSync *sy, int32_t *status) {
    __shared__ double part[kSvdWarps][4];
    __shared__ double rc;
    __shared__ T rse, rsec;
    __shared__ int rdo;
    __shared__ uint32_t agreed;
    const int nn = N + (N & 1), np = nn / 2;
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const int cta = blockIdx.x, nct = gridDim.x;
    const int slot0 = cta * spc, slot1 = min(np, slot0 + spc);
    const int total = M + N;  // a column of W, then its column of V
    uint32_t done = 0;        // rounds completed, over all sweeps
    const long long per_round = svd_wait_round(kWaitTimeoutCycles, M, N, spc);
    const long long per_sweep = svd_wait_sweep(kWaitTimeoutCycles, M, N, spc, nct);
    auto pair = [&](int pi, int r, int &p, int &q) {
        p = circle(pi, r, nn);
        q = circle(nn - 1 - pi, r, nn);
        if (p > q) {
            const int t = p;
            p = q;
            q = t;
        }
    };
    bool ok = true;
    int sweep = 0;
    for (; sweep < kMaxSweeps; ++sweep) {
        bool rotated = false;
        for (int r = 0; r + 1 < nn; ++r, ++done) {
            bool here = true;
            if (tid == 0 && cta > 0) here = svd_wait(&sy->cta[cta - 1].rounds, ~0u, done, per_round, sy, status);
            if (tid == 32 && cta + 1 < nct) here = svd_wait(&sy->cta[cta + 1].rounds, ~0u, done, per_round, sy, status);
            if (!__syncthreads_and(here)) {
                ok = false;
                break;
            }
            for (int pi = slot0; pi < slot1; ++pi) {
                int p, q;
                pair(pi, r, p, q);
                if (q >= N) continue;  // the padding player of an odd N
                T *wp = W + (int64_t)p * M, *wq = W + (int64_t)q * M;
                T *vp = V + (int64_t)p * N - M, *vq = V + (int64_t)q * N - M;
                T x[R], y[R];
                double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
                for (int k = 0; k < R; ++k) {
                    const int i = tid + k * kSvdThreads;
                    if (i < total) {
                        x[k] = ldcg((i < M ? wp : vp) + i);
                        y[k] = ldcg((i < M ? wq : vq) + i);
                    }
                }
#pragma unroll
                for (int k = 0; k < R; ++k)
                    if (tid + k * kSvdThreads < M) dot_push(s, x[k], y[k]);
                for (int i = tid + R * kSvdThreads; i < M; i += kSvdThreads) dot_push(s, ldcg(wp + i), ldcg(wq + i));
                const int nw = min(kSvdWarps, (M + 31) / 32);  // warps that hold part of the sums
                if (warp < nw) {
                    warp_sum4(s, lane);
                    if (lane < 4) part[warp][lane] = lane == 0 ? s[0] : lane == 1 ? s[1] : lane == 2 ? s[2] : s[3];
                }
                __syncthreads();
                if (warp == 0) {
                    // lane 4 w + i: sum i of warp w
                    double v = lane / 4 < nw ? part[lane / 4][lane % 4] : 0.0;
#pragma unroll
                    for (int d = 4; d < 4 * kSvdWarps; d <<= 1)
                        if (d < 4 * nw) v += __shfl_xor_sync(0xffffffffu, v, d);
#pragma unroll
                    for (int i = 0; i < 4; ++i) s[i] = __shfl_sync(0xffffffffu, v, i);
                    double c = 1.0;
                    T se = zero_of(T()), sec = zero_of(T());
                    const bool rot = rotation<T>(s[0], s[1], dot_g(s, T()), tol2, c, se, sec);
                    if (lane == 0) {
                        rc = c;
                        rse = se;
                        rsec = sec;
                        rdo = rot;
                    }
                }
                __syncthreads();
                if (rdo) {
                    rotated = true;
                    const double c = rc;
                    const T se = rse, sec = rsec;
#pragma unroll
                    for (int k = 0; k < R; ++k) {
                        const int i = tid + k * kSvdThreads;
                        if (i < total) {
                            (i < M ? wp : vp)[i] = sadd(sscale(x[k], c), smul(sec, y[k]));
                            (i < M ? wq : vq)[i] = sadd(smul(se, x[k]), sscale(y[k], c));
                        }
                    }
                    for (int i = tid + R * kSvdThreads; i < total; i += kSvdThreads) {
                        T *a = (i < M ? wp : vp) + i, *b = (i < M ? wq : vq) + i;
                        const T u = ldcg(a), v = ldcg(b);
                        *a = sadd(sscale(u, c), smul(sec, v));
                        *b = sadd(smul(se, u), sscale(v, c));
                    }
                }
            }
            __syncthreads();  // the round's columns are written
            if (tid == 0) {
                __threadfence();
                st_release(&sy->cta[cta].rounds, done + 1);
            }
        }
        if (!ok) break;
        if (tid == 0) {
            atomicAdd(&sy->sweep[sweep], rotated ? 0x10001u : 1u);
            const bool met = svd_wait(&sy->sweep[sweep], 0xFFFFu, (uint32_t)nct, per_sweep, sy, status);
            agreed = met ? ld_acquire(&sy->sweep[sweep]) : 0u;  // final: every CTA has added its part
        }
        __syncthreads();
        if (agreed < 0x10000u) break;  // nobody rotated (or a wait gave up)
        __syncthreads();               // everyone has read it
    }
    // the norms of this CTA's columns (the arrangement at the start of a sweep)
    for (int pi = slot0; pi < slot1 && ok; ++pi)
        for (int h = 0; h < 2; ++h) {
            int pq[2];
            pair(pi, 0, pq[0], pq[1]);
            const int j = pq[h];
            if (j >= N) continue;
            double a = 0.0;
            for (int i = tid; i < M; i += kSvdThreads) a += abs2(ldcg(W + (int64_t)j * M + i));
            a = warp_sum(a);
            __syncthreads();
            if (lane == 0) part[warp][0] = a;
            __syncthreads();
            if (tid == 0) {
                a = 0.0;
                for (int w = 0; w < kSvdWarps; ++w) a += part[w][0];
                sy->sv[j] = sqrt(a);
            }
        }
    if (cta == 0 && tid == 0) sy->info = sweep;
}

// ---- the same sweeps inside one thread-block cluster --------------------------
__device__ __forceinline__ uint32_t map_cta(uint32_t addr, uint32_t cta) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(cta));
    return r;
}
// Stores into another CTA's shared memory that count their bytes on its mbarrier
__device__ __forceinline__ void st_async(uint32_t addr, double v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_async(uint32_t addr, double2 v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(addr),
                 "l"(__double_as_longlong(v.x)), "l"(__double_as_longlong(v.y)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ bool try_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait of a whole warp; after a time-out (or another warp's) every
// wait of the CTA returns at once, so that the sweep still reaches its barriers.
__device__ __forceinline__ void wait_cluster(uint32_t bar, uint32_t parity, volatile int *abort_flag, int32_t *status) {
    if (try_cluster(bar, parity)) return;
    const long long t0 = clock64();
    for (uint32_t n = 1;; ++n) {
        if (try_cluster(bar, parity)) return;
        if ((n & 255) == 0) {
            if (*abort_flag) return;
            if (clock64() - t0 > kWaitTimeoutCycles) {
                *abort_flag = 1;
                atomicCAS(status, 0, (int32_t)MGB_ERR_DEVICE_TIMEOUT);
                return;
            }
        }
    }
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

constexpr int kSvdRing = 4;          // rotations a slot's V warp may lag behind its W warp
constexpr int kSvdClusterRows = 256; // rows of W (8 per lane)
constexpr int kSvdClusterCols = 128;

template <typename T>
struct SvdSlot {
    uint64_t w_full[2], v_full[2];               // a round's two columns have arrived
    uint64_t r_full[kSvdRing], r_empty[kSvdRing];
    double c[kSvdRing];
    T se[kSvdRing];
    int32_t rot[kSvdRing];
};
template <typename T>
__host__ __device__ constexpr int svd_slot_header() {
    return ((int)sizeof(SvdSlot<T>) + 127) / 128 * 128;
}
// Bytes of one slot: its header, then W[round parity][upper, lower][M] and V the same with N.
template <typename T>
__host__ __device__ inline int svd_slot_bytes(int M, int N) {
    return svd_slot_header<T>() + (4 * (M + N) * (int)sizeof(T) + 127) / 128 * 128;
}

// The sweeps of k_svd_jacobi for matrices whose columns fit the shared memory
// of one cluster (up to 16 CTAs). The rounds of a small matrix are a chain of
// latencies, and the hand-over of columns through L2 (store, fence, flag,
// poll, load) is about half of it: 5 us a round at 64 x 64 ComplexF64, and
// 2.6 us here (1.80 ms for the SVD; 3.1 ms with the cooperative kernel, 16.8 ms
// in one block). Beyond 128 columns the 16 SMs' FP64 pipes are the longer
// part (192 columns: 14.3 ms on the cooperative grid, 391 ms in one block).
// Every slot has a warp for its two columns of W and one for those of V; a warp
// holds its columns in registers for the round and stores them straight into
// the shared memory of the slots that own them next (st.async), whose
// mbarrier counts the bytes. The V warps apply the rotations behind the W warps (a
// ring of kSvdRing rotations per slot), off the chain. A slot's two buffers
// suffice: it receives round r + 1 only from neighbours that have its columns
// of round r, which it sent after reading those of round r - 1.
template <typename T, int R>
__global__ void __launch_bounds__(512) k_svd_cluster(const T *__restrict__ A, int64_t lda, int trans, T *__restrict__ W,
                                                     int M, int N, T *__restrict__ V, double tol2, int spc, SvdSync *sy,
                                                     int32_t *status) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ int abort_flag;
    __shared__ uint32_t any[kMaxSweeps];  // CTA 0's: somebody rotated in sweep s
    const int nn = N + (N & 1), np = nn / 2;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int cta = blockIdx.x;
    const int ls = warp / 2, pi = cta * spc + ls;  // this warp's slot
    const bool vside = warp & 1, live = ls < spc && pi < np;
    const int sb = svd_slot_bytes<T>(M, N);
    const uint32_t smem0 = smem_u32(smem_raw);
    SvdSlot<T> *slot = (SvdSlot<T> *)(smem_raw + ls * sb);
    const int len = vside ? N : M;
    // columns of this side in this slot: [parity][upper, lower][len]
    T *cols = (T *)((unsigned char *)slot + svd_slot_header<T>()) + (vside ? 4 * M : 0);
    const uint32_t cols_off = smem_u32(cols) - smem_u32(slot);
    if (threadIdx.x == 0) abort_flag = 0;
    for (int i = threadIdx.x; i < kMaxSweeps; i += blockDim.x) any[i] = 0;
    if (live) {
        if (!vside && lane == 0) {
            for (int i = 0; i < 2; ++i) {
                mbar_init(smem_u32(slot->w_full + i), 1);
                mbar_init(smem_u32(slot->v_full + i), 1);
            }
            for (int i = 0; i < kSvdRing; ++i) {
                mbar_init(smem_u32(slot->r_full + i), 1);
                mbar_init(smem_u32(slot->r_empty + i), 1);
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        for (int h = 0; h < 2; ++h) {
            const int j = h ? circle(nn - 1 - pi, 0, nn) : circle(pi, 0, nn);
            for (int i = lane; i < len; i += 32) {
                T x = zero_of(T());  // the padding player of an odd N is a zero column
                if (vside) x = i == j ? one_of(T()) : zero_of(T());
                else if (j < N) x = trans ? sconj(A[(int64_t)i * lda + j]) : A[(int64_t)j * lda + i];
                cols[h * len + i] = x;
            }
        }
    }
    // where the upper and the lower column go after a round: the slot, and
    // its upper (0) or lower (1) place
    int dslot[2], dplace[2];
    dslot[0] = pi == 0 ? 0 : pi - 1;
    dplace[0] = pi == 1 ? 1 : 0;  // slot 0's upper column stays; slot 1's becomes slot 0's lower one
    dslot[1] = pi == np - 1 ? pi : pi + 1;
    dplace[1] = (pi == np - 1 && np > 1) ? 0 : 1;  // the last slot's lower column becomes its upper one
    uint32_t dcol[2], dbar[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int to = live ? dslot[h] : 0;
        const uint32_t base = map_cta(smem0 + (to % spc) * sb, to / spc);
        dcol[h] = base + cols_off + dplace[h] * len * (int)sizeof(T);
        dbar[h] = base + (uint32_t)(vside ? offsetof(SvdSlot<T>, v_full) : offsetof(SvdSlot<T>, w_full));
    }
    const uint32_t mybar = smem_u32(vside ? slot->v_full : slot->w_full);
    const uint32_t bytes = 2u * len * (uint32_t)sizeof(T);  // of a round's two columns
    __syncthreads();  // the barriers are initialised
    if (live && lane == 0) {
        mbar_expect_tx(mybar + 8, bytes);  // round 1's columns
        mbar_expect_tx(mybar, bytes);      // round 2's
    }
    __syncwarp();
    cluster_barrier();

    uint32_t G = 0;  // rounds so far, over all sweeps
    int sweep = 0;
    for (; sweep < kMaxSweeps; ++sweep) {
        bool rotated = false;
        for (int r = 0; live && r + 1 < nn; ++r, ++G) {
            const uint32_t buf = G & 1u, k = G % kSvdRing, kpar = (G / kSvdRing) & 1u;
            // buffer b's first arrivals are those of round 1 (b = 1) or 2 (b = 0)
            if (G > 0) {
                wait_cluster(mybar + 8 * buf, ((G - 1) / 2) & 1u, &abort_flag, status);
                if (lane == 0) mbar_expect_tx(mybar + 8 * buf, bytes);  // those of round G + 2
            }
            const bool swap = circle(pi, r, nn) > circle(nn - 1 - pi, r, nn);  // p is the smaller player
            const T *cp = cols + (2 * buf + (swap ? 1 : 0)) * len, *cq = cols + (2 * buf + (swap ? 0 : 1)) * len;
            T x[R], y[R];
#pragma unroll
            for (int i = 0; i < R; ++i) {
                x[i] = y[i] = zero_of(T());
                if (lane + 32 * i < len) {
                    x[i] = cp[lane + 32 * i];
                    y[i] = cq[lane + 32 * i];
                }
            }
            double c = 1.0;
            T se = zero_of(T()), sec = zero_of(T());
            bool rot;
            if (!vside) {
                double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
                for (int i = 0; i < R; ++i) dot_push(s, x[i], y[i]);
                warp_sum4(s, lane);
                rot = rotation<T>(s[0], s[1], dot_g(s, T()), tol2, c, se, sec);
            } else {
                wait_cluster(smem_u32(slot->r_full + k), kpar, &abort_flag, status);
                c = slot->c[k];
                se = slot->se[k];
                sec = sscale(sconj(se), -1.0);
                rot = slot->rot[k] != 0;
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(slot->r_empty + k));
            }
            // to the next round's owners (the buffer of the other parity)
            const uint32_t off = (buf ^ 1u) * 2 * len * (uint32_t)sizeof(T);
            const uint32_t dp = (swap ? dcol[1] : dcol[0]) + off, dq = (swap ? dcol[0] : dcol[1]) + off;
            const uint32_t bp = (swap ? dbar[1] : dbar[0]) + 8 * (buf ^ 1u), bq = (swap ? dbar[0] : dbar[1]) + 8 * (buf ^ 1u);
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int e = lane + 32 * i;
                if (e < len) {
                    const T u = rot ? sadd(sscale(x[i], c), smul(sec, y[i])) : x[i];
                    const T v = rot ? sadd(smul(se, x[i]), sscale(y[i], c)) : y[i];
                    st_async(dp + e * (int)sizeof(T), u, bp);
                    st_async(dq + e * (int)sizeof(T), v, bq);
                }
            }
            if (!vside) {  // the rotation, for the V warp
                wait_cluster(smem_u32(slot->r_empty + k), kpar ^ 1u, &abort_flag, status);
                if (lane == 0) {
                    slot->c[k] = c;
                    slot->se[k] = se;
                    slot->rot[k] = rot;
                    mbar_arrive(smem_u32(slot->r_full + k));
                }
                rotated |= rot;
            }
            __syncwarp();
        }
        if (live && !vside && rotated && lane == 0)
            asm volatile("red.relaxed.cluster.shared::cluster.or.b32 [%0], %1;" ::"r"(map_cta(smem_u32(any + sweep), 0)),
                         "r"(1u)
                         : "memory");
        __syncwarp();
        cluster_barrier();
        uint32_t go;
        asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(go) : "r"(map_cta(smem_u32(any + sweep), 0)) : "memory");
        if (!go) break;
    }
    // the columns lie as at the start of a sweep; nothing may be on its way to
    // this CTA's shared memory when it ends
    if (live && G > 0) {
        const long long t0 = clock64();
        while (!try_cluster(mybar + 8 * (G & 1u), ((G - 1) / 2) & 1u))
            if (clock64() - t0 > kWaitTimeoutCycles) break;
    }
    for (int h = 0; h < 2 && live; ++h) {
        const int j = h ? circle(nn - 1 - pi, 0, nn) : circle(pi, 0, nn);
        if (j >= N) continue;
        const T *src = cols + (2 * (G & 1u) + h) * len;
        T *dst = (vside ? V + (int64_t)j * N : W + (int64_t)j * M);
        double a = 0.0;
        for (int i = lane; i < len; i += 32) {
            const T x = src[i];
            dst[i] = x;
            a += abs2(x);
        }
        if (!vside) {
            a = warp_sum(a);
            if (lane == 0) sy->sv[j] = sqrt(a);
        }
    }
    if (cta == 0 && threadIdx.x == 0) sy->info = sweep;
    cluster_barrier();  // CTA 0's shared memory is read until here
}

// One block: the columns by descending norm (ties by column), the squared
// norm of the kept ones, and the left vectors of zero singular values (they
// come last): Gram-Schmidt of unit vectors against the columns before them.
template <typename T>
__global__ void __launch_bounds__(1024) k_svd_rank(T *__restrict__ W, int M, int N, int keep, SvdSync *sy) {
    __shared__ double sv[kSvdMaxCols];
    __shared__ int col_of_rank[kSvdMaxCols];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    for (int j = threadIdx.x; j < N; j += blockDim.x) sv[j] = sy->sv[j];
    __syncthreads();
    // norms are not negative, so their bits order them: integer compares
    for (int j = warp; j < N; j += blockDim.x / 32) {
        const long long bj = __double_as_longlong(sv[j]);
        int rk = 0;
        for (int k = lane; k < N; k += 32) {
            const long long bk = __double_as_longlong(sv[k]);
            rk += (bk > bj || (bk == bj && k < j)) ? 1 : 0;
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) rk += __shfl_xor_sync(0xffffffffu, rk, d);
        if (lane == 0) {
            col_of_rank[rk] = j;
            sy->col_of_rank[rk] = j;
        }
    }
    __syncthreads();
    if (warp != 0) return;
    double s2 = 0.0;
    for (int r = lane; r < keep; r += 32) s2 += sv[col_of_rank[r]] * sv[col_of_rank[r]];
    s2 = warp_sum(s2);
    if (lane == 0) sy->norm2 = s2;
    int first = N;  // the first zero singular value
    for (int r = lane; r < N; r += 32)
        if (!(sv[col_of_rank[r]] > 0.0)) first = min(first, r);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) first = min(first, __shfl_xor_sync(0xffffffffu, first, d));
    for (int r = first; r < N; ++r) {
        const int j = col_of_rank[r];
        if (sv[j] > 0.0) continue;
        T *wj = W + (int64_t)j * M;
        for (int cand = 0; cand < M; ++cand) {
            for (int i = lane; i < M; i += 32) wj[i] = (i == cand) ? one_of(T()) : zero_of(T());
            __syncwarp();
            for (int pass = 0; pass < 2; ++pass)
                for (int rr = 0; rr < r; ++rr) {
                    const int jr = col_of_rank[rr];
                    const T *u = W + (int64_t)jr * M;
                    const double inv = sv[jr] > 0.0 ? 1.0 / sv[jr] : 1.0;  // completed columns are unit vectors
                    T d = zero_of(T());
                    for (int i = lane; i < M; i += 32) d = sadd(d, smul(sconj(u[i]), wj[i]));
                    d = sscale(warp_sum(d), inv);
                    __syncwarp();
                    for (int i = lane; i < M; i += 32) wj[i] = sadd(wj[i], sscale(smul(sscale(u[i], inv), d), -1.0));
                    __syncwarp();
                }
            double a = 0.0;
            for (int i = lane; i < M; i += 32) a += abs2(wj[i]);
            a = warp_sum(a);
            if (a > 0.25) {
                for (int i = lane; i < M; i += 32) wj[i] = sscale(wj[i], 1.0 / sqrt(a));
                __syncwarp();
                break;
            }
        }
    }
}

// Triplet r = blockIdx.x of `keep`: U_out is (rows of A) x keep, V_out
// (columns of A) x keep. The left vectors of W are its normalised columns,
// the right ones the columns of V; for a wide A (trans) the roles swap:
// A = W^H = V S Uw^H. Flags as mgb_svd.
template <typename T>
__global__ void __launch_bounds__(kSvdThreads) k_svd_output(const T *__restrict__ W, int M, int N,
                                                            const T *__restrict__ V, int trans, int flags,
                                                            const SvdSync *__restrict__ sy, T *__restrict__ U_out,
                                                            double *__restrict__ s_out, T *__restrict__ V_out) {
    const int r = blockIdx.x, j = sy->col_of_rank[r];
    const double sj = sy->sv[j], inv = sj > 0.0 ? 1.0 / sj : 1.0;
    const T *w = W + (int64_t)j * M, *v = V + (int64_t)j * N;
    T *uo = (trans ? V_out : U_out) + (int64_t)r * M, *vo = (trans ? U_out : V_out) + (int64_t)r * N;
    const bool cu = trans && (flags & MGB_SVD_CONJ_V), cv = !trans && (flags & MGB_SVD_CONJ_V);
    for (int i = threadIdx.x; i < M; i += blockDim.x) {
        const T x = sscale(w[i], inv);
        uo[i] = cu ? sconj(x) : x;
    }
    for (int i = threadIdx.x; i < N; i += blockDim.x) vo[i] = cv ? sconj(v[i]) : v[i];
    if (threadIdx.x == 0) {
        const double scale = (flags & MGB_SVD_NORMALIZE) && sy->norm2 > 0.0 ? 1.0 / sqrt(sy->norm2) : 1.0;
        s_out[r] = (flags & MGB_SVD_SQRT_S) ? sqrt(sj * scale) : sj * scale;
    }
}

// W = A (M >= N) or A^H, from A with leading dimension lda; V = I; the
// waiting state cleared.
template <typename T>
__global__ void k_svd_load(const T *__restrict__ A, int64_t lda, int m, int n, int trans, T *__restrict__ W,
                           T *__restrict__ V, uint32_t *sync) {
    const int M = trans ? n : m, N = trans ? m : n;
    const int64_t id = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t idx = id; idx < (int64_t)M * N; idx += step) {
        const int64_t i = idx % M, j = idx / M;
        W[idx] = trans ? sconj(A[i * lda + j]) : A[j * lda + i];
    }
    for (int64_t idx = id; idx < (int64_t)N * N; idx += step) V[idx] = (idx % (N + 1) == 0) ? one_of(T()) : zero_of(T());
    for (int64_t idx = id; idx < (int64_t)(sizeof(SvdSync) / 4); idx += step) sync[idx] = 0;
}

constexpr uint64_t kSvdSyncBytes = (sizeof(SvdSync) + 255) & ~uint64_t(255);

static uint64_t svd_ws(int dtype, int64_t m, int64_t n) {
    const int64_t M = std::max(m, n), N = std::min(m, n);
    const uint64_t eb = dtype == MGB_C64 ? 16 : 8;
    return kSvdSyncBytes + ((M * N * eb + 255) & ~uint64_t(255)) + N * N * eb;
}

template <typename T, int R>
static int run_jacobi(T *W, int M, int N, T *V, double tol2, SvdSync *sy, cudaStream_t st) {
    int32_t *status = device_status_ptr();
    if (!status) return fail(MGB_ERR_CUDA, "device status word unavailable");
    int dev = 0, sms = 0, per_sm = 0;
    MGB_CUDA_CHECK(cudaGetDevice(&dev));
    MGB_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    MGB_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_svd_jacobi<T, R>, kSvdThreads, 0));
    // at most one CTA per SM (the FP64 pipe of an SM is what a CTA works with)
    const int np = (N + 1) / 2, most = std::min(std::max(per_sm > 0 ? sms : 1, 1), kSvdMaxCtas);
    int spc = (np + most - 1) / most;
    const int grid = (np + spc - 1) / spc;
    void *args[] = {&W, &M, &N, &V, &tol2, &spc, &sy, &status};
    MGB_CUDA_CHECK(cudaLaunchCooperativeKernel((const void *)k_svd_jacobi<T, R>, dim3(grid), dim3(kSvdThreads), args, 0, st));
    return MGB_OK;
}

// Largest cluster of at most `want` CTAs in which k_svd_cluster<T, R> can run
// `np` slots (0: none); `spc` slots per CTA, `smem` bytes of shared memory.
// The answer of the occupancy query is the same for every call (per device
// and slots per CTA), so a race between first callers only repeats it.
template <typename T, int R>
static int svd_cluster_size(int want, int np, int slot_bytes, int &spc, int &smem) {
    constexpr int kDevices = 64, kSpc = 9;
    static std::atomic<int8_t> known[kDevices][kSpc][5];  // by log2 of the size; 1: fits, -1: does not
    auto kern = k_svd_cluster<T, R>;
    int dev = 0, optin = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return 0;
    for (int cs = want, lg = 31 - __builtin_clz(want); cs >= 1; cs /= 2, --lg) {
        spc = (np + cs - 1) / cs;
        smem = spc * slot_bytes;
        // the largest shared memory a CTA of this kernel and `spc` asks for
        const int most = spc * svd_slot_bytes<T>(std::min(32 * R, kSvdClusterRows), std::min(32 * R, kSvdClusterCols));
        if (spc >= kSpc || most + 1024 > optin) return 0;
        int8_t k = dev < kDevices ? known[dev][spc][lg].load(std::memory_order_acquire) : 0;
        if (k == 0) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = cs;
            at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
            cfg.gridDim = dim3(cs);
            cfg.blockDim = dim3(64 * spc);
            cfg.dynamicSmemBytes = most;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int n = 0;
            // the attribute only ever grows: `optin` covers every caller
            const bool fits =
                cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - 1024) == cudaSuccess &&
                cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0;
            if (!fits) (void)cudaGetLastError();
            k = fits ? 1 : -1;
            if (dev < kDevices) known[dev][spc][lg].store(k, std::memory_order_release);
        }
        if (k > 0) return cs;
    }
    return 0;
}

template <typename T, int R>
static int run_cluster(const T *A, int64_t lda, int trans, T *W, int M, int N, T *V, double tol2, SvdSync *sy,
                       cudaStream_t st, bool &taken) {
    taken = false;
    const int np = (N + 1) / 2, sb = svd_slot_bytes<T>(M, N);
    int want = 16;
    while (want > 1 && want / 2 >= np) want /= 2;
    int spc = 0, smem = 0;
    const int cs = svd_cluster_size<T, R>(want, np, sb, spc, smem);
    if (cs == 0) return MGB_OK;
    int32_t *status = device_status_ptr();
    if (!status) return fail(MGB_ERR_CUDA, "device status word unavailable");
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(cs);
    cfg.blockDim = dim3(64 * spc);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    MGB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, k_svd_cluster<T, R>, A, lda, trans, W, M, N, V, tol2, spc, sy, status));
    taken = true;
    return MGB_OK;
}

template <typename T>
static int run_svd(int64_t m, int64_t n, const T *A, int64_t lda, T *U, double *s, T *Vout, int keep, int flags,
                   uint8_t *w, cudaStream_t st) {
    const int64_t M = std::max(m, n), N = std::min(m, n);
    const int trans = m < n ? 1 : 0;
    SvdSync *sy = (SvdSync *)w;
    T *W = (T *)(w + kSvdSyncBytes);
    T *V = (T *)(w + kSvdSyncBytes + ((M * N * sizeof(T) + 255) & ~uint64_t(255)));
    // relative orthogonality at which a pair is left alone
    const double tol = 4.0 * 1.1102230246251565e-16 * std::sqrt((double)M), tol2 = tol * tol;
    int rc;
    bool taken = false;
    if (M <= kSvdClusterRows && N <= kSvdClusterCols) {
        const int64_t per = (M + 31) / 32;  // elements of a column per lane
        if (per <= 1) rc = run_cluster<T, 1>(A, lda, trans, W, (int)M, (int)N, V, tol2, sy, st, taken);
        else if (per <= 2) rc = run_cluster<T, 2>(A, lda, trans, W, (int)M, (int)N, V, tol2, sy, st, taken);
        else if (per <= 4) rc = run_cluster<T, 4>(A, lda, trans, W, (int)M, (int)N, V, tol2, sy, st, taken);
        else rc = run_cluster<T, 8>(A, lda, trans, W, (int)M, (int)N, V, tol2, sy, st, taken);
        if (rc) return rc;
    }
    if (!taken) {
        const unsigned lb = (unsigned)std::min<int64_t>((M * N + 255) / 256, 152 * 8);
        k_svd_load<T><<<lb, 256, 0, st>>>(A, lda, (int)m, (int)n, trans, W, V, (uint32_t *)sy);
        MGB_CUDA_CHECK(cudaGetLastError());
        const int64_t per = (M + N + kSvdThreads - 1) / kSvdThreads;  // elements of a column pair per thread
        if (per <= 1) rc = run_jacobi<T, 1>(W, (int)M, (int)N, V, tol2, sy, st);
        else if (per <= 2) rc = run_jacobi<T, 2>(W, (int)M, (int)N, V, tol2, sy, st);
        else rc = run_jacobi<T, 4>(W, (int)M, (int)N, V, tol2, sy, st);
        if (rc) return rc;
    }
    k_svd_rank<T><<<1, N <= 256 ? 256 : 1024, 0, st>>>(W, (int)M, (int)N, keep, sy);
    MGB_CUDA_CHECK(cudaGetLastError());
    k_svd_output<T><<<(unsigned)keep, kSvdThreads, 0, st>>>(W, (int)M, (int)N, V, trans, flags, sy, U, s, Vout);
    MGB_CUDA_CHECK(cudaGetLastError());
    return MGB_OK;
}

}  // namespace mgb

using namespace mgb;

extern "C" int mgb_svd_workspace_size(int32_t dtype, int64_t m, int64_t n, uint64_t *bytes) {
    if (!bytes || (dtype != MGB_F64 && dtype != MGB_C64) || m < 0 || n < 0)
        return fail(MGB_ERR_ARGUMENT, "svd: Float64 or ComplexF64, nonnegative sizes");
    *bytes = svd_ws(dtype, m, n);
    return MGB_OK;
}

extern "C" int mgb_svd(int32_t dtype, int64_t m, int64_t n, const void *A, int64_t lda, void *U, void *s, void *V,
                       int32_t keep, int32_t flags, void *workspace, uint64_t workspace_bytes, void *stream) {
    if ((dtype != MGB_F64 && dtype != MGB_C64) || m < 0 || n < 0 || lda < std::max<int64_t>(m, 1))
        return fail(MGB_ERR_ARGUMENT, "svd: Float64 or ComplexF64, nonnegative sizes, lda >= m");
    const int64_t M = std::max(m, n), N = std::min(m, n);
    if (N == 0) return MGB_OK;
    if (N > kSvdMaxCols || M * N > (int64_t)1 << 28)
        return fail(MGB_ERR_UNSUPPORTED, "svd: min(m, n) above 1024 or m n above 2^28");
    if (keep <= 0 || keep > N) keep = (int32_t)N;
    if (flags & ~(MGB_SVD_NORMALIZE | MGB_SVD_CONJ_V | MGB_SVD_SQRT_S))
        return fail(MGB_ERR_ARGUMENT, "svd: unknown flags");
    if (!A || !U || !s || !V) return fail(MGB_ERR_ARGUMENT, "svd: null pointer");
    if (!workspace || workspace_bytes < svd_ws(dtype, m, n))
        return fail(MGB_ERR_WORKSPACE, "svd: workspace smaller than mgb_svd_workspace_size");
    if (((uintptr_t)workspace & 255) != 0) return fail(MGB_ERR_WORKSPACE, "svd: workspace must be 256-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    uint8_t *w = (uint8_t *)workspace;
    return dtype == MGB_C64
               ? run_svd<double2>(m, n, (const double2 *)A, lda, (double2 *)U, (double *)s, (double2 *)V, keep, flags, w, st)
               : run_svd<double>(m, n, (const double *)A, lda, (double *)U, (double *)s, (double *)V, keep, flags, w, st);
}
