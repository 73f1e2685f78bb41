// unary_einsum: Y[out] = sum over the remaining labels of X, where a label
// repeated in X walks the diagonal (src/Operations/unary_einsum.jl:26-46,
// ext/MuscleOMEinsumExt.jl:25-38; cases pinned by
// test/integration/omeinsum.jl:6-100: axis sum, full sum, ii->i, iji->ij,
// ii->, iji->j). The plan folds each distinct label into one mode whose X
// stride is the sum of its positions' strides, so the kernel is a strided
// reduction: y(o) = sum_r x(off_o + off_r). Memory-bound.
#include <algorithm>

#include "mgb_fxsum.h"
#include "mgb_internal.h"

namespace mgb {

// Loads in flight per thread: 64 bytes of them (with four 4-byte loads, sums of
// Float32 over a slower label ran at half the HBM rate).
template <typename T>
struct UnaryLoads {
    static constexpr int N = 64 / (int)sizeof(T);
};
constexpr int kUnaryThreads = 256;

// Accumulators: R is a thread's running sum (groups of elements, or single
// ones), V a sum that can be merged with others. Float32 / ComplexF32 add in
// FP32 into four independent partial sums. Float64 / ComplexF64 add into
// fixed-point sums on the integer pipes (mgb_fxsum.h): GB300's FP64 pipe would
// bound an FP64 sum at about half the HBM rate, and the fixed-point sum is also
// exact within 10 binades of the largest term.
template <typename T>
struct Acc;
template <>
struct Acc<float> {
    struct R {
        float s[4];
    };
    using V = float;
    __device__ static R zero() { return R{}; }
    template <int N>
    __device__ static void push(R &a, const float (&x)[N]) {
#pragma unroll
        for (int u = 0; u < N; ++u) a.s[u % 4] += x[u];
    }
    __device__ static void push1(R &a, float x) { a.s[0] += x; }
    __device__ static V fold(const R &a) { return (a.s[0] + a.s[1]) + (a.s[2] + a.s[3]); }
    __device__ static V none() { return 0.f; }
    __device__ static void merge(V &a, V b) { a += b; }
    __device__ static V shfl(V a, int d) { return __shfl_down_sync(0xffffffffu, a, d); }
    __device__ static float out(V a) { return a; }
};
template <>
struct Acc<float2> {
    struct R {
        float2 s[4];
    };
    using V = float2;
    __device__ static void add(float2 &a, float2 x) {
        a.x += x.x;
        a.y += x.y;
    }
    __device__ static R zero() { return R{}; }
    template <int N>
    __device__ static void push(R &a, const float2 (&x)[N]) {
#pragma unroll
        for (int u = 0; u < N; ++u) add(a.s[u % 4], x[u]);
    }
    __device__ static void push1(R &a, float2 x) { add(a.s[0], x); }
    __device__ static V fold(const R &a) {
        return make_float2((a.s[0].x + a.s[1].x) + (a.s[2].x + a.s[3].x), (a.s[0].y + a.s[1].y) + (a.s[2].y + a.s[3].y));
    }
    __device__ static V none() { return make_float2(0.f, 0.f); }
    __device__ static void merge(V &a, V b) { add(a, b); }
    __device__ static V shfl(V a, int d) {
        return make_float2(__shfl_down_sync(0xffffffffu, a.x, d), __shfl_down_sync(0xffffffffu, a.y, d));
    }
    __device__ static float2 out(V a) { return a; }
};
__device__ __forceinline__ FxSum fx_shfl(const FxSum &a, int d) {
    FxSum r;
    r.lo = __shfl_down_sync(0xffffffffu, (unsigned long long)a.lo, d);
    r.hi = __shfl_down_sync(0xffffffffu, (long long)a.hi, d);
    r.e = __shfl_down_sync(0xffffffffu, a.e, d);
    r.flags = __shfl_down_sync(0xffffffffu, a.flags, d);
    return r;
}
template <>
struct Acc<double> {
    using R = FxAcc;
    using V = FxSum;
    __device__ static R zero() { return fx_acc_zero(); }
    template <int N>
    __device__ static void push(R &a, const double (&x)[N]) {
        fx_acc_push(a, x);
    }
    __device__ static void push1(R &a, double x) {
        const double v[1] = {x};
        fx_acc_push(a, v);
    }
    __device__ static V fold(const R &a) { return fx_acc_sum(a); }
    __device__ static V none() { return fx_zero(); }
    __device__ static void merge(V &a, const V &b) { fx_merge(a, b); }
    __device__ static V shfl(const V &a, int d) { return fx_shfl(a, d); }
    __device__ static double out(const V &a) { return fx_value(a); }
};
struct FxAcc2 {
    FxAcc re, im;
};
struct FxSum2 {
    FxSum re, im;
};
template <>
struct Acc<double2> {
    using R = FxAcc2;
    using V = FxSum2;
    __device__ static R zero() { return FxAcc2{fx_acc_zero(), fx_acc_zero()}; }
    template <int N>
    __device__ static void push(R &a, const double2 (&x)[N]) {
        double v[N];
#pragma unroll
        for (int u = 0; u < N; ++u) v[u] = x[u].x;
        fx_acc_push(a.re, v);
#pragma unroll
        for (int u = 0; u < N; ++u) v[u] = x[u].y;
        fx_acc_push(a.im, v);
    }
    __device__ static void push1(R &a, double2 x) {
        const double re[1] = {x.x}, im[1] = {x.y};
        fx_acc_push(a.re, re);
        fx_acc_push(a.im, im);
    }
    __device__ static V fold(const R &a) { return FxSum2{fx_acc_sum(a.re), fx_acc_sum(a.im)}; }
    __device__ static V none() { return FxSum2{fx_zero(), fx_zero()}; }
    __device__ static void merge(V &a, const V &b) {
        fx_merge(a.re, b.re);
        fx_merge(a.im, b.im);
    }
    __device__ static V shfl(const V &a, int d) { return FxSum2{fx_shfl(a.re, d), fx_shfl(a.im, d)}; }
    __device__ static double2 out(const V &a) { return make_double2(fx_value(a.re), fx_value(a.im)); }
};

// Kernel arguments, in the parameter space (__grid_constant__): the mode
// groups are indexed where they lie, never copied to local memory.
struct UnaryArgs {
    ModeGroup go;        // outputs: tensor 0 = X stride, 1 = Y stride
    ModeGroup rest;      // reduced modes after the fastest one (X strides)
    int64_t e0, s0;      // fastest reduced mode: extent and X stride
    int64_t O, R;        // outputs, terms per output
    int32_t parts;       // blocks that share an output's terms
    void *part;          // their sums [O][parts] (V), when parts > 1
};

// X offset of term r of an output.
__device__ __forceinline__ int64_t unary_term(const UnaryArgs &a, int64_t r) {
    const int64_t q = ((uint64_t)r | (uint64_t)a.e0) <= 0x7FFFFFFFu ? (int64_t)((uint32_t)r / (uint32_t)a.e0) : r / a.e0;
    return (r - q * a.e0) * a.s0 + group_offset(a.rest, 0, q);
}
// Adds terms r0 + first, r0 + first + STEP, ... of [r0, r1) of one output, 64
// bytes of loads in flight. The fastest mode is walked without division, STEP terms
// apart within each of its runs, unless the runs are so short that lanes
// (STEP of them) would have none of it: then term by term.
template <typename T, int STEP>
__device__ __forceinline__ void unary_range(const T *__restrict__ xo, const UnaryArgs &a, int64_t r0, int64_t r1,
                                            int first, typename Acc<T>::R &acc) {
    constexpr int UU = UnaryLoads<T>::N;
    const int64_t e0 = a.e0, s0 = a.s0;
    if (e0 < (STEP > 1 ? 2 * STEP : UU)) {
        int64_t r = r0 + first;
        for (; r + (UU - 1) * STEP < r1; r += UU * STEP) {
            T v[UU];
#pragma unroll
            for (int u = 0; u < UU; ++u) v[u] = __ldg(xo + unary_term(a, r + u * STEP));
            Acc<T>::push(acc, v);
        }
        for (; r < r1; r += STEP) Acc<T>::push1(acc, __ldg(xo + unary_term(a, r)));
        return;
    }
    for (int64_t q = r0 / e0, base = q * e0; base < r1; ++q, base += e0) {
        const int64_t lo = max(r0 - base, (int64_t)0), hi = min(e0, r1 - base);
        const T *xq = xo + group_offset(a.rest, 0, q) + (lo + first) * s0;
        int64_t i = lo + first;
        for (; i + (UU - 1) * STEP < hi; i += UU * STEP, xq += UU * STEP * s0) {
            T v[UU];
#pragma unroll
            for (int u = 0; u < UU; ++u) v[u] = __ldg(xq + u * STEP * s0);
            Acc<T>::push(acc, v);
        }
        for (; i < hi; i += STEP, xq += STEP * s0) Acc<T>::push1(acc, __ldg(xq));
    }
}
template <typename T, int LANES = 32>
__device__ __forceinline__ typename Acc<T>::V warp_merge(typename Acc<T>::V v) {
#pragma unroll
    for (int d = LANES / 2; d > 0; d >>= 1) Acc<T>::merge(v, Acc<T>::shfl(v, d));
    return v;
}

// One thread per output: consecutive threads take consecutive outputs, so
// the loads are coalesced when Y's fastest mode is also X's (a sum over a
// slower label).
template <typename T>
__global__ void __launch_bounds__(kUnaryThreads) k_unary_thread(const T *__restrict__ x, T *__restrict__ y,
                                                                const __grid_constant__ UnaryArgs a) {
    for (int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < a.O; o += (int64_t)gridDim.x * blockDim.x) {
        typename Acc<T>::R acc = Acc<T>::zero();
        unary_range<T, 1>(x + group_offset(a.go, 0, o), a, 0, a.R, 0, acc);
        y[group_offset(a.go, 1, o)] = Acc<T>::out(Acc<T>::fold(acc));
    }
}

// LANES lanes per output: they take every LANES-th element of the fastest
// reduced mode; their sums are merged by shuffles. Fewer lanes for shorter
// reductions, since a merge of two fixed-point sums costs as much as several
// terms (200 k ComplexF64 sums of 64 terms: 272 us with 32 lanes each).
template <typename T, int LANES>
__global__ void __launch_bounds__(kUnaryThreads) k_unary_warp(const T *__restrict__ x, T *__restrict__ y,
                                                              const __grid_constant__ UnaryArgs a) {
    const int lane = threadIdx.x % LANES;
    const int64_t n = (int64_t)gridDim.x * blockDim.x / LANES;
    // whole warps stay in the loop, for the shuffles
    for (int64_t o = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / LANES;
         o - (threadIdx.x % 32) / LANES < a.O; o += n) {
        typename Acc<T>::R acc = Acc<T>::zero();
        if (o < a.O) unary_range<T, LANES>(x + group_offset(a.go, 0, o), a, 0, a.R, lane, acc);
        const typename Acc<T>::V v = warp_merge<T, LANES>(Acc<T>::fold(acc));
        if (lane == 0 && o < a.O) y[group_offset(a.go, 1, o)] = Acc<T>::out(v);
    }
}

// Few outputs: a block per (output, part of its terms) when the reduction runs
// along X's contiguous mode (ROW), else a block per (32 outputs, part), a lane
// per output and a warp per eighth of the part. With one part the block
// writes the outputs, otherwise its sums go to `part` for k_unary_merge. One
// warp per output, or one thread, left the GPU idle: summing 254 k ComplexF64
// elements into one took 1.8 ms.
template <typename T, bool ROW>
__global__ void __launch_bounds__(kUnaryThreads) k_unary_split(const T *__restrict__ x, T *__restrict__ y,
                                                               const __grid_constant__ UnaryArgs a) {
    using A = Acc<T>;
    constexpr int NW = kUnaryThreads / 32;
    __shared__ alignas(16) unsigned char raw[sizeof(typename A::V) * NW * (ROW ? 1 : 32)];
    typename A::V *sums = reinterpret_cast<typename A::V *>(raw);
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    const int64_t unit = blockIdx.x / a.parts;
    const int part = (int)(blockIdx.x - unit * a.parts);
    const int64_t o = ROW ? unit : unit * 32 + lane;
    typename A::R acc = A::zero();
    if constexpr (ROW) {
        const int64_t r0 = a.R * part / a.parts, r1 = a.R * (part + 1) / a.parts;
        unary_range<T, kUnaryThreads>(x + group_offset(a.go, 0, o), a, r0, r1, threadIdx.x, acc);
        const typename A::V v = warp_merge<T>(A::fold(acc));
        if (lane == 0) sums[warp] = v;
    } else {
        const int64_t n = (int64_t)a.parts * NW, i = (int64_t)part * NW + warp;
        if (o < a.O)
            unary_range<T, 1>(x + group_offset(a.go, 0, o), a, a.R * i / n, a.R * (i + 1) / n, 0, acc);
        sums[warp * 32 + lane] = A::fold(acc);
    }
    __syncthreads();
    if (warp != 0 || (ROW && lane != 0) || o >= a.O) return;
    typename A::V v = sums[ROW ? 0 : lane];
    for (int w = 1; w < NW; ++w) A::merge(v, sums[ROW ? w : w * 32 + lane]);
    if (a.parts == 1) y[group_offset(a.go, 1, o)] = A::out(v);
    else ((typename A::V *)a.part)[o * a.parts + part] = v;
}
// A warp per output adds its parts.
template <typename T>
__global__ void __launch_bounds__(kUnaryThreads) k_unary_merge(T *__restrict__ y, const __grid_constant__ UnaryArgs a) {
    using A = Acc<T>;
    const int lane = threadIdx.x % 32;
    const int64_t o = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / 32;
    if (o >= a.O) return;
    typename A::V v = A::none();
    for (int i = lane; i < a.parts; i += 32) A::merge(v, ((const typename A::V *)a.part)[o * a.parts + i]);
    v = warp_merge<T>(v);
    if (lane == 0) y[group_offset(a.go, 1, o)] = A::out(v);
}

// How a reduction is spread over the GPU.
struct UnarySplit {
    int lanes;       // lanes that share an output's terms: 1 (a thread per output), or 4 .. 32
    bool split;      // few outputs: blocks share them (k_unary_split)
    int32_t parts;
};
// Lanes share an output's terms when the reduction runs along X's contiguous
// mode (or no mode of the output is contiguous in X and the reduction is
// long), 8 terms or more each; otherwise a thread per output, coalesced over
// the outputs. Either way about kUnaryThreadsWanted threads (with 64 bytes
// of loads each, an SM needs some 700 to cover HBM's latency) should have work: below
// half of them blocks share outputs, and outputs are cut into parts of at
// least 8 terms per thread, when `ws` allows.
constexpr int64_t kUnaryThreadsWanted = 152 * 1024;
static UnarySplit unary_split(const UnaryPlan &p, bool ws) {
    const bool red_contig = p.gr.n > 0 && std::llabs(p.gr.str[0][0]) == 1 && p.gr.ext[0] > 1;
    const bool out_contig = p.go.n > 0 && std::llabs(p.go.str[0][0]) == 1 && p.go.ext[0] > 1;
    UnarySplit s;
    s.lanes = 1;
    s.split = false;
    s.parts = 1;
    if (p.O == 0) return s;  // nothing to share
    if (red_contig ? p.R >= 32 : p.R >= 64 && !out_contig) s.lanes = p.R >= 256 ? 32 : p.R >= 128 ? 16 : p.R >= 64 ? 8 : 4;
    s.split = p.O * s.lanes < kUnaryThreadsWanted / 2 && p.R >= (s.lanes > 1 ? 1024 : 16);
    if (s.split && ws) {
        const int64_t units = s.lanes > 1 ? p.O : (p.O + 31) / 32;
        const int64_t most = p.R / ((s.lanes > 1 ? kUnaryThreads : kUnaryThreads / 32) * 8);
        s.parts = (int32_t)std::max<int64_t>(1, std::min(kUnaryThreadsWanted / kUnaryThreads / units, most));
    }
    return s;
}
static int64_t unary_sum_bytes(int dtype) {
    switch (dtype) {
    case MGB_F32: return sizeof(Acc<float>::V);
    case MGB_F64: return sizeof(Acc<double>::V);
    case MGB_C32: return sizeof(Acc<float2>::V);
    default: return sizeof(Acc<double2>::V);
    }
}
uint64_t unary_workspace(const UnaryPlan &p) {
    const UnarySplit s = unary_split(p, true);
    return s.parts > 1 ? (uint64_t)(p.O * s.parts * unary_sum_bytes(p.x.dtype)) : 0;
}

template <typename T>
static int run_unary(const UnaryPlan &p, const T *x, T *y, void *ws, uint64_t ws_bytes, cudaStream_t s) {
    UnaryArgs a;
    a.go = p.go;
    ModeGroup gr = p.gr;
    if (a.go.n == 0) {
        a.go.n = 1;
        a.go.ext[0] = 1;
        a.go.str[0][0] = a.go.str[1][0] = a.go.str[2][0] = 0;
    }
    if (gr.n == 0) {
        gr.n = 1;
        gr.ext[0] = 1;
        gr.str[0][0] = gr.str[1][0] = gr.str[2][0] = 0;
    }
    a.e0 = std::max<int64_t>(gr.ext[0], 1);  // an empty sum has R = 0
    a.s0 = gr.str[0][0];
    a.rest.n = gr.n - 1;
    for (int i = 0; i + 1 < gr.n; ++i) {
        a.rest.ext[i] = gr.ext[i + 1];
        for (int t = 0; t < 3; ++t) a.rest.str[t][i] = gr.str[t][i + 1];
    }
    a.O = p.O;
    a.R = p.R;
    const bool fits = ws && ws_bytes >= unary_workspace(p) && ((uintptr_t)ws & 15) == 0;
    const UnarySplit sp = unary_split(p, fits);
    a.parts = sp.parts;
    a.part = ws;
    auto blocks = [&](int lanes) {
        return (unsigned)std::max<int64_t>(1, std::min<int64_t>((p.O * lanes + kUnaryThreads - 1) / kUnaryThreads, 152 * 16));
    };
    if (sp.split) {
        const int64_t units = sp.lanes > 1 ? p.O : (p.O + 31) / 32;
        const unsigned grid = (unsigned)(units * sp.parts);
        if (sp.lanes > 1) k_unary_split<T, true><<<grid, kUnaryThreads, 0, s>>>(x, y, a);
        else k_unary_split<T, false><<<grid, kUnaryThreads, 0, s>>>(x, y, a);
        MGB_CUDA_CHECK(cudaGetLastError());
        if (sp.parts > 1) k_unary_merge<T><<<(unsigned)((p.O * 32 + 255) / 256), kUnaryThreads, 0, s>>>(y, a);
    } else {
        switch (sp.lanes) {
        case 1: k_unary_thread<T><<<blocks(1), kUnaryThreads, 0, s>>>(x, y, a); break;
        case 4: k_unary_warp<T, 4><<<blocks(4), kUnaryThreads, 0, s>>>(x, y, a); break;
        case 8: k_unary_warp<T, 8><<<blocks(8), kUnaryThreads, 0, s>>>(x, y, a); break;
        case 16: k_unary_warp<T, 16><<<blocks(16), kUnaryThreads, 0, s>>>(x, y, a); break;
        default: k_unary_warp<T, 32><<<blocks(32), kUnaryThreads, 0, s>>>(x, y, a); break;
        }
    }
    MGB_CUDA_CHECK(cudaGetLastError());
    return MGB_OK;
}

int launch_unary(const UnaryPlan &p, const void *X, void *Y, void *ws, uint64_t ws_bytes, cudaStream_t s) {
    switch (p.x.dtype) {
    case MGB_F32: return run_unary<float>(p, (const float *)X, (float *)Y, ws, ws_bytes, s);
    case MGB_F64: return run_unary<double>(p, (const double *)X, (double *)Y, ws, ws_bytes, s);
    case MGB_C32: return run_unary<float2>(p, (const float2 *)X, (float2 *)Y, ws, ws_bytes, s);
    case MGB_C64: return run_unary<double2>(p, (const double2 *)X, (double2 *)Y, ws, ws_bytes, s);
    }
    return fail(MGB_ERR_ARGUMENT, "unary: bad dtype");
}

}  // namespace mgb
