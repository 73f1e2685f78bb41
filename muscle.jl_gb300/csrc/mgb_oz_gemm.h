// The tensor-core GEMM of the emulated forms over digit slices (OZAKI) or
// pieces (BF16X3), shared by its translation units: one contraction of a
// fixed slice count (mgb_oz_gemm_one.cu), one whose slice count the device
// chose (mgb_oz_gemm_any.cu), either in wide tiles (mgb_oz_gemm_wide.cu), and a
// table of contractions (mgb_oz_gemm_table.cu).
#pragma once

#include <cuda.h>

#include <atomic>
#include <type_traits>

#include "mgb_internal.h"
#include "mgb_ptx.h"
#include "mgb_x96.h"

namespace mgb {

constexpr int OZ_KC = 256;     // BF16X3: embedded k between readouts
constexpr int OZ_BM = 128;     // rows of A per CTA (TMEM lanes)
constexpr int OZ_BK = 32;      // k per stage (64-byte swizzled rows)
// Row tiles per rasterisation band. The resident CTAs drift apart in k over
// many waves, so L2 keeps a band's A slices only while they are small: on the
// 8192^3 ComplexF64 case (S = 6) DRAM traffic per launch is 222 GB for bands
// of 1, 135 GB for 2, 124 GB for 3, 145 GB for 4 and 187-224 GB for 8. The
// default is the widest band up to 3 whose A slices (band x 128 rows x all
// of K x S slices) stay within OZ_BAND_BYTES: on the same case S = 8 (two
// stages, so exposed to every L2 miss) ran 173 ms with bands of 3 (96 MiB),
// 133 ms with 2 and 142 ms with 1, while S = 6 (72 MiB at 3) ran 76.0 ms
// with 3 and 78.0 ms with 2.
constexpr int OZ_GROUP_M = 3;
constexpr int64_t OZ_BAND_BYTES = 90ll << 20;  // S = 7 at K_e = 16384: 84 MiB; S = 8: 96 MiB
// warp 0 TMA, warp 1 MMA issuer (and TMEM owner), warps 2..9 epilogue, warp 10
// second MMA issuer (narrow tiles)
constexpr int OZ_EPI_WARPS = 8;
__host__ __device__ constexpr int oz_threads(bool wide) { return 64 + 32 * OZ_EPI_WARPS + (wide ? 0 : 32); }
constexpr int OZ_ISSUER2_WARP = 2 + OZ_EPI_WARPS;
constexpr int OZ_A_TILE = OZ_BM * OZ_BK * 2;  // 8192 bytes per slice
constexpr int OZ_SMEM_BUDGET = 220 * 1024;
constexpr int OZ_MAX_STAGES = 6;
constexpr int OZ_NAN_EXP = 1 << 20;  // exponent of a row or column whose results are NaN

// Columns per digit group (= embedded rows of B per CTA): two banks of S
// groups must fit the 512 TMEM columns, and one MMA covers at most 256.
// BF16X3 (S = 3, two float registers per column) takes 64; the exact forms
// keep 32, where their three 32-bit words per column stay in registers.
// Wide tiles of the exact forms take 64 with one bank (see oz_gemm_body).
__host__ __device__ constexpr int oz_bn(int S, bool exact, bool wide = false) {
    return wide || (!exact && S <= 3) ? 64 : 32;
}
// Slice counts with wide tiles: 3, and 6, the usual one. With 5 they were 2 to
// 12 % slower (narrow tiles have a stage more there), with 4 between 3 % faster
// and 2 % slower; 7 and 8 have no room for three stages.
__host__ __device__ constexpr bool oz_wide(int S) { return S == 3 || S == 6; }
__host__ __device__ constexpr int oz_b_tile(int S, bool exact, bool wide = false) {  // bytes per slice
    return oz_bn(S, exact, wide) * OZ_BK * 2;
}
__host__ __device__ constexpr int oz_stage_bytes(int S, bool exact, bool wide = false) {
    return S * (OZ_A_TILE + oz_b_tile(S, exact, wide));
}
// Digit width and exact chunk length (in 32-wide k blocks) per slice count.
// W = 8 for S <= 6: |s1| <= 256, |si| <= 128, group bound max(d+1,4) 2^14, so a
// float32 accumulator stays exact over 4 blocks (128 k) for every d <= 7.
// W = 7 for S >= 7: group bound max(d+1,4) 2^12, exact over 8 blocks (256 k)
// for d <= 15. Both hold about the same number of mantissa bits (W S = 48 / 49).
__host__ __device__ constexpr int oz_digit_bits(int S) { return S <= 6 ? 8 : 7; }
__host__ __device__ constexpr int oz_chunk_blocks(int S) { return oz_digit_bits(S) == 8 ? 4 : 8; }
// k blocks between readouts
__host__ __device__ constexpr int oz_chunk(int S, bool exact) { return exact ? oz_chunk_blocks(S) : OZ_KC / OZ_BK; }
__host__ __device__ constexpr int oz_stages(int S, bool exact, bool wide = false) {
    return (OZ_SMEM_BUDGET / oz_stage_bytes(S, exact, wide)) < OZ_MAX_STAGES
               ? (OZ_SMEM_BUDGET / oz_stage_bytes(S, exact, wide))
               : OZ_MAX_STAGES;
}
// two banks of S groups of oz_bn columns; bank bases at columns 0 and 256
__host__ __device__ constexpr int oz_tmem_cols(int) { return 512; }
// More than half of the SM's shared memory for every S, so one CTA (and one
// TMEM allocation) per SM.
__host__ __device__ constexpr int oz_smem_bytes(int S, bool exact, bool wide = false) {
    return oz_stages(S, exact, wide) * oz_stage_bytes(S, exact, wide) + 1024 /*align*/ + 256 /*barriers*/;
}
static_assert(2 * oz_smem_bytes(3, true) > 228 * 1024 && 2 * oz_smem_bytes(8, true) > 228 * 1024 &&
                  2 * oz_smem_bytes(3, false) > 228 * 1024,
              "one CTA per SM");

// =============================================================================
// PTX wrappers
// =============================================================================
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *tm, int c0, int c1,
                                            int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(tm)), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                       uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// tcgen05.ld of 16 consecutive columns of this warp's 32 lanes (no wait)
__device__ __forceinline__ void tc_ld16_issue(uint32_t taddr, uint32_t *v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
          "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
          "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
// zeroes 16 consecutive columns of this warp's 32 lanes (no wait)
__device__ __forceinline__ void tc_st16_zero(uint32_t taddr) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr),
        "r"(0u)
        : "memory");
}
// stores 16 consecutive columns of this warp's 32 lanes (no wait)
__device__ __forceinline__ void tc_st16(uint32_t taddr, const float (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]),
        "f"(v[9]), "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15])
        : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// NC consecutive columns (a multiple of 16), then wait for the loads
template <int NC>
__device__ __forceinline__ void tc_ld(uint32_t taddr, uint32_t (&v)[NC]) {
#pragma unroll
    for (int c = 0; c < NC; c += 16) tc_ld16_issue(taddr + c, v + c);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// hi:lo += x m over 96 bits: one register less at a time than shifting x first,
// which wide tiles need (2-6 % faster there; the shift is 1-5 % faster in narrow
// ones, whose issue slots it spares).
__device__ __forceinline__ void add96(uint32_t &lo, int64_t &hi, int32_t x, int32_t m) {
    asm("{\n\t.reg .b64 p;\n\t.reg .b32 a, b, c, l, h;\n\t"
        "mul.wide.s32 p, %2, %3;\n\t"
        "mov.b64 {a, b}, p;\n\t"
        "shr.s32 c, b, 31;\n\t"
        "mov.b64 {l, h}, %1;\n\t"
        "add.cc.u32 %0, %0, a;\n\t"
        "addc.cc.u32 l, l, b;\n\t"
        "addc.u32 h, h, c;\n\t"
        "mov.b64 %1, {l, h};\n\t}"
        : "+r"(lo), "+l"(hi)
        : "r"(x), "r"(m));
}
// hi:lo += x over 96 bits
__device__ __forceinline__ void add96(uint32_t &lo, int64_t &hi, int64_t x) {
    asm("{\n\t.reg .b32 l, h;\n\t"
        "mov.b64 {l, h}, %1;\n\t"
        "add.cc.u32 %0, %0, %2;\n\t"
        "addc.cc.u32 l, l, %3;\n\t"
        "addc.u32 h, h, %4;\n\t"
        "mov.b64 %1, {l, h};\n\t}"
        : "+r"(lo), "+l"(hi)
        : "r"((uint32_t)x), "r"((uint32_t)((uint64_t)x >> 32)), "r"(x < 0 ? 0xFFFFFFFFu : 0u));
}
// f(integral_constant<int, s>) for s = 0 .. N-1, unrolled at compile time.
template <int N, int s = 0, typename F>
__device__ __forceinline__ void oz_static_for(F &&f) {
    if constexpr (s < N) {
        f(std::integral_constant<int, s>{});
        oz_static_for<N, s + 1>(f);
    }
}

// K-major operand tile, 64-byte swizzle: rows of 64 B, 8-row atoms of 512 B.
__device__ __forceinline__ uint64_t sw64_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);  // start address
    d |= (uint64_t)1 << 16;                   // leading byte offset (unused here)
    d |= (uint64_t)(512 >> 4) << 32;          // stride byte offset: 8 rows x 64 B
    d |= (uint64_t)1 << 46;                   // descriptor version (sm_100 family)
    d |= (uint64_t)4 << 61;                   // swizzle mode: 64 B
    return d;
}
// kind::f16 instruction descriptor: f32 accumulate, Float16 digits (EXACT) or
// bf16 pieces for both A and B, both K-major, M = 128, N = n (a multiple of 16
// up to 256).
__host__ __device__ constexpr uint32_t oz_idesc(int n, bool exact) {
    const uint32_t type = exact ? 0u : 1u;
    return (1u << 4) | (type << 7) | (type << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(OZ_BM >> 4) << 24);
}

// =============================================================================
// The tcgen05 GEMM over slices
// =============================================================================
struct OzGemmArgs {
    int64_t M, Ne, N;      // rows of A, embedded rows of B, un-embedded N
    int32_t nkb;           // number of 32-wide k blocks
    const int32_t *expA;   // [L][M] biased exponents (OZAKI)
    const int32_t *expB;   // [L][N]
    void *C;
    void *const *cptr;     // per-batch-entry output pointers (grouped execution) or null
    ModeGroup gm, gn, gl;  // C offsets live in tensor slot 2
    int32_t *status;
    const int32_t *sel;    // adaptive choice (nullable): run only when it holds S
    // Work units: the first `full` tiles are one unit each, every tile after
    // them is `splits` units of `kbs` k blocks (see oz_split). A split tile's
    // units leave their sums in `part` and count in `cnt` (zero before and
    // after); the last one adds them up and writes the outputs.
    int32_t splits, kbs;
    int64_t full;
    uint32_t *part;
    int32_t *cnt;
    // BF16X3: chunks per partial sum of a whole tile (0: one sum), those of the
    // units that it would be cut into (see oz_sum_blocks)
    int32_t fold;
};

// One contraction (or one bucket of a group) as the GEMM sees it: the slice
// tensor maps, the arguments and its tile grid (column tiles x row tiles x
// batch entries).
struct OzJobShape {
    OzGemmArgs a;
    int32_t tiles_n, tiles_m, L;
    __host__ __device__ int64_t units() const {
        const int64_t t = (int64_t)tiles_n * tiles_m * L;
        return a.full + (t - a.full) * a.splits;
    }
};
struct OzJob : OzJobShape {  // aligned as its tensor maps
    CUtensorMap tmA, tmB;
    int32_t band;  // row tiles per rasterisation band
};
// A contraction whose slice count a.sel holds: the tensor maps and the band of
// every candidate count (3 .. 8), and the candidates (bit S).
struct OzAnyJob : OzJobShape {
    CUtensorMap tm[6][2];
    int32_t band[6];
    uint32_t cand;
    int32_t S;  // the count when a.sel is null
};

// Tile sources of the kernel: one job in the parameter space, or a table of
// jobs in global memory (a group) whose work units (whole tiles, or parts of
// a split tile) are numbered consecutively. `hint` is the caller's job index
// of its previous unit (0 at first): a CTA visits its units in increasing
// order, so the next one usually lies in the same job or the one after it.
struct OzOneJob {
    static constexpr bool kTable = false;
    const OzJob *j;
    __device__ int64_t units() const { return j->units(); }
    __device__ bool any(int) const { return true; }
    __device__ const OzJobShape &job(int64_t t, int64_t &local, int &) const {
        local = t;
        return *j;
    }
    __device__ const CUtensorMap *map_a(int) const { return &j->tmA; }
    __device__ const CUtensorMap *map_b(int) const { return &j->tmB; }
    __device__ int band(int) const { return j->band; }
};
template <int S>
struct OzChosenJob {
    static constexpr bool kTable = false;
    const OzAnyJob *j;
    __device__ int64_t units() const { return j->units(); }
    __device__ bool any(int) const { return true; }
    __device__ const OzJobShape &job(int64_t t, int64_t &local, int &) const {
        local = t;
        return *j;
    }
    __device__ const CUtensorMap *map_a(int) const { return &j->tm[S - 3][0]; }
    __device__ const CUtensorMap *map_b(int) const { return &j->tm[S - 3][1]; }
    __device__ int band(int) const { return j->band[S - 3]; }
};
struct OzJobTable {
    static constexpr bool kTable = true;  // jobs may carry their own adaptive choice (skipped unless it is S)
    const OzJob *jobs;
    const int64_t *start;  // [n + 1]: first unit of each job, then the total
    int n;
    __device__ int64_t units() const { return start[n]; }
    __device__ bool any(int S) const {
        bool mine = false;
        for (int i = threadIdx.x; i < n; i += blockDim.x) mine = mine || !jobs[i].a.sel || *jobs[i].a.sel == S;
        return __syncthreads_or(mine);
    }
    __device__ const CUtensorMap *map_a(int i) const { return &jobs[i].tmA; }
    __device__ const CUtensorMap *map_b(int i) const { return &jobs[i].tmB; }
    __device__ int band(int i) const { return jobs[i].band; }
    __device__ const OzJobShape &job(int64_t t, int64_t &local, int &hint) const {
        int lo = hint;  // the last job with start <= t, at or after the hint
        if (lo + 1 < n && start[lo + 1] <= t) {
            ++lo;
            if (lo + 1 < n && start[lo + 1] <= t) {
                int hi = n - 1;
                ++lo;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) / 2;
                    if (start[mid] <= t) lo = mid;
                    else hi = mid - 1;
                }
            }
        }
        hint = lo;
        local = t - start[lo];
        return jobs[lo];
    }
    // The first tile after job `hint` that the CTA striding by `grid` from
    // `first` visits: a skipped job costs one step, not one per tile.
    __device__ int64_t after_job(int hint, int64_t first, int64_t grid) const {
        const int64_t e = start[hint + 1];
        return e + (((first - e) % grid) + grid) % grid;
    }
};

// The tile before this CTA's first tile after job `hint` (the tile loop then
// adds the grid stride): every role of the CTA skips a job of another slice
// count in one step, and all roles see the same choice, so their tile
// sequences stay equal.
template <typename Src>
__device__ __forceinline__ int64_t skip_job(const Src &src, int hint, int64_t t) {
    if constexpr (Src::kTable) return src.after_job(hint, blockIdx.x, gridDim.x) - gridDim.x;
    return t;
}

// Tile `local` of a job: batch entry, then grouped rasterisation within the
// entry, so that consecutive tiles walk a band of `band` row tiles across all
// column tiles and the CTAs resident at the same time share slices in L2.
template <typename I>
__device__ __forceinline__ void oz_tile_t(I local, I nn, I nm, I gm, int bn, int64_t &m0, int64_t &n0, int &l) {
    const I per = nn * nm;
    const I ll = local / per;
    const I t = local - ll * per;
    const I band = t / (gm * nn);
    const I first = band * gm;
    const I rows = min(gm, nm - first);
    const I r = t - band * gm * nn;
    l = (int)ll;
    m0 = (int64_t)(first + r % rows) * OZ_BM;
    n0 = (int64_t)(r / rows) * bn;
}
__device__ __forceinline__ void oz_tile(const OzJobShape &J, int64_t local, int64_t gm, int bn, int64_t &m0, int64_t &n0,
                                        int &l) {
    const int64_t nn = J.tiles_n, nm = J.tiles_m;
    // 32-bit divisions whenever the job's tile numbers fit (a 64-bit division
    // is a long software sequence)
    if (local <= INT32_MAX && (int64_t)J.L * nn * nm <= INT32_MAX && gm * nn <= INT32_MAX)
        oz_tile_t<uint32_t>((uint32_t)local, (uint32_t)nn, (uint32_t)nm, (uint32_t)gm, bn, m0, n0, l);
    else
        oz_tile_t<int64_t>(local, nn, nm, gm, bn, m0, n0, l);
}

// Work unit `local` of a job: its tile and k blocks [kb0, kb1), and its index
// among the units of split tiles (-1 for a whole tile). A job's split
// units are a few waves at most, so their numbers fit 32 bits.
struct OzUnit {
    int64_t m0, n0;
    int l, kb0, kb1, part;
};
__device__ __forceinline__ OzUnit oz_unit(const OzJobShape &J, int64_t local, int band, int bn) {
    OzUnit u;
    u.kb0 = 0;
    u.kb1 = J.a.nkb;
    u.part = -1;
    if (local >= J.a.full) {
        u.part = (int)(local - J.a.full);
        const int t = u.part / J.a.splits;
        u.kb0 = (u.part - t * J.a.splits) * J.a.kbs;
        u.kb1 = min(J.a.nkb, u.kb0 + J.a.kbs);
        local = J.a.full + t;
    }
    oz_tile(J, local, band, bn, u.m0, u.n0, u.l);
    return u;
}

// The compensation of a sum that overflowed is not a number, while the sum is
// an infinity that the next addition keeps: zero then, else c.
__device__ __forceinline__ float finite_comp(float c) { return fabsf(c) <= 3.402823466e38f ? c : 0.f; }
// Adds a partial sum x with its compensation c to a compensated sum (BF16X3);
// the parts of a tile always in the order of k.
__device__ __forceinline__ void add_part(float &sum, float &comp, float x, float c) {
    const float t = x - (c + comp), s = sum + t;
    comp = (s - sum) - t;
    sum = s;
}

// ---- sums of a split tile ------------------------------------------------------
// An epilogue warp's share of a unit: NW words per lane, as 16-byte vectors
// of consecutive lanes.
template <int NW>
__device__ __forceinline__ uint4 *oz_part_at(uint32_t *part, int unit, int w) {
    return (uint4 *)part + (((int64_t)unit * OZ_EPI_WARPS + w) * (NW / 4)) * 32 + threadIdx.x % 32;
}
// Publishes this warp's share and counts it; true for the warp that finds all
// `splits` shares of its tile published, whose count wraps to zero:
// the GEMM may run again on the same slices. Nobody waits for anybody.
__device__ __forceinline__ bool oz_part_last(int32_t *cnt, int tile, int w, int splits) {
    __threadfence();
    __syncwarp();
    uint32_t old = 0;
    if (threadIdx.x % 32 == 0)  // the last increment wraps to zero
        old = atomicInc((uint32_t *)cnt + tile * OZ_EPI_WARPS + w, (uint32_t)splits - 1);
    const bool last = __shfl_sync(0xffffffffu, old, 0) == (uint32_t)splits - 1;
    if (last) __threadfence();
    return last;
}

// One CTA computes 128 x BN tiles of the embedded output, in turn for the
// tiles t = blockIdx.x, blockIdx.x + gridDim.x, ...: the stage ring, the
// TMEM banks and their barriers run on across tiles, so the loads of the
// next tile overlap the MMAs and the readout of the current one. Digit group
// g = i + j (0-based slice indices of A and B) owns BN TMEM columns; the S
// groups of a chunk form one bank of BN S columns, and two banks alternate
// so that the epilogue reads chunk c while the MMAs fill chunk c + 1.
// The B slices of a stage lie back to back (BN rows each), so the products
// of A slice i with B slices 0 .. S-1-i are ONE tcgen05.mma with
// N = BN (S - i) whose accumulator columns are exactly groups i .. S-1:
// S wide MMAs per 16 k instead of S (S+1)/2 narrow ones, and every A slice
// is read from shared memory once per 16 k. BN = 64 for BF16X3 and 32 for
// the exact forms: the widest that two banks leave room for while the
// epilogue's accumulators (96-bit integers, or float sums and their
// compensations) stay in registers.
//
// WIDE (EXACT, see oz_wide): 128 x 64 tiles. Shared memory bounds the narrow ones:
// per 16 k a tile's slices are written once and A's are read once, whatever
// its width, so twice the columns save 26 % of the bytes (112 KB against
// 2 x 76 at S = 6). Two banks of 64-column groups do not fit TMEM, so there is
// one, and the readout of a chunk overlaps the MMAs of the next by groups
// instead of by banks: the epilogue reads, clears and releases the groups from
// the last to the first, and the issuer starts a chunk with its last A slice,
// whose products touch the last group only, then the one before it, and so on,
// each over the chunk's first two k blocks. An MMA covers at most 256 columns,
// so the first two A slices take two MMAs each. With MMAs this long one issuer
// keeps the tensor core's queue filled across its polls. 8192^3, S = 6: 18.6 ms
// in narrow tiles, 16.8 in wide ones (Float64), 75.2 and 67.3 (ComplexF64). A
// chunk takes 9.4 k cycles, of which the readout 3.3 k; two places for the last
// two groups, a readout without conversions (eight cycles of their unit per
// warp) or with more registers, and sixteen epilogue warps were slower.
template <int S, bool EXACT, bool CX, bool WIDE, typename Src>
__device__ __forceinline__ void oz_gemm_body(const Src &src) {
    constexpr int W = oz_digit_bits(S);  // digit width (EXACT)
    constexpr int KCB = oz_chunk(S, EXACT);  // k blocks per chunk
    constexpr int NST = oz_stages(S, EXACT, WIDE);
    constexpr int STAGE = oz_stage_bytes(S, EXACT, WIDE);
    constexpr int BN = oz_bn(S, EXACT, WIDE);  // columns per digit group, embedded B rows per CTA
    constexpr int HALF = BN / 2;     // columns per group read by one epilogue warp
    constexpr int TCOLS = oz_tmem_cols(S);
    constexpr int BANK = TCOLS / 2;  // TMEM column offset of the second bank
    constexpr int SUMS = BN * S;  // BF16X3: first free TMEM column of a bank
    static_assert(EXACT || SUMS + BN <= BANK, "BF16X3: two sums per column beside the banks");
    static_assert(NST >= 2, "need at least two pipeline stages");
    static_assert(WIDE ? BN * S <= TCOLS : BN * S <= BANK, "the accumulators must fit in TMEM");
    static_assert(WIDE ? EXACT && oz_wide(S) : BN * S <= 256, "one MMA covers at most 256 columns");
    static_assert(oz_smem_bytes(S, EXACT, WIDE) <= 227 * 1024, "shared memory of a CTA");
    static_assert(HALF % 16 == 0, "epilogue reads 16 columns at a time");
    // MMA-issuing threads. Each mbarrier poll by an issuing thread stalls it
    // for ~150 cycles while the tensor core's queue holds only ~200 cycles of
    // MMAs, so a single issuer leaves a bubble at every k block. Two issuers
    // (warps 1 and 10) take alternate k blocks and keep the queue fed while
    // the other polls. Their MMAs into a bank interleave in an unspecified
    // order, which changes nothing for the exact integer sums of the OZAKI
    // form; BF16X3 sums round, so it keeps one issuer and stays deterministic.
    constexpr int NI = EXACT && !WIDE ? 2 : 1;
    constexpr int NF = WIDE ? S : 2;  // accumulator parts released one by one: groups, or banks

    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *bars = (uint64_t *)(smem + NST * STAGE);
    uint64_t *full = bars;               // [2 NST] see full_idx
    uint64_t *empty = bars + 2 * NST;    // [NST]
    uint64_t *acc_full = bars + 3 * NST; // [2] bank filled (one commit per issuer)
    uint64_t *acc_empty = acc_full + 2;  // [NF] part read and cleared (one arrive per epilogue warp)
    uint64_t *done = acc_empty + NF;     // [2] per issuer: all its MMAs complete
    uint32_t *tmem_slot = (uint32_t *)(done + 2);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);

    // Stage-landed barriers, indexed by the CTA's running k-block count g
    // (across its tiles). Each barrier is waited on by a single issuer and in
    // order of its phases: an mbarrier parity wait cannot tell phase r from
    // phase r - 2, so a waiter that could run two phases ahead of a barrier
    // would pass early. With two issuers and an odd stage count the rounds of
    // a stage alternate between the issuers, so every stage gets one barrier
    // per issuer (index 2 s + g % 2) and each of those is used every other
    // round; otherwise stage s always has the same issuer (index 2 s + s % 2,
    // or 2 s for one issuer), used every round.
    auto full_idx = [](uint32_t g) { return 2 * (int)(g % NST) + (NI == 2 ? (int)(g & 1u) : 0); };
    auto full_par = [](uint32_t g) {
        const uint32_t r = g / NST;
        return (NI == 2 && (NST & 1)) ? (r >> 1) & 1u : r & 1u;
    };
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const int64_t T = src.units();
    int32_t *status;
    {
        int64_t unused;
        int h0 = 0;
        const OzGemmArgs &a0 = src.job(0, unused, h0).a;
        status = a0.status;
    }
    // a table none of whose contractions chose this count returns before it
    // touches shared memory or TMEM
    if (!src.any(S)) return;

    if (tid == 0) {
        for (int s = 0; s < NST; ++s) {
            mbar_init(smem_u32(full + 2 * s), 1);
            mbar_init(smem_u32(full + 2 * s + 1), 1);
            mbar_init(smem_u32(empty + s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(acc_full + b), NI);
            mbar_init(smem_u32(done + b), 1);
        }
        for (int b = 0; b < NF; ++b) mbar_init(smem_u32(acc_empty + b), OZ_EPI_WARPS);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"((uint32_t)TCOLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // Every MMA accumulates (the issuers' order within a bank is free); the
    // epilogue warps clear both banks here and each bank again after reading it.
    if (warp >= 2 && warp < 2 + OZ_EPI_WARPS) {
        const int q = warp % 4, h = (warp - 2) / 4;
        for (int c = 0; c < TCOLS / 2; c += 16) tc_st16_zero(tmem + ((uint32_t)(32 * q) << 16) + h * (TCOLS / 2) + c);
        tc_wait_st();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    // ---------------- TMA producer ----------------
    auto produce = [&]() {
        if (lane == 0) {
            uint32_t g = 0;  // k blocks issued so far, over all tiles of this CTA
            bool ok = true;
            int hint = 0;
            for (int64_t t = blockIdx.x; t < T && ok; t += gridDim.x) {
                int64_t local;
                const OzJobShape &J = src.job(t, local, hint);
                if (Src::kTable && J.a.sel && *J.a.sel != S) {  // a job of another slice count
                    t = skip_job(src, hint, t);
                    continue;
                }
                const OzUnit u = oz_unit(J, local, src.band(hint), BN);
                for (int kb = u.kb0; kb < u.kb1; ++kb, ++g) {
                    const int s = (int)(g % NST);
                    const uint32_t round = g / NST;
                    if (!mbar_wait(smem_u32(empty + s), (round & 1) ^ 1, abort_flag, status)) {
                        ok = false;
                        break;
                    }
                    uint8_t *st = smem + s * STAGE;
                    const uint32_t fb = smem_u32(full + full_idx(g));
                    mbar_expect_tx(fb, STAGE);
                    tma_load_3d(smem_u32(st), src.map_a(hint), kb * OZ_BK, (int)u.m0, u.l * S, fb);
                    tma_load_3d(smem_u32(st + S * OZ_A_TILE), src.map_b(hint), kb * OZ_BK, (int)u.n0, u.l * S, fb);
                }
            }
            // make sure no bulk copy is still writing into shared memory
            for (uint32_t gg = g > (uint32_t)NST ? g - NST : 0u; gg < g; ++gg)
                mbar_drain(smem_u32(full + full_idx(gg)), full_par(gg));
        }
    };
    // ---------------- MMA issuer (wide tiles) ----------------
    auto issue_wide = [&]() {
        if (lane == 0) {
            bool ok = true;
            uint32_t g = 0, C = 0;
            int hint = 0;
            // the products of A slice i over 16 k of a stage
            auto issue = [&](uint32_t stage, int i, int k16) {
                const uint32_t a_base = smem_u32(smem + stage * STAGE);
                const uint64_t ad = sw64_desc(a_base) + (uint64_t)((i * OZ_A_TILE + k16 * 32) >> 4);
                const uint64_t bd = sw64_desc(a_base + S * OZ_A_TILE) + (uint64_t)((k16 * 32) >> 4);
                // columns of the first MMA: both of a pair at least 128 wide,
                // below which an MMA waits for A's slice
                const int n = BN * (S - i), n1 = n > 256 ? 192 : n;
                tc_mma(tmem + BN * i, ad, bd, oz_idesc(n1, true), 1u);
                if (n > n1)
                    tc_mma(tmem + BN * i + n1, ad, bd + (uint64_t)((n1 / BN) * oz_b_tile(S, true, true) >> 4),
                           oz_idesc(n - n1, true), 1u);
            };
            for (int64_t t = blockIdx.x; t < T && ok; t += gridDim.x) {
                int64_t local;
                const OzJobShape &J = src.job(t, local, hint);
                const OzUnit u = oz_unit(J, local, src.band(hint), BN);
                const int nkb = u.kb1 - u.kb0;
                for (int c0 = 0; c0 < nkb && ok; c0 += KCB, ++C) {
                    const int c1 = min(nkb, c0 + KCB), r1 = min(c1, c0 + 2);
                    for (int kb = c0; kb < r1 && ok; ++kb)
                        ok = mbar_wait(smem_u32(full + full_idx(g + kb)), full_par(g + kb), abort_flag, status);
#pragma unroll
                    for (int i = S - 1; i >= 0; --i) {
                        // group i of the previous chunk read and cleared
                        ok = ok && mbar_wait(smem_u32(acc_empty + i), (C & 1u) ^ 1u, abort_flag, status);
                        if (!ok) break;
                        tc_fence_after();
                        for (int kb = c0; kb < r1; ++kb)
#pragma unroll
                            for (int k16 = 0; k16 < OZ_BK / 16; ++k16) issue((g + kb) % NST, i, k16);
                    }
                    if (!ok) break;
                    for (int kb = c0; kb < r1; ++kb) tc_commit(smem_u32(empty + (g + kb) % NST));
                    for (int kb = r1; kb < c1; ++kb) {
                        if (!mbar_wait(smem_u32(full + full_idx(g + kb)), full_par(g + kb), abort_flag, status)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
#pragma unroll
                        for (int k16 = 0; k16 < OZ_BK / 16; ++k16)
#pragma unroll
                            for (int i = S - 1; i >= 0; --i) issue((g + kb) % NST, i, k16);
                        tc_commit(smem_u32(empty + (g + kb) % NST));
                    }
                    if (ok) tc_commit(smem_u32(acc_full));
                }
                g += (uint32_t)nkb;
            }
            // wait for every MMA before TMEM is released
            tc_commit(smem_u32(done));
            mbar_drain(smem_u32(done), 0);
        }
    };
    // ---------------- MMA issuers (narrow tiles) ----------------
    auto issue_narrow = [&]() {
        // Issuer `me` takes the k blocks whose running count g has g % NI == me.
        // Per chunk C (counted over all tiles) it waits until the epilogue has
        // read and cleared the bank's previous chunk (C - 2), issues its k
        // blocks, and commits the chunk's acc_full barrier once (also when it
        // owns no k block of it).
        if (lane == 0) {
            const int me = warp == 1 ? 0 : 1;
            bool ok = true;
            uint32_t g = 0, C = 0;
            int hint = 0;
            for (int64_t t = blockIdx.x; t < T && ok; t += gridDim.x) {
                int64_t local;
                const OzJobShape &J = src.job(t, local, hint);
                if (Src::kTable && J.a.sel && *J.a.sel != S) {  // a job of another slice count
                    t = skip_job(src, hint, t);
                    continue;
                }
                const OzUnit u = oz_unit(J, local, src.band(hint), BN);
                const int nkb = u.kb1 - u.kb0;
                for (int c0 = 0; c0 < nkb && ok; c0 += KCB, ++C) {
                    const uint32_t bank = C & 1u;
                    if (!mbar_wait(smem_u32(acc_empty + bank), ((C >> 1) & 1u) ^ 1u, abort_flag, status)) {
                        ok = false;
                        break;
                    }
                    const int c1 = min(nkb, c0 + KCB);
                    for (int kb = c0; kb < c1; ++kb) {
                        const uint32_t gg = g + (uint32_t)kb;
                        if (NI == 2 && (int)(gg & 1u) != me) continue;
                        const int s = (int)(gg % NST);
                        if (!mbar_wait(smem_u32(full + full_idx(gg)), full_par(gg), abort_flag, status)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t a_base = smem_u32(smem + s * STAGE);
                        const uint64_t ad0 = sw64_desc(a_base);
                        const uint64_t bd0 = sw64_desc(a_base + S * OZ_A_TILE);
                        const uint32_t d0 = tmem + bank * BANK;
#pragma unroll
                        for (int k16 = 0; k16 < OZ_BK / 16; ++k16)
#pragma unroll
                            for (int i = 0; i < S; ++i)
                                tc_mma(d0 + BN * i, ad0 + (uint64_t)((i * OZ_A_TILE + k16 * 32) >> 4),
                                       bd0 + (uint64_t)((k16 * 32) >> 4), oz_idesc(BN * (S - i), EXACT), 1u);
                        tc_commit(smem_u32(empty + s));
                    }
                    if (ok) tc_commit(smem_u32(acc_full + bank));
                }
                g += (uint32_t)nkb;
            }
            // wait for every MMA this thread issued before TMEM is released
            tc_commit(smem_u32(done + me));
            mbar_drain(smem_u32(done + me), 0);
        }
    };
    // ---------------- epilogue ----------------
    auto epilogue = [&]() {
        const int q = warp % 4;        // TMEM lane quarter this warp may access
        const int h = (warp - 2) / 4;  // column half (HALF columns) of each group
        const uint32_t tbase = tmem + ((uint32_t)(32 * q) << 16) + HALF * h;
        bool ok = true;
        uint32_t C = 0;  // chunks read so far, over all tiles of this CTA
        int hint = 0;
        for (int64_t t = blockIdx.x; t < T && ok; t += gridDim.x) {
            int64_t local;
            const OzJobShape &J = src.job(t, local, hint);
            if (Src::kTable && J.a.sel && *J.a.sel != S) {  // a job of another slice count
                t = skip_job(src, hint, t);
                continue;
            }
            const OzGemmArgs &args = J.a;
            const OzUnit u = oz_unit(J, local, src.band(hint), BN);
            const int64_t n0 = u.n0;
            const int l = u.l;
            const int64_t row = u.m0 + 32 * q + lane;
            const int nchunks = (u.kb1 - u.kb0 + KCB - 1) / KCB;
            // Output addressing of the tile, fetched before the first chunk
            // wait so that its loads overlap the MMAs: the thread's row (offset
            // and exponent), and one output column per lane (lane j < NCOL
            // holds column j of this warp's half, broadcast by shuffles). A
            // row or column without finite values has the exponent OZ_NAN_EXP.
            constexpr int NCOL = CX ? HALF / 2 : HALF;
            const bool row_ok = row < args.M;
            int64_t rowoff = 0;
            int erow = 0;
            if (row_ok) {
                rowoff = (args.cptr ? 0 : group_offset(args.gl, 2, l)) + group_offset(args.gm, 2, row);
                if (EXACT) {
                    const int be = args.expA[(int64_t)l * args.M + row];
                    erow = be == 0x7FF ? OZ_NAN_EXP : be == 0 ? -1022 : be - 1022;
                }
            }
            long long lcoff = 0;
            int lexp = 0;  // the column's exponent and the scale of X's last bit
            bool lcol = false;
            {
                const int64_t ne = n0 + HALF * h + (int64_t)lane * (CX ? 2 : 1);
                if (lane < NCOL && ne < args.Ne) {
                    const int64_t n = CX ? (ne >> 1) : ne;
                    lcoff = group_offset(args.gn, 2, n);
                    lcol = true;
                    if (EXACT) {
                        const int be = args.expB[(int64_t)l * args.N + n];
                        lexp = (be == 0x7FF ? OZ_NAN_EXP : be == 0 ? -1022 : be - 1022) - W * (S + 1);
                    }
                }
            }
            const uint32_t cols = __ballot_sync(0xffffffffu, lcol);
            void *const Cl = args.cptr ? args.cptr[l] : args.C;
            // EXACT: one 96-bit integer X = sum_d G_d 2^(W (S + 1 - d)) per
            // output column, x0 + x1 2^32
            uint32_t x0[EXACT ? HALF : 1];
            int64_t x1[EXACT ? HALF : 1];
            // BF16X3: Kahan-compensated float32 sum over the chunks (of a part)
            int left = args.fold;  // chunks to the end of the part
            float accf[EXACT ? 1 : HALF], comp[EXACT ? 1 : HALF];
#pragma unroll
            for (int j = 0; j < HALF; ++j) {
                if (EXACT) {
                    x0[j] = 0;
                    x1[j] = 0;
                } else {
                    accf[j] = 0.f;
                    comp[j] = 0.f;
                }
            }
#pragma unroll 1
            for (int c = 0; c < nchunks; ++c, ++C) {
                const uint32_t bank = WIDE ? 0u : C & 1u;
                // warp-uniform outcome: the warp-collective loads below need every lane
                if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(acc_full + bank), (WIDE ? C : C >> 1) & 1u, abort_flag,
                                                       status))) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t tb = tbase + bank * BANK;
                // adds 16 columns' partial sums of a group, shifted into place
                auto add_group = [&](auto gc, auto jc, const uint32_t (&v)[16]) {
                    constexpr int sh = W * (S - 1 - decltype(gc)::value);  // W (S + 1 - d), d = g + 2
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const int32_t x = __float2int_rn(__uint_as_float(v[j]));
                        const int k = decltype(jc)::value + j;
                        if constexpr (sh < 32 && !WIDE) add96(x0[k], x1[k], (int64_t)x << sh);
                        else if constexpr (sh < 32) add96(x0[k], x1[k], x, 1 << sh);
                        else x1[k] += (int64_t)x << (sh - 32);
                    }
                };
                if constexpr (WIDE) {
                    oz_static_for<S>([&](auto ic) {
                        constexpr int g = S - 1 - decltype(ic)::value;  // from the last to the first
                        const uint32_t at = tb + BN * g;
                        oz_static_for<HALF / 16>([&](auto hc) {
                            constexpr int c2 = 16 * decltype(hc)::value;
                            uint32_t v[16];
                            tc_ld<16>(at + c2, v);
                            tc_st16_zero(at + c2);
                            if constexpr (c2 + 16 == HALF) {  // this warp's share of the group read and cleared
                                tc_wait_st();
                                tc_fence_before();
                                __syncwarp();
                                if (lane == 0) mbar_arrive(smem_u32(acc_empty + g));
                            }
                            add_group(std::integral_constant<int, g>{}, std::integral_constant<int, c2>{}, v);
                        });
                    });
                } else if constexpr (EXACT) {
                    oz_static_for<S>([&](auto gc) {
                        constexpr int g = decltype(gc)::value;
                        uint32_t v[16];
                        tc_ld<16>(tb + BN * g, v);
                        tc_st16_zero(tb + BN * g);
                        if constexpr (g == S - 1) {  // every group of the bank read and cleared
                            tc_wait_st();
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(smem_u32(acc_empty + bank));
                        }
                        add_group(gc, std::integral_constant<int, 0>{}, v);
                    });
                }
                if constexpr (!EXACT) {
                    // pieces hi*hi, then the products of piece-index sum 1 and 2;
                    // 16 columns at a time, so that the three groups' registers
                    // stay beside the running sums and their compensations
#pragma unroll
                    for (int c2 = 0; c2 < HALF; c2 += 16) {
                        uint32_t v0[16], v1[16], v2[16];
                        tc_ld<16>(tb + c2, v0);
                        tc_ld<16>(tb + BN + c2, v1);
                        tc_ld<16>(tb + 2 * BN + c2, v2);
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            float x = __uint_as_float(v0[j]) + (__uint_as_float(v1[j]) + __uint_as_float(v2[j]));
                            float y = x - comp[c2 + j];
                            float s2 = accf[c2 + j] + y;
                            comp[c2 + j] = (s2 - accf[c2 + j]) - y;
                            accf[c2 + j] = s2;
                        }
                    }
#pragma unroll
                    for (int g = 0; g < 3; ++g)
#pragma unroll
                        for (int c2 = 0; c2 < HALF; c2 += 16) tc_st16_zero(tb + BN * g + c2);
                    tc_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(acc_empty + bank));
                    // A whole tile adds its parts as a cut one does: the sums so
                    // far wait in the TMEM columns that the banks leave free.
                    const bool last = c + 1 == nchunks;
                    if (args.fold && u.part < 0 && (--left == 0 || last)) {
                        left = args.fold;
#pragma unroll
                        for (int c2 = 0; c2 < HALF; c2 += 16) {
                            float sum[16], cs[16];
                            if (c >= args.fold) {
                                uint32_t v0[16], v1[16];
                                tc_ld16_issue(tbase + SUMS + c2, v0);
                                tc_ld<16>(tbase + BANK + SUMS + c2, v1);
#pragma unroll
                                for (int j = 0; j < 16; ++j) {
                                    sum[j] = __uint_as_float(v0[j]);
                                    cs[j] = __uint_as_float(v1[j]);
                                }
                            } else {
#pragma unroll
                                for (int j = 0; j < 16; ++j) sum[j] = cs[j] = 0.f;
                            }
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                add_part(sum[j], cs[j], accf[c2 + j], finite_comp(comp[c2 + j]));
                                accf[c2 + j] = last ? sum[j] : 0.f;
                                comp[c2 + j] = 0.f;
                            }
                            if (!last) {
                                tc_st16(tbase + SUMS + c2, sum);
                                tc_st16(tbase + BANK + SUMS + c2, cs);
                            }
                        }
                        tc_wait_st();
                    }
                }
            }
            if (!ok) break;
            // column j's X in three words, two's complement
            struct X96 {
                uint32_t w0, w1, w2;
            };
            auto words = [&](int j) {
                return X96{x0[j], (uint32_t)x1[j], (uint32_t)((uint64_t)x1[j] >> 32)};
            };
            if (u.part >= 0) {  // part of a split tile
                constexpr int NW = EXACT ? 3 * HALF : 2 * HALF;
                const int w = warp - 2, sp = u.part % args.splits, first = u.part - sp;
                uint4 *mine = oz_part_at<NW>(args.part, u.part, w);
                if constexpr (EXACT) {
#pragma unroll
                    for (int j0 = 0; j0 < HALF; j0 += 4) {
                        const X96 a = words(j0), b = words(j0 + 1), c = words(j0 + 2), d = words(j0 + 3);
                        __stcg(mine + (j0 / 4) * 32, make_uint4(a.w0, b.w0, c.w0, d.w0));
                        __stcg(mine + ((HALF + j0) / 4) * 32, make_uint4(a.w1, b.w1, c.w1, d.w1));
                        __stcg(mine + ((2 * HALF + j0) / 4) * 32, make_uint4(a.w2, b.w2, c.w2, d.w2));
                    }
                } else {
#pragma unroll
                    for (int j0 = 0; j0 < HALF; j0 += 4) {
                        __stcg(mine + (j0 / 4) * 32,
                               make_uint4(__float_as_uint(accf[j0]), __float_as_uint(accf[j0 + 1]),
                                          __float_as_uint(accf[j0 + 2]), __float_as_uint(accf[j0 + 3])));
                        __stcg(mine + ((HALF + j0) / 4) * 32,
                               make_uint4(__float_as_uint(finite_comp(comp[j0])), __float_as_uint(finite_comp(comp[j0 + 1])),
                                          __float_as_uint(finite_comp(comp[j0 + 2])),
                                          __float_as_uint(finite_comp(comp[j0 + 3]))));
                    }
                }
                if (!oz_part_last(args.cnt, u.part / args.splits, w, args.splits)) continue;
                if constexpr (EXACT) {  // integers: any order gives the same sum
#pragma unroll 1
                    for (int o = 0; o < args.splits; ++o) {
                        if (o == sp) continue;
                        const uint4 *p = oz_part_at<NW>(args.part, first + o, w);
#pragma unroll
                        for (int j0 = 0; j0 < HALF; j0 += 4) {
                            const uint4 x = __ldcg(p + (j0 / 4) * 32), y = __ldcg(p + ((HALF + j0) / 4) * 32),
                                        z = __ldcg(p + ((2 * HALF + j0) / 4) * 32);
                            const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w},
                                           zs[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const int64_t hi = (int64_t)(((uint64_t)zs[e] << 32) | ys[e]);
                                const uint64_t lo = (uint64_t)x0[j0 + e] + xs[e];
                                x0[j0 + e] = (uint32_t)lo;
                                x1[j0 + e] += hi + (int64_t)(lo >> 32);
                            }
                        }
                    }
                } else {  // compensated float sums, always in the order of k
#pragma unroll
                    for (int j = 0; j < HALF; ++j) accf[j] = comp[j] = 0.f;
#pragma unroll 1
                    for (int o = 0; o < args.splits; ++o) {
                        const uint4 *p = oz_part_at<NW>(args.part, first + o, w);
#pragma unroll
                        for (int j0 = 0; j0 < HALF; j0 += 4) {
                            const uint4 x = __ldcg(p + (j0 / 4) * 32), y = __ldcg(p + ((HALF + j0) / 4) * 32);
                            const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                add_part(accf[j0 + e], comp[j0 + e], __uint_as_float(xs[e]), __uint_as_float(ys[e]));
                        }
                    }
                }
            }
            if constexpr (EXACT) {
                // Four conversions at a time, so that their integer sequences
                // interleave (one alone is a chain of dependent instructions):
                // in 64 bits where all of the warp's X fit, as they do unless K
                // is huge, and through the general routine where an exponent
                // leaves the plain range. A loop, whose columns move down to
                // the same registers each time: unrolled, the instructions
                // alone took longer to fetch than to run. S = 6, a tile's 16
                // columns per thread: 4800 cycles for 96-bit conversions that
                // handle every exponent, 2800 so; 4864 tiles of 4 k blocks
                // 178 -> 151 us, one tile of 4 k blocks (with its launch) 14.0
                // -> 11.7.
                constexpr int GQ = CX ? 2 : 4;  // output columns per group
                constexpr int NP = CX ? 2 : 1;  // parts per output column
                const uint64_t nanb = 0x7FF8000000000000ull;
                X96 xs[HALF];
#pragma unroll
                for (int j = 0; j < HALF; ++j) xs[j] = words(j);
#pragma unroll 1
                for (int j0 = 0; j0 < NCOL; j0 += GQ) {
                    uint64_t bits[GQ][NP];
                    int Eq[GQ];
                    bool plain = true, fit = true;
#pragma unroll
                    for (int q2 = 0; q2 < GQ; ++q2) {
                        Eq[q2] = erow + __shfl_sync(0xffffffffu, lexp, j0 + q2);
                        plain = plain && x96_plain_exponent(Eq[q2]);
#pragma unroll
                        for (int pp = 0; pp < NP; ++pp) fit = fit && x96_is_64(xs[NP * q2 + pp].w1, xs[NP * q2 + pp].w2);
                    }
                    if (__all_sync(0xffffffffu, plain && fit)) {
#pragma unroll
                        for (int q2 = 0; q2 < GQ; ++q2)
#pragma unroll
                            for (int pp = 0; pp < NP; ++pp) {
                                const X96 &w = xs[NP * q2 + pp];
                                bits[q2][pp] = x96_pack(x64_normalise(w.w0, w.w1), Eq[q2]);
                            }
                    } else if (__all_sync(0xffffffffu, plain)) {
#pragma unroll
                        for (int q2 = 0; q2 < GQ; ++q2)
#pragma unroll
                            for (int pp = 0; pp < NP; ++pp) {
                                const X96 &w = xs[NP * q2 + pp];
                                bits[q2][pp] = x96_pack(x96_normalise(w.w0, w.w1, w.w2), Eq[q2]);
                            }
                    } else {
#pragma unroll
                        for (int q2 = 0; q2 < GQ; ++q2)
#pragma unroll
                            for (int pp = 0; pp < NP; ++pp) {
                                const X96 &w = xs[NP * q2 + pp];
                                const double v = x96_ldexp_rn(w.w0, w.w1, w.w2, Eq[q2]);
                                bits[q2][pp] = Eq[q2] > OZ_NAN_EXP / 2 ? nanb : (uint64_t)__double_as_longlong(v);
                            }
                    }
#pragma unroll
                    for (int q2 = 0; q2 < GQ; ++q2) {
                        const int64_t off = rowoff + __shfl_sync(0xffffffffu, lcoff, j0 + q2);
                        if (!row_ok || !(cols >> (j0 + q2) & 1u)) continue;
                        const double v0 = __longlong_as_double((long long)bits[q2][0]);
                        if constexpr (CX) {
                            const double v1 = __longlong_as_double((long long)bits[q2][NP - 1]);
                            ((double2 *)Cl)[off] = make_double2(v0, v1);
                        } else {
                            ((double *)Cl)[off] = v0;
                        }
                    }
#pragma unroll
                    for (int j = 0; j + GQ * NP < HALF; ++j) xs[j] = xs[j + GQ * NP];
                }
            } else {
#pragma unroll
                for (int jj = 0; jj < NCOL; ++jj) {
                    const int64_t coff = __shfl_sync(0xffffffffu, lcoff, jj);
                    if (!row_ok || !(cols >> jj & 1u)) continue;
                    const int j = CX ? 2 * jj : jj;
                    const int64_t off = rowoff + coff;
                    if (CX) ((float2 *)Cl)[off] = make_float2(accf[j], accf[j + 1]);
                    else ((float *)Cl)[off] = accf[j];
                }
            }
        }
    };
    if (warp == 0) {
        produce();
    } else if (warp == 1 || (NI == 2 && warp == OZ_ISSUER2_WARP)) {
        if constexpr (WIDE) issue_wide();
        else issue_narrow();
    } else if (warp < 2 + OZ_EPI_WARPS) {
        epilogue();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"((uint32_t)TCOLS)
                     : "memory");
}

// =============================================================================
// Launches
// =============================================================================
// Per-device caches, safe for concurrent callers: the values are idempotent,
// so a race only repeats the query or the attribute call.
constexpr int OZ_MAX_DEVICES = 64;

inline int sm_count() {
    static std::atomic<int> count[OZ_MAX_DEVICES];
    int dev = 0;
    cudaGetDevice(&dev);
    const bool cached = dev >= 0 && dev < OZ_MAX_DEVICES;
    int n = cached ? count[dev].load(std::memory_order_relaxed) : 0;
    if (n <= 0) {
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 1;
        if (cached) count[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

template <typename K>
inline int set_smem_attr(K kern, int smem, std::atomic<bool> (&done)[OZ_MAX_DEVICES]) {
    int dev = 0;
    cudaGetDevice(&dev);
    const bool cached = dev >= 0 && dev < OZ_MAX_DEVICES;
    if (!cached || !done[dev].load(std::memory_order_acquire)) {
        MGB_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        if (cached) done[dev].store(true, std::memory_order_release);
    }
    return MGB_OK;
}

// Dispatch on (slices, exact, complex): BF16X3 is S = 3 and not exact.
#define OZ_DISPATCH(CALL)                                                        \
    if (!exact) return cx ? CALL(3, false, true) : CALL(3, false, false);       \
    switch (S) {                                                                 \
    case 3: return cx ? CALL(3, true, true) : CALL(3, true, false);             \
    case 4: return cx ? CALL(4, true, true) : CALL(4, true, false);             \
    case 5: return cx ? CALL(5, true, true) : CALL(5, true, false);             \
    case 6: return cx ? CALL(6, true, true) : CALL(6, true, false);             \
    case 7: return cx ? CALL(7, true, true) : CALL(7, true, false);             \
    case 8: return cx ? CALL(8, true, true) : CALL(8, true, false);             \
    }                                                                            \
    return fail(MGB_ERR_ARGUMENT, "unsupported slice count");

// The contraction of `job`, on a persistent grid (one CTA per SM, each
// walking its share of the units), in narrow tiles.
int oz_launch_one(int S, bool exact, bool cx, const OzJob &job, int64_t units, cudaStream_t s);
// The contraction of `job` with the slice count that the device chose (exact
// form; nothing when that is 0, the plain form, or not in job.cand).
int oz_launch_any(bool cx, const OzAnyJob &job, int64_t units, cudaStream_t s);
// In wide tiles, with the count that the device chose (nothing unless it is in
// job.cand) or job.S.
int oz_launch_wide(bool cx, const OzAnyJob &job, int64_t units, cudaStream_t s);
// Every contraction of a device table of one kernel variant.
int oz_launch_table(int S, bool exact, bool cx, const OzJob *jobs, const int64_t *start, int njobs, int64_t units,
                    cudaStream_t s);

}  // namespace mgb
