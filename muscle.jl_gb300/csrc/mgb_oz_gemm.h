// The tensor-core GEMM of the emulated forms over digit slices (OZAKI) or
// pieces (BF16X3), shared by its translation units: one contraction of a
// fixed slice count (mgb_oz_gemm_one.cu), one whose slice count the device
// chose (mgb_oz_gemm_any.cu), and a table of contractions
// (mgb_oz_gemm_table.cu).
#pragma once

#include <cuda.h>

#include <atomic>

#include "mgb_internal.h"
#include "mgb_ptx.h"
#include "mgb_x96.h"

namespace mgb {

constexpr int OZ_KC = 256;     // BF16X3: embedded k between readouts
constexpr int OZ_BM = 128;     // rows of A per CTA (TMEM lanes)
constexpr int OZ_BK = 32;      // k per stage (64-byte swizzled rows)
constexpr int OZ_EPI_WARPS = 8;
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
// warp 0 TMA, warp 1 MMA issuer (and TMEM owner), warps 2..9 epilogue,
// warp 10 second MMA issuer
constexpr int OZ_THREADS = 96 + 32 * OZ_EPI_WARPS;
constexpr int OZ_ISSUER2_WARP = 2 + OZ_EPI_WARPS;
constexpr int OZ_A_TILE = OZ_BM * OZ_BK * 2;  // 8192 bytes per slice
constexpr int OZ_SMEM_BUDGET = 220 * 1024;
constexpr int OZ_MAX_STAGES = 6;

// Columns per digit group (= embedded rows of B per CTA): two banks of S
// groups must fit the 512 TMEM columns, and one MMA covers at most 256.
// BF16X3 (S = 3, two float registers per column) takes 64; the exact forms
// keep 32, where their three 32-bit words per column stay in registers.
__host__ __device__ constexpr int oz_bn(int S, bool exact) { return (!exact && S <= 3) ? 64 : 32; }
__host__ __device__ constexpr int oz_b_tile(int S, bool exact) { return oz_bn(S, exact) * OZ_BK * 2; }  // bytes per slice
__host__ __device__ constexpr int oz_stage_bytes(int S, bool exact) { return S * (OZ_A_TILE + oz_b_tile(S, exact)); }
// Digit width and exact chunk length (in 32-wide k blocks) per slice count.
// W = 8 for S <= 6: |s1| <= 256, |si| <= 128, group bound max(d+1,4) 2^14, so a
// float32 accumulator stays exact over 4 blocks (128 k) for every d <= 7.
// W = 7 for S >= 7: group bound max(d+1,4) 2^12, exact over 8 blocks (256 k)
// for d <= 15. Both hold about the same number of mantissa bits (W S = 48 / 49).
__host__ __device__ constexpr int oz_digit_bits(int S) { return S <= 6 ? 8 : 7; }
__host__ __device__ constexpr int oz_chunk_blocks(int S) { return oz_digit_bits(S) == 8 ? 4 : 8; }
// k blocks between readouts
__host__ __device__ constexpr int oz_chunk(int S, bool exact) { return exact ? oz_chunk_blocks(S) : OZ_KC / OZ_BK; }
__host__ __device__ constexpr int oz_stages(int S, bool exact) {
    return (OZ_SMEM_BUDGET / oz_stage_bytes(S, exact)) < OZ_MAX_STAGES ? (OZ_SMEM_BUDGET / oz_stage_bytes(S, exact))
                                                                       : OZ_MAX_STAGES;
}
// two banks of S groups of oz_bn columns; bank bases at columns 0 and 256
__host__ __device__ constexpr int oz_tmem_cols(int) { return 512; }
// More than half of the SM's shared memory for every S, so one CTA (and one
// TMEM allocation) per SM.
__host__ __device__ constexpr int oz_smem_bytes(int S, bool exact) {
    return oz_stages(S, exact) * oz_stage_bytes(S, exact) + 1024 /*align*/ + 256 /*barriers*/;
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
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// NC consecutive columns (a multiple of 16), then wait for the loads
template <int NC>
__device__ __forceinline__ void tc_ld(uint32_t taddr, uint32_t (&v)[NC]) {
#pragma unroll
    for (int c = 0; c < NC; c += 16) tc_ld16_issue(taddr + c, v + c);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// 96-bit two's-complement accumulation (carry chain) and conversion.
__device__ __forceinline__ void add96(uint32_t &w0, uint32_t &w1, uint32_t &w2, uint32_t a0, uint32_t a1,
                                      uint32_t a2) {
    asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
        : "+r"(w0), "+r"(w1), "+r"(w2)
        : "r"(a0), "r"(a1), "r"(a2));
}
__device__ __forceinline__ void add64hi(uint32_t &w1, uint32_t &w2, uint32_t a1, uint32_t a2) {
    asm("add.cc.u32 %0, %0, %2;\n\taddc.u32 %1, %1, %3;" : "+r"(w1), "+r"(w2) : "r"(a1), "r"(a2));
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
    // units leave their sums in `part` and count in `cnt`; the last one adds
    // them up and writes the outputs.
    int32_t splits, kbs;
    int64_t full;
    uint32_t *part;
    int32_t *cnt;
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

// ---- sums of a split tile ------------------------------------------------------
// An epilogue warp's share of a unit: NW words per lane, as 16-byte vectors
// of consecutive lanes.
template <int NW>
__device__ __forceinline__ uint4 *oz_part_at(uint32_t *part, int unit, int w) {
    return (uint4 *)part + (((int64_t)unit * OZ_EPI_WARPS + w) * (NW / 4)) * 32 + threadIdx.x % 32;
}
// Publishes this warp's share and counts it; true for the warp that finds all
// `splits` shares of its tile published. Nobody waits for anybody.
__device__ __forceinline__ bool oz_part_last(int32_t *cnt, int tile, int w, int splits) {
    __threadfence();
    __syncwarp();
    int old = 0;
    if (threadIdx.x % 32 == 0) old = atomicAdd(cnt + tile * OZ_EPI_WARPS + w, 1);
    const bool last = __shfl_sync(0xffffffffu, old, 0) == splits - 1;
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
template <int S, bool EXACT, bool CX, typename Src>
__device__ __forceinline__ void oz_gemm_body(const Src &src) {
    constexpr int W = oz_digit_bits(S);  // digit width (EXACT)
    constexpr int KCB = oz_chunk(S, EXACT);  // k blocks per chunk
    constexpr int NST = oz_stages(S, EXACT);
    constexpr int STAGE = oz_stage_bytes(S, EXACT);
    constexpr int BN = oz_bn(S, EXACT);  // columns per digit group, embedded B rows per CTA
    constexpr int HALF = BN / 2;     // columns per group read by one epilogue warp
    constexpr int TCOLS = oz_tmem_cols(S);
    constexpr int BANK = TCOLS / 2;  // TMEM column offset of the second bank
    static_assert(NST >= 2, "need at least two pipeline stages");
    static_assert(BN * S <= BANK && TCOLS <= 512, "two banks must fit in TMEM");
    static_assert(BN * S <= 256, "one MMA covers at most 256 columns");
    static_assert(HALF % 16 == 0, "epilogue reads 16 columns at a time");
    // MMA-issuing threads. Each mbarrier poll by an issuing thread stalls it
    // for ~150 cycles while the tensor core's queue holds only ~200 cycles of
    // MMAs, so a single issuer leaves a bubble at every k block. Two issuers
    // (warps 1 and 10) take alternate k blocks and keep the queue fed while
    // the other polls. Their MMAs into a bank interleave in an unspecified
    // order, which changes nothing for the exact integer sums of the OZAKI
    // form; BF16X3 sums round, so it keeps one issuer and stays deterministic.
    constexpr int NI = EXACT ? 2 : 1;

    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *bars = (uint64_t *)(smem + NST * STAGE);
    uint64_t *full = bars;               // [2 NST] see full_idx
    uint64_t *empty = bars + 2 * NST;    // [NST]
    uint64_t *acc_full = bars + 3 * NST; // [2] bank filled (one commit per issuer)
    uint64_t *acc_empty = acc_full + 2;  // [2] bank read and cleared (one arrive per epilogue warp)
    uint64_t *done = acc_empty + 2;      // [2] per issuer: all its MMAs complete
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
            mbar_init(smem_u32(acc_empty + b), OZ_EPI_WARPS);
            mbar_init(smem_u32(done + b), 1);
        }
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

    if (warp == 0) {
        // ---------------- TMA producer ----------------
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
    } else if (warp == 1 || (NI == 2 && warp == OZ_ISSUER2_WARP)) {
        // ---------------- MMA issuers ----------------
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
    } else if (warp < 2 + OZ_EPI_WARPS) {
        // ---------------- epilogue ----------------
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
            // holds column j of this warp's half, broadcast by shuffles).
            constexpr int NCOL = CX ? HALF / 2 : HALF;
            const bool row_ok = row < args.M;
            int64_t rowoff = 0;
            int erow = 0;
            bool badrow = false;
            if (row_ok) {
                rowoff = (args.cptr ? 0 : group_offset(args.gl, 2, l)) + group_offset(args.gm, 2, row);
                if (EXACT) {
                    const int be = args.expA[(int64_t)l * args.M + row];
                    badrow = be == 0x7FF;
                    erow = be == 0 ? -1022 : be - 1022;
                }
            }
            long long lcoff = 0;
            int lexp = -1;  // the column's exponent (0 without one), -1 beyond the output
            {
                const int64_t ne = n0 + HALF * h + (int64_t)lane * (CX ? 2 : 1);
                if (lane < NCOL && ne < args.Ne) {
                    const int64_t n = CX ? (ne >> 1) : ne;
                    lcoff = group_offset(args.gn, 2, n);
                    lexp = EXACT ? args.expB[(int64_t)l * args.N + n] : 0;
                }
            }
            void *const Cl = args.cptr ? args.cptr[l] : args.C;
            // EXACT: one 96-bit two's-complement integer per output column,
            // X = sum_d G_d 2^(W (S + 1 - d)), held in w0 (bits 0-31), w1, w2.
            uint32_t w0[EXACT ? HALF : 1], w1[EXACT ? HALF : 1], w2[EXACT ? HALF : 1];
            // BF16X3: Kahan-compensated float32 sum over the chunks
            float accf[EXACT ? 1 : HALF], comp[EXACT ? 1 : HALF];
#pragma unroll
            for (int j = 0; j < HALF; ++j) {
                if (EXACT) {
                    w0[j] = 0;
                    w1[j] = 0;
                    w2[j] = 0;
                } else {
                    accf[j] = 0.f;
                    comp[j] = 0.f;
                }
            }
#pragma unroll 1
            for (int c = 0; c < nchunks; ++c, ++C) {
                const uint32_t bank = C & 1u;
                // warp-uniform outcome: the warp-collective loads below need every lane
                if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(acc_full + bank), (C >> 1) & 1u, abort_flag, status))) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t tb = tbase + bank * BANK;
                if constexpr (EXACT) {
#pragma unroll
                    for (int g = 0; g < S; ++g) {
                        uint32_t v[HALF];
                        tc_ld<HALF>(tb + BN * g, v);
#pragma unroll
                        for (int c2 = 0; c2 < HALF; c2 += 16) tc_st16_zero(tb + BN * g + c2);
                        if (g == S - 1) {  // every group of the bank read and cleared
                            tc_wait_st();
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(smem_u32(acc_empty + bank));
                        }
                        const int sh = W * (S - 1 - g);  // W (S + 1 - d), d = g + 2
                        if (sh < 32) {
#pragma unroll
                            for (int j = 0; j < HALF; ++j) {
                                int64_t x = (int64_t)__float2int_rn(__uint_as_float(v[j])) << sh;
                                add96(w0[j], w1[j], w2[j], (uint32_t)x, (uint32_t)((uint64_t)x >> 32),
                                      x < 0 ? 0xFFFFFFFFu : 0u);
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < HALF; ++j) {
                                int64_t x = (int64_t)__float2int_rn(__uint_as_float(v[j])) << (sh - 32);
                                add64hi(w1[j], w2[j], (uint32_t)x, (uint32_t)((uint64_t)x >> 32));
                            }
                        }
                    }
                } else {
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
                }
            }
            if (!ok) break;
            if (u.part >= 0) {  // part of a split tile
                constexpr int NW = EXACT ? 3 * HALF : 2 * HALF;
                const int w = warp - 2, sp = u.part % args.splits, first = u.part - sp;
                uint4 *mine = oz_part_at<NW>(args.part, u.part, w);
#pragma unroll
                for (int i = 0; i < NW / 4; ++i) {
                    uint32_t v[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int k = 4 * i + e;  // a constant: the loops are unrolled
                        if constexpr (EXACT) v[e] = k < HALF ? w0[k % HALF] : k < 2 * HALF ? w1[k % HALF] : w2[k % HALF];
                        else v[e] = __float_as_uint(k < HALF ? accf[k % HALF] : comp[k % HALF]);
                    }
                    __stcg(mine + i * 32, make_uint4(v[0], v[1], v[2], v[3]));
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
                            add96(w0[j0], w1[j0], w2[j0], x.x, y.x, z.x);
                            add96(w0[j0 + 1], w1[j0 + 1], w2[j0 + 1], x.y, y.y, z.y);
                            add96(w0[j0 + 2], w1[j0 + 2], w2[j0 + 2], x.z, y.z, z.z);
                            add96(w0[j0 + 3], w1[j0 + 3], w2[j0 + 3], x.w, y.w, z.w);
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
                            for (int e = 0; e < 4; ++e) {
                                const float t = __uint_as_float(xs[e]) - (__uint_as_float(ys[e]) + comp[j0 + e]);
                                const float s2 = accf[j0 + e] + t;
                                comp[j0 + e] = (s2 - accf[j0 + e]) - t;
                                accf[j0 + e] = s2;
                            }
                        }
                    }
                }
            }
            if constexpr (EXACT) {
                // Four conversions at a time through the straight-line routine,
                // so that their integer sequences interleave (one conversion
                // alone is a chain of dependent instructions); a group with a
                // subnormal result (rare) goes through the general routine;
                // then the group's stores.
                constexpr int GQ = CX ? 2 : 4;  // output columns per group
                constexpr int NP = CX ? 2 : 1;  // parts per output column
                const uint64_t nanb = 0x7FF8000000000000ull;
#pragma unroll
                for (int j0 = 0; j0 < NCOL; j0 += GQ) {
                    uint64_t bits[GQ][NP];
                    int Eq[GQ];
                    bool slow = false;
#pragma unroll
                    for (int q2 = 0; q2 < GQ; ++q2) {
                        const int bc = __shfl_sync(0xffffffffu, lexp, j0 + q2);
                        Eq[q2] = erow + (bc == 0 ? -1022 : bc - 1022) - W * (S + 1);
#pragma unroll
                        for (int pp = 0; pp < NP; ++pp) {
                            const int j = NP * (j0 + q2) + pp;
                            bits[q2][pp] = x96_ldexp_bits_fast(w0[j], w1[j], w2[j], Eq[q2], slow);
                        }
                    }
                    if (slow) {
#pragma unroll
                        for (int q2 = 0; q2 < GQ; ++q2)
#pragma unroll
                            for (int pp = 0; pp < NP; ++pp) {
                                const int j = NP * (j0 + q2) + pp;
                                bits[q2][pp] =
                                    (uint64_t)__double_as_longlong(x96_ldexp_rn_general(w0[j], w1[j], w2[j], Eq[q2]));
                            }
                    }
#pragma unroll
                    for (int q2 = 0; q2 < GQ; ++q2) {
                        const int jj = j0 + q2;
                        const int64_t coff = __shfl_sync(0xffffffffu, lcoff, jj);
                        const int bc = __shfl_sync(0xffffffffu, lexp, jj);
                        if (!row_ok || bc < 0) continue;
                        const int64_t off = rowoff + coff;
                        const bool bad = badrow || bc == 0x7FF;
                        const double v0 = __longlong_as_double((long long)(bad ? nanb : bits[q2][0]));
                        if constexpr (CX) {
                            const double v1 = __longlong_as_double((long long)(bad ? nanb : bits[q2][NP - 1]));
                            ((double2 *)Cl)[off] = make_double2(v0, v1);
                        } else {
                            ((double *)Cl)[off] = v0;
                        }
                    }
                }
            } else {
#pragma unroll
                for (int jj = 0; jj < NCOL; ++jj) {
                    const int64_t coff = __shfl_sync(0xffffffffu, lcoff, jj);
                    const int bc = __shfl_sync(0xffffffffu, lexp, jj);
                    if (!row_ok || bc < 0) continue;
                    const int j = CX ? 2 * jj : jj;
                    const int64_t off = rowoff + coff;
                    if (CX) ((float2 *)Cl)[off] = make_float2(accf[j], accf[j + 1]);
                    else ((float *)Cl)[off] = accf[j];
                }
            }
        }
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
// walking its share of the units).
int oz_launch_one(int S, bool exact, bool cx, const OzJob &job, int64_t units, cudaStream_t s);
// The contraction of `job` with the slice count that the device chose (exact
// form; nothing when that is 0, the plain form).
int oz_launch_any(bool cx, const OzAnyJob &job, int64_t units, cudaStream_t s);
// Every contraction of a device table of one kernel variant.
int oz_launch_table(int S, bool exact, bool cx, const OzJob *jobs, const int64_t *start, int njobs, int64_t units,
                    cudaStream_t s);

}  // namespace mgb
