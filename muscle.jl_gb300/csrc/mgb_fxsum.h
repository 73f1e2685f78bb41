// Fixed-point sums of float64 values on the integer pipes, for the unary
// reductions (traces, partial sums) of Float64 / ComplexF64 tensors. GB300
// retires about two FP64 operations per clock per SM, so a sum that adds one
// FP64 value per element is bound by the FP64 pipe at about half the HBM
// rate. Here each value is aligned to the running largest exponent and added
// into a 128-bit two's-complement integer with integer instructions only.
//
// The sum is A * 2^(e - 1075 - kFxFrac): e is the largest biased exponent
// seen (at least 1, the exponent of the subnormals), A a 128-bit integer.
// A value with biased exponent be contributes its 53-bit significand shifted
// left by kFxFrac - (e - be) (right when that is negative); values within
// kFxFrac binades of the largest are added exactly, smaller ones are
// truncated below 2^-kFxFrac units in the last place of the largest (a
// relative 2^-62 of the largest term per term, where an FP64 sum rounds by
// up to 2^-53 of the running sum per term). Contributions stay below 2^63,
// so 2^63 of them cannot overflow A. The result is rounded once, to nearest
// with ties to even. Inf and NaN elements set flags that decide the result
// as in an FP64 sum (Inf, -Inf, or NaN for NaN or Inf - Inf). Host and
// device alike, so that the arithmetic is checked on the CPU against exact
// rational sums.
#pragma once

#include <cstdint>
#include <cstring>

#include "mgb_x96.h"

namespace mgb {

constexpr int kFxFrac = 10;

// Non-finite elements seen, as flags (integer work, so that no FP64
// instruction sits in the per-element path, not even a predicated one).
constexpr uint32_t kFxPosInf = 1, kFxNegInf = 2, kFxNaN = 4;

struct FxSum {
    uint64_t lo;
    int64_t hi;
    int32_t e;
    uint32_t flags;  // kFxPosInf | kFxNegInf | kFxNaN
};

MGB_HD uint64_t fx_bits(double x) {
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t b;
    std::memcpy(&b, &x, sizeof b);
    return b;
#endif
}

MGB_HD FxSum fx_zero() { return FxSum{0ull, 0ll, 1, 0u}; }

// A >>= d (arithmetic, d >= 0)
MGB_HD void fx_shr(FxSum &a, int d) {
    if (d <= 0) return;
    if (d >= 128) {
        a.lo = a.hi < 0 ? ~0ull : 0ull;
        a.hi = a.hi < 0 ? -1ll : 0ll;
    } else if (d >= 64) {
        a.lo = (uint64_t)(a.hi >> (d - 64));
        a.hi = a.hi >> 63;
    } else {
        a.lo = (a.lo >> d) | ((uint64_t)a.hi << (64 - d));
        a.hi = a.hi >> d;
    }
}

MGB_HD void fx_add128(FxSum &a, uint64_t lo, uint64_t hi) {
    const uint64_t s = a.lo + lo;
    const uint64_t carry = s < lo ? 1ull : 0ull;
    a.lo = s;
    a.hi = (int64_t)((uint64_t)a.hi + hi + carry);
}

// The signed significand scaled by 2^kFxFrac (below 2^63), shifted right
// (arithmetically) by the distance to the largest exponent, and added into
// the 128-bit sum with its sign extended. Straight-line apart from the two
// rare cases: a non-finite value, a new largest exponent.
MGB_HD void fx_push(FxSum &a, double x) {
    const uint64_t b = fx_bits(x);
    const int be = (int)((b >> 52) & 0x7FF);
    if (be == 0x7FF) {
        a.flags |= (b & 0xFFFFFFFFFFFFFull) ? kFxNaN : ((b >> 63) ? kFxNegInf : kFxPosInf);
        return;
    }
    const int bn = be ? be : 1;  // subnormals share the exponent of 2^-1022
    if (bn > a.e) {
        fx_shr(a, bn - a.e);
        a.e = bn;
    }
    const uint64_t m = (b & 0xFFFFFFFFFFFFFull) | ((uint64_t)(be != 0) << 52);
    const int64_t sgn = (int64_t)b >> 63;  // 0 or -1
    const int64_t v = ((int64_t)(m << kFxFrac) ^ sgn) - sgn;
    const int d = a.e - bn < 63 ? a.e - bn : 63;
    const int64_t c = v >> d;
    fx_add128(a, (uint64_t)c, (uint64_t)(c >> 63));
}

MGB_HD void fx_merge(FxSum &a, FxSum b) {
    if (b.e > a.e) {
        fx_shr(a, b.e - a.e);
        a.e = b.e;
    } else {
        fx_shr(b, a.e - b.e);
    }
    fx_add128(a, b.lo, (uint64_t)b.hi);
    a.flags |= b.flags;
}

// A running sum as the reduction kernels keep it: A = lo + hi * 2^32 + neg.
// Each value's aligned magnitude, two 32-bit words, is complemented when it is
// negative (~c = -c - 1; `neg` counts the missing ones) and its words go to two
// 64-bit sums, one multiply-add each on the FMA pipe: the 128-bit add with its
// carries and sign extension costs twice as many instructions on the integer
// ALU, the pipe that bounds these sums. Values are aligned to the largest
// exponent of a group first, so that the rare work (a new largest exponent,
// Inf, NaN) is one test per group. Words stay below 2^32, so 2^31 values fit.
// Values within kFxFrac binades of the largest are exact as in fx_push;
// smaller ones are truncated towards zero.
struct FxAcc {
    uint64_t lo;
    int64_t hi;
    int32_t neg;
    int32_t e;
    uint32_t flags;
    uint32_t one;  // 1, opaque to the compiler (it would turn the multiply-adds into adds)
};

MGB_HD FxAcc fx_acc_zero() {
    uint32_t one;
#if defined(__CUDA_ARCH__)
    asm volatile("mov.u32 %0, 1;" : "=r"(one));
#else
    one = 1;
#endif
    return FxAcc{0ull, 0ll, 0, 1, 0u, one};
}
MGB_HD FxSum fx_acc_sum(const FxAcc &a) {
    FxSum r{0ull, 0ll, a.e, a.flags};
    fx_add128(r, a.lo, 0ull);
    fx_add128(r, (uint64_t)a.hi << 32, (uint64_t)(a.hi >> 32));
    fx_add128(r, (uint64_t)(int64_t)a.neg, (uint64_t)((int64_t)a.neg >> 63));
    return r;
}
// Aligns the sum to the larger exponent e.
MGB_HD void fx_acc_rise(FxAcc &a, int e) {
    FxSum r = fx_acc_sum(a);
    fx_shr(r, e - a.e);
    a.lo = r.lo & 0xFFFFFFFFull;
    a.hi = (int64_t)((r.lo >> 32) | ((uint64_t)r.hi << 32));
    a.neg = 0;
    a.e = e;
}
MGB_HD int fx_bexp(uint64_t b) { return (int)((uint32_t)(b >> 52) & 0x7FFu); }
// Adds a finite value whose biased exponent is at most a.e.
MGB_HD void fx_acc_add(FxAcc &a, uint64_t b) {
    const uint32_t bl = (uint32_t)b, bh = (uint32_t)(b >> 32);
    const int be = (int)((bh >> 20) & 0x7FFu);
    const uint32_t mh = (bh & 0xFFFFFu) | (be ? 0x100000u : 0u);
    const uint64_t m = (((uint64_t)mh << 32) | bl) << kFxFrac;  // below 2^63
    const int d = a.e - (be > 1 ? be : 1);
    const uint64_t c = m >> (d < 63 ? d : 63);
    const int32_t s = (int32_t)bh >> 31;
    const uint32_t cl = (uint32_t)c ^ (uint32_t)s;
    const int32_t ch = (int32_t)((uint32_t)(c >> 32) ^ (uint32_t)s);
#if defined(__CUDA_ARCH__)
    asm("mad.wide.u32 %0, %1, %2, %0;" : "+l"(a.lo) : "r"(cl), "r"(a.one));
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(a.hi) : "r"(ch), "r"(a.one));
#else
    a.lo += cl;
    a.hi += ch;
#endif
    a.neg -= s;
}
// Adds N values.
template <int N>
MGB_HD void fx_acc_push(FxAcc &a, const double (&x)[N]) {
    uint64_t b[N];
    int m = 0;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int i = 0; i < N; ++i) {
        b[i] = fx_bits(x[i]);
        const int be = fx_bexp(b[i]);
        m = be > m ? be : m;
    }
    if (m > a.e) {
        if (m == 0x7FF) {  // Inf or NaN among them: flags; the others as usual
            m = 0;
            for (int i = 0; i < N; ++i) {
                const int be = fx_bexp(b[i]);
                if (be == 0x7FF) {
                    a.flags |= (b[i] & 0xFFFFFFFFFFFFFull) ? kFxNaN : ((b[i] >> 63) ? kFxNegInf : kFxPosInf);
                    b[i] = 0;
                } else if (be > m) {
                    m = be;
                }
            }
        }
        if (m > a.e) fx_acc_rise(a, m);
    }
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int i = 0; i < N; ++i) fx_acc_add(a, b[i]);
}

// A * 2^(e - 1075 - kFxFrac) rounded to float64 (nearest, ties to even),
// with overflow to infinity and subnormal results; a zero sum gives +0.
MGB_HD double fx_value(const FxSum &a) {
    if (a.flags) {  // as an FP64 sum: Inf - Inf and any NaN give NaN
        const bool nan = (a.flags & kFxNaN) || (a.flags & (kFxPosInf | kFxNegInf)) == (kFxPosInf | kFxNegInf);
        return x96_bits_to_double(nan ? 0x7FF8000000000000ull
                                      : ((a.flags & kFxNegInf) ? 0xFFF0000000000000ull : 0x7FF0000000000000ull));
    }
    const bool neg = a.hi < 0;
    uint64_t ml = a.lo, mh = (uint64_t)a.hi;
    if (neg) {
        ml = ~ml + 1ull;
        mh = ~mh + (ml == 0 ? 1ull : 0ull);
    }
    if (mh == 0 && ml == 0) return 0.0;
    const int p = mh ? 127 - x96_clz64(mh) : 63 - x96_clz64(ml);  // leading one
    int be = p + a.e - 1075 - kFxFrac + 1023;                      // biased exponent of the result
    uint64_t bits;
    if (be >= 1) {
        const int sh = 127 - p;  // leading one to bit 127
        uint64_t nh, nl;
        if (sh >= 64) {
            nh = ml << (sh - 64);
            nl = 0;
        } else if (sh > 0) {
            nh = (mh << sh) | (ml >> (64 - sh));
            nl = ml << sh;
        } else {
            nh = mh;
            nl = ml;
        }
        uint64_t mant = nh >> 11;  // bits 127..75: 53 bits with the leading one
        const bool round = (nh >> 10) & 1ull;
        const bool sticky = (nh & 0x3FFull) != 0 || nl != 0;
        if (round && (sticky || (mant & 1ull))) {
            ++mant;
            if (mant == (1ull << 53)) {
                mant >>= 1;
                ++be;
            }
        }
        if (be >= 2047) return x96_bits_to_double((neg ? 1ull << 63 : 0ull) | 0x7FF0000000000000ull);
        bits = ((uint64_t)be << 52) | (mant & 0xFFFFFFFFFFFFFull);
    } else {
        // subnormal: round(|A| * 2^(e - 1 - kFxFrac)) units of 2^-1074
        const int sh = kFxFrac + 1 - a.e;
        uint64_t q;
        if (sh <= 0) {
            q = ml << (-sh);  // exact: the result is below 2^52 units
        } else {
            q = (ml >> sh) | (sh < 64 ? (mh << (64 - sh)) : 0ull);
            const bool round = (ml >> (sh - 1)) & 1ull;
            const bool sticky = sh > 1 && (ml & ((1ull << (sh - 1)) - 1ull)) != 0;
            if (round && (sticky || (q & 1ull))) ++q;  // 2^52 becomes the smallest normal
        }
        bits = q;
    }
    if (neg) bits |= 1ull << 63;
    return x96_bits_to_double(bits);
}

}  // namespace mgb
