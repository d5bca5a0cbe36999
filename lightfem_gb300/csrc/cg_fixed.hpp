// Fixed-point sums of the resident PCG (cg_resident.cu): a share of a dot product as
// integer limbs that threads and warps add, a CTA's sum as two counted 64-bit words that
// the CTAs add, and the words' sums back as a total.  Arithmetic only, for the device and
// for the host (a test runs it there).
#pragma once

#include <cmath>
#include <cstring>

#ifdef __CUDACC__
#define LF_FIXED __host__ __device__ __forceinline__
#else
#define LF_FIXED inline
#endif

namespace lfgpu {

// Each rounded on its own, on either side.
#ifdef __CUDA_ARCH__
__device__ __forceinline__ float fx_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fx_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fx_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ int fx_bits(float v) { return __float_as_int(v); }
__device__ __forceinline__ float fx_float(int v) { return __int_as_float(v); }
__device__ __forceinline__ long long fx_bits(double v) { return __double_as_longlong(v); }
__device__ __forceinline__ double fx_double(long long v) { return __longlong_as_double(v); }
__device__ __forceinline__ int fx_clz(long long v) { return __clzll(v); }
#else
LF_FIXED float fx_mul(float a, float b) { return a * b; }
LF_FIXED float fx_add(float a, float b) { return a + b; }
LF_FIXED float fx_fma(float a, float b, float c) { return std::fma(a, b, c); }
template <typename To, typename From>
LF_FIXED To fx_cast(From v) {
    To t;
    std::memcpy(&t, &v, sizeof(t));
    return t;
}
LF_FIXED int fx_bits(float v) { return fx_cast<int>(v); }
LF_FIXED float fx_float(int v) { return fx_cast<float>(v); }
LF_FIXED long long fx_bits(double v) { return fx_cast<long long>(v); }
LF_FIXED double fx_double(long long v) { return fx_cast<double>(v); }
LF_FIXED int fx_clz(long long v) { return v == 0 ? 64 : __builtin_clzll(static_cast<unsigned long long>(v)); }
#endif

// A share of a sum is cut into limbs of 21 bits (FP32 pairs: three, in
// units of 2^-15, 2^-36 and 2^-56 of the scale 2^e) or 22 bits (FP64: four, in units
// of 2^-78, 2^-56, 2^-34 and 2^-12), each a 32-bit integer that a warp adds with one
// instruction: no more than 1024 threads (FP32 pairs) or 512 (FP64), then no sum of limbs
// overflows.
template <bool MIXED>
constexpr int kLimbs = MIXED ? 3 : 4;
template <bool MIXED>
constexpr int kLimbThreads = MIXED ? 1024 : 512;
constexpr int kScaleBits = 78;   // FP64: bits below the scale
constexpr int kNoScale = 1 << 20;

// Exponent of a positive normal total with room for the arithmetic around it, or kNoScale.
LF_FIXED int exponent_of(double v) {
    const int e = static_cast<int>(static_cast<unsigned long long>(fx_bits(v)) >> 52);  // the sign counts too
    return e > 123 && e < 1923 ? e - 1023 : kNoScale;
}
LF_FIXED int exponent_of_pair(float hi) {
    const int e = static_cast<int>(static_cast<unsigned>(fx_bits(hi)) >> 23);
    return e > 0 && e < 250 ? e - 127 : kNoScale;
}
// FP32 pairs: 2^-e, and 2^(e - 36) as a product of two floats (e in [-126, 122]).
LF_FIXED void pair_scale(int e, float& up, float (&down)[2]) {
    up = fx_float((127 - e) << 23);
    const int n = e - 36, a = n >> 1;
    down[0] = fx_float((a + 127) << 23);
    down[1] = fx_float((n - a + 127) << 23);
}

// The limbs of a thread's share; false when it is out of range.  FP32 pair: each limb
// is the remainder so far rounded to the limb's unit, by adding 1.5 x 2^23, and the
// remainders are exact.  |share| < 2^5 of the scale.
LF_FIXED bool pair_limbs(float up, float vhi, float vlo, int (&l)[3]) {
    constexpr float kRound = 12582912.f;
    constexpr int kBits = 0x4b400000;
    const float hi = fx_mul(vhi, up), lo = fx_mul(vlo, up);
    const float a = fx_fma(hi, 0x1p15f, kRound);
    const float r = fx_fma(fx_add(a, -kRound), -0x1p-15f, hi);
    const float b = fx_fma(r, 0x1p36f, kRound), c = fx_fma(lo, 0x1p36f, kRound);
    const float s = fx_fma(fx_add(b, -kRound), -0x1p-36f, r), t = fx_fma(fx_add(c, -kRound), -0x1p-36f, lo);
    l[2] = fx_bits(a) - kBits;
    l[1] = (fx_bits(b) - kBits) + (fx_bits(c) - kBits);
    l[0] = fx_bits(fx_fma(fx_add(s, t), 0x1p56f, kRound)) - kBits;
    return fabsf(hi) < 0x1p5f && fabsf(lo) < 0x1p-17f;
}
// FP64: the mantissa shifted to its place in units of 2^-78 of the scale.  |share| <
// 2^9 of the scale.
LF_FIXED bool fp64_limbs(int e, double v, int (&l)[4]) {
    const unsigned long long b = static_cast<unsigned long long>(fx_bits(v));
    const int ex = static_cast<int>((b >> 52) & 0x7ff);
    const unsigned long long m = (b & 0xfffffffffffffull) | (ex ? 1ull << 52 : 0ull);
    const int n = (ex > 1 ? ex : 1) - 1075 + kScaleBits - e;
    const bool ok = ex != 0x7ff && (m == 0 || n <= 34);
    const int up = n < 0 ? 0 : n > 34 ? 34 : n, dn = -n < 0 ? 0 : -n > 63 ? 63 : -n;
    const unsigned long long lo = dn > 0 ? (m + (1ull << (dn - 1))) >> dn : m << up;
    const unsigned long long hi = up > 0 ? m >> (64 - up) : 0ull;
    constexpr unsigned mask = 0x3fffffu;
    const int l0 = static_cast<int>(static_cast<unsigned>(lo) & mask);
    const int l1 = static_cast<int>(static_cast<unsigned>(lo >> 22) & mask);
    const int l2 = static_cast<int>((static_cast<unsigned>(lo >> 44) | (static_cast<unsigned>(hi) << 20)) & mask);
    const int l3 = static_cast<int>(hi >> 2);
    const int sign = static_cast<int>(static_cast<long long>(b) >> 63);  // 0 or -1
    l[0] = (l0 ^ sign) - sign;
    l[1] = (l1 ^ sign) - sign;
    l[2] = (l2 ^ sign) - sign;
    l[3] = (l3 ^ sign) - sign;
    return ok;
}

// A CTA's sum of a quantity travels in two words, low and high (a sector holds the four
// words of r.r and r.z): arrivals in the top byte, CTAs out of range in the next, and
// below them 40 bits of the sum, or the rest plus 2^39; 48 bits hold 255 CTAs' shares.
// Units: 2^-56 of the scale (pairs), 2^-70 (FP64, rounded from the threads' 2^-78: with 152
// CTAs of 512 threads a total of 2^-10 of the scale is off by less than 2^-51 of itself, as
// little as a sum in FP64 leaves; with units of 2^-62 it was 2^-44).
constexpr long long kHighBias = 1ll << 39;
constexpr long long kLowMask = (1ll << 40) - 1;
template <bool MIXED>
LF_FIXED unsigned long long sum_word(const int* l, bool high, bool bad) {
    long long lo, hi;
    if (MIXED) {
        // The top limb goes to the high part as it is: at 2^22 units and more (2^7 of the
        // scale) it does not fit beside the others in 64 bits.
        lo = static_cast<long long>(l[0]) + static_cast<long long>(l[1]) * (1ll << 20);
        hi = static_cast<long long>(l[2]) * 2;
    } else {
        hi = static_cast<long long>(l[2]) + (static_cast<long long>(l[3]) << 22);  // units of 2^44
        lo = (static_cast<long long>(l[0]) + (static_cast<long long>(l[1]) << 22) + 128) >> 8;
        lo += (hi & 15) << 36;
        hi >>= 4;
    }
    hi += lo >> 40;
    lo &= kLowMask;
    bad = bad || hi >= kHighBias || hi < -kHighBias;
    return (1ull << 56) | (bad ? 1ull << 48 : 0ull) |
           (high ? (bad ? 0ull : static_cast<unsigned long long>(hi + kHighBias)) : static_cast<unsigned long long>(lo));
}

// A quantity's total from its two words' sums over n CTAs; false when it is not positive
// and within ten bits of the scale (then it is formed in FP64).
LF_FIXED void word_parts(unsigned long long low, unsigned long long high, int n, long long& lo, long long& hi) {
    lo = static_cast<long long>(low & 0xffffffffffffull);
    hi = static_cast<long long>(high & 0xffffffffffffull) - n * kHighBias;
}
LF_FIXED bool pair_total(const float (&down)[2], unsigned long long low, unsigned long long high, int n, float& out_hi,
                         float& out_lo) {
    long long lo, hi;
    word_parts(low, high, n, lo, hi);
    const bool ok = hi > -(1ll << 20) && hi < (1ll << 20);
    const long long s = static_cast<long long>((static_cast<unsigned long long>(hi) << 40)) + lo;  // units of 2^-56
    // Parts of 20 or 21 bits, exact in FP32; their sum as a pair in units of 2^-36.
    const float f2 = static_cast<float>(static_cast<int>(s >> 41));
    const float f1 = static_cast<float>(static_cast<int>(s >> 20) & 0x1fffff);
    const float f0 = static_cast<float>(static_cast<int>(s) & 0xfffff);
    const float h = fx_fma(f2, 0x1p21f, f1);
    const float l = fx_fma(f0, 0x1p-20f, fx_add(fx_fma(f2, 0x1p21f, -h), f1));
    out_hi = fx_mul(fx_mul(h, down[0]), down[1]);
    out_lo = fx_mul(fx_mul(l, down[0]), down[1]);
    return ok && s >= (1ll << 46);
}
LF_FIXED bool fp64_total(int e, unsigned long long low, unsigned long long high, int n, double& out) {
    long long lo, hi;
    word_parts(low, high, n, lo, hi);
    hi += lo >> 40;
    lo &= kLowMask;
    const bool ok = hi >= (1ll << 20) && hi < (1ll << 45);  // units of 2^-30
    const int lead = fx_clz(hi);  // 19 to 43
    const unsigned long long w = (static_cast<unsigned long long>(hi) << lead) |
                                 ((static_cast<unsigned long long>(lo) << 24) >> ((64 - lead) & 63));
    const unsigned long long m = (w >> 11) + ((w >> 10) & 1);  // 53 bits, rounded
    out = fx_double(static_cast<long long>(static_cast<unsigned long long>(1023 + 33 - lead + e - 1) << 52) +
                    static_cast<long long>(m));
    return ok;
}

}  // namespace lfgpu
