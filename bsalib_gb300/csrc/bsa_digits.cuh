// bsa_digits.cuh -- FP64 operands as base-256 digits for the tensor cores (the error-free splitting of
// bsa_pair64_tc.cu, which derives it): cutting values into digits, the stacked digit MMA and the
// combination of the level sums.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "bsa_tc.cuh"

namespace bsa {
namespace p64 {

using namespace tc;

constexpr int kDig = 8;            // digits per operand
constexpr int kPassMax = 128;      // k of one exact pass: 8 x 128 products of at most 2^14 within 2^24
constexpr int kBad = 1 << 20;      // exponent of a row left to the FP64 pipe
constexpr int kNone = -(1 << 20);  // of a row of zeros

// Biased exponent field, 1 for denormals and 0 for zeros only; 2047 for infinities and NaN.
__device__ __forceinline__ int expo(double v) {
    const int h = __double2hiint(v) & 0x7fffffff, e = h >> 20;
    return e ? e : (h | __double2loint(v)) != 0;
}

// Row exponents.  Digits are cut from finite, normal numbers: a row that holds an infinity or a NaN, one
// whose entries are products of two factors and may overflow, and one whose smaller entries are near the
// denormals is kBad, and its elements are formed on the FP64 pipe as they come.
__device__ __forceinline__ int expo_row(int e) { return e > 1024 || e < -900 ? kBad : e; }
// Exponent field sum of a product's factors: 0 where one is zero, kBad where one is not finite;
// expo_of_pairs: the exponent e with |u v| < 2^e from the largest such sum.
__device__ __forceinline__ int expo_pair(int u, int v) { return (u == 2047 || v == 2047) ? kBad : (u && v) ? u + v : 0; }
__device__ __forceinline__ int expo_of_pairs(int m) { return m == kBad ? kBad : m == 0 ? kNone : expo_row(m - 2044); }

// Whether an element of these row and column exponents is the FP64 pipe's: also where the result itself
// may leave the normal range.
__device__ __forceinline__ bool fp64_only(int eu, int ev) {
    if (eu == kBad || ev == kBad) return true;
    return eu != kNone && ev != kNone && (eu + ev < -900 || eu + ev > 1000);
}

// |v| 2^-e as FP32 from below, at least 2^-60 unless v is zero.
__device__ __forceinline__ float scaled_abs(double v, int e) {
    const int h = __double2hiint(v) & 0x7fffffff, l = __double2loint(v);
    if ((h | l) == 0) return 0.f;
    const int d = min(max((h >> 20) - 1023 - e, -60), 0);
    return __int_as_float(((d + 127) << 23) | ((h & 0xfffff) << 3) | ((uint32_t)l >> 29));
}

// Balanced digits of an integer of at most 62 bits and sign, as floats that are exact in bf16 (low half
// zero): add 128 to every digit, read the bytes, take 128 away.
__device__ __forceinline__ void digits_of(unsigned long long x, uint32_t *f) {
    const unsigned long long u = x + 0x8080808080808080ull;
    const uint32_t h = (uint32_t)(u >> 32), l = (uint32_t)u;
#pragma unroll
    for (int s = 0; s < kDig; ++s) {
        const uint32_t w = __byte_perm(s < 4 ? h : l, 0x4B400000u, 0x7640u | (uint32_t)(3 - (s & 3)));
        f[s] = __float_as_uint(__uint_as_float(w) - 12583040.f);
    }
}

// NV (8 or 16) values of one row, scaled by 2^(62 - e), as digits: dst[s plane + 0 .. NV - 1].
template <int NV>
__device__ __forceinline__ void put_digits(const double *v, int e, __nv_bfloat16 *dst, size_t plane) {
    uint32_t w[kDig][NV / 2];
#pragma unroll
    for (int q = 0; q < NV / 2; ++q) {
        uint32_t f[2][kDig];
#pragma unroll
        for (int z = 0; z < 2; ++z) {
            const double x = v[2 * q + z];
            const int ex = expo(x), sh = 10 + (ex - 1023) - e;
            unsigned long long m = ((unsigned long long)__double_as_longlong(x) & 0xfffffffffffffull) | 0x10000000000000ull;
            if (sh >= 0) m <<= sh;
            else if (sh > -60) m = (m + (1ull << (-sh - 1))) >> -sh;
            else m = 0;
            if (ex == 0) m = 0;
            digits_of(__double2hiint(x) < 0 ? 0ull - m : m, f[z]);
        }
#pragma unroll
        for (int s = 0; s < kDig; ++s) w[s][q] = __byte_perm(f[0][s], f[1][s], 0x7632);
    }
#pragma unroll
    for (int s = 0; s < kDig; ++s) {
        uint4 *o = reinterpret_cast<uint4 *>(dst + s * plane);
#pragma unroll
        for (int z = 0; z < NV / 8; ++z) o[z] = make_uint4(w[s][4 * z], w[s][4 * z + 1], w[s][4 * z + 2], w[s][4 * z + 3]);
    }
}

__device__ __forceinline__ void mma_n(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t *v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr));
}

// Level sums (exact integers) joined: hi of levels 0 .. 3, lo of 4 .. 7.
__device__ __forceinline__ long long join_levels(const int *D) {
    return (((long long)D[0] * 256 + D[1]) * 256 + D[2]) * 256 + D[3];
}

// (hi 2^32 + lo) 2^ex rounded once to FP64, in integer instructions.
__device__ __forceinline__ double combine(long long hi, long long lo, int ex) {
    long long h = hi + (lo >> 32);
    uint32_t l = (uint32_t)lo;
    const bool neg = h < 0;
    if (neg) {
        h = -h - (l != 0);
        l = 0u - l;
    }
    if (h == 0 && l == 0) return 0.0;
    const int lz = __clzll(h), E = 95 - lz + ex;
    if (lz > 35 || E < -1022 || E > 1022) {  // small sums (29 bits of h at least otherwise) and the ends of the range
        const double v = scalbn(fma((double)h, 4294967296.0, (double)l), ex);
        return neg ? -v : v;
    }
    const unsigned long long w = ((unsigned long long)h << lz) |
                                 (lz >= 32 ? (unsigned long long)l << (lz - 32) : (unsigned long long)l >> (32 - lz));
    // top bit of w at 63: 53 bits and the rounding bit
    unsigned long long b = (w >> 11) + ((w >> 10) & 1ull) + ((unsigned long long)(E + 1022) << 52);
    if (neg) b |= 0x8000000000000000ull;
    return __longlong_as_double((long long)b);
}

}  // namespace p64
}  // namespace bsa
