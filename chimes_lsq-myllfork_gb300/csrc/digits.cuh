// Products of table entries on the tensor cores without loss: entries are scaled by
// powers of two to fixed point and split into signed base-256 digits that FP16 holds
// exactly; digit products are summed exactly in FP32 accumulators, one per diagonal
// a + b of the digit pairs, and the diagonals are packed into one 64-bit integer (the
// scheme of Ozaki, Ogita, Oishi, Rump, Numer. Algorithms 59, 2012).
//
// |X| < 2^63, 8 digits, X = sum_a d_a 256^(7-a) with -128 <= d_a <= 127; the 36 pairs with
// a + b < 8 are formed, the others are below 7 * 2^14 * 256^-10 = 2^-63.2 of the scaled
// product (a few times 2^-61 of the largest one).
#pragma once
#include <cstdint>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "units.h"

namespace cgd {

constexpr int DIG_ND = 8;          // digits, and diagonals
constexpr int DIG_FIX = 63;        // log2 of the bound on |X|
// Bytes of one table row in shared memory: 8 digits of 8 clusters, 16 bytes each, and 16
// more so that the 8 rows an ldmatrix reads fall into different banks.
constexpr int DIG_STRIDE = 144;

// ---------------------------------------------------------------- magnitudes
// Sixteenths of log2 |x|, rounded up (zero: about -1023 * 16); LG_BAD for infinities and NaN.
constexpr int LG_BAD = 32767;
__device__ __forceinline__ int lg_up(double x) {
    const int b = __double2hiint(x) & 0x7fffffff;
    // the mantissa's leading bits as a fraction are at most 0.0861 below log2(1 + m): +2/16
    return b >= 0x7ff00000 ? LG_BAD : (b >> 16) - 1023 * 16 + 3;
}
// The least exponent e with 2^e at least 1.04 times a product whose lg_up sum is lg.
__device__ __forceinline__ int pow2_above(int lg) { return max((lg + 1) >> 4, -960) + 1; }

// ---------------------------------------------------------------- fixed point
// x 2^sh rounded to an integer (|result| < 2^63 by the choice of sh).
__device__ __forceinline__ long long to_fixed(double x, int sh) {
    const long long b = __double_as_longlong(x);
    const int ex = (int)((b >> 52) & 0x7ff);
    const unsigned long long m = (((unsigned long long)b << 11) | 0x8000000000000000ull);   // 53 bits, leading bit 63
    const int rs = max(1085 - ex - sh, 0);      // x 2^sh = (m / 2^11) 2^(ex + sh - 1075) = m / 2^(rs + 1)
    const unsigned long long v = rs > 63 || ex == 0 ? 0ull : ((m >> rs) + 1) >> 1;
    return b < 0 ? -(long long)v : (long long)v;
}
// The digits of two clusters' entries into p, p + 16, p + 32, ... bytes (FP16 pairs).
// Adding 128 to every digit makes them the bytes of X + 0x80..80; 0x6400 | byte is the
// FP16 number 1024 + byte, and subtracting 1152 leaves the digit.
__device__ __forceinline__ void put_digit_pair(unsigned char* p, unsigned w0, unsigned w1, int byte) {
    unsigned q = __byte_perm(w0, w1, (unsigned)byte | (unsigned)byte << 4 | (unsigned)(4 + byte) << 8 | (unsigned)byte << 12);
    q = (q & 0x00ff00ffu) | 0x64006400u;
    __half2 h = *reinterpret_cast<__half2*>(&q);
    h = __hsub2(h, __half2half2(__ushort_as_half(0x6480)));   // 1152
    *reinterpret_cast<__half2*>(p) = h;
}
__device__ __forceinline__ void put_digits(unsigned char* p, long long X0, long long X1) {
    constexpr unsigned long long bias = 0x8080808080808080ull;
    const unsigned long long u0 = (unsigned long long)X0 + bias, u1 = (unsigned long long)X1 + bias;
#pragma unroll
    for (int a = 0; a < DIG_ND; ++a) {
        const int byte = DIG_ND - 1 - a;
        put_digit_pair(p + 16 * a, byte < 4 ? (unsigned)u0 : (unsigned)(u0 >> 32),
                       byte < 4 ? (unsigned)u1 : (unsigned)(u1 >> 32), byte & 3);
    }
}

// ---------------------------------------------------------------- fragments and products
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

// A fragments of 16 table rows: a[digit][0] rows 0..7, [1] rows 8..15 (8 clusters).
// rows: shared address of the first row.
__device__ __forceinline__ void load_a(uint32_t (&a)[DIG_ND][2], uint32_t rows) {
    const int lane = threadIdx.x & 31;
    const uint32_t base = rows + (lane & 15) * DIG_STRIDE + (lane >> 4) * 16;
#pragma unroll
    for (int d = 0; d < DIG_ND; d += 2) {
        uint32_t r[4];
        ldsm4(r, base + d * 16);
        a[d][0] = r[0]; a[d][1] = r[1];
        a[d + 1][0] = r[2]; a[d + 1][1] = r[3];
    }
}
// B fragments of 8 table rows (8 columns of the product).
__device__ __forceinline__ void load_b(uint32_t (&b)[DIG_ND], uint32_t rows) {
    const int lane = threadIdx.x & 31;
    const uint32_t base = rows + (lane & 7) * DIG_STRIDE + (lane >> 3) * 16;
#pragma unroll
    for (int d = 0; d < DIG_ND; d += 4) {
        uint32_t r[4];
        ldsm4(r, base + d * 16);
#pragma unroll
        for (int k = 0; k < 4; ++k) b[d + k] = r[k];
    }
}

// acc[D] += sum over the 8 clusters and the digit pairs a + b = D of A_a B_b.  One
// mma.sync (16 rows, 8 columns, K = 16) takes two digit pairs of the 8 clusters.
__device__ __forceinline__ void mma_digits(float (&acc)[DIG_ND][4], const uint32_t (&a)[DIG_ND][2],
                                           const uint32_t (&b)[DIG_ND]) {
#pragma unroll
    for (int D = 0; D < DIG_ND; ++D) {
#pragma unroll
        for (int k = 0; k <= D; k += 2) {
            const int k2 = k + 1 <= D ? k + 1 : k;
            const uint32_t b1 = k + 1 <= D ? b[D - k2] : 0u;
            asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                         "{%0,%1,%2,%3};"
                         : "+f"(acc[D][0]), "+f"(acc[D][1]), "+f"(acc[D][2]), "+f"(acc[D][3])
                         : "r"(a[k][0]), "r"(a[k][1]), "r"(a[k2][0]), "r"(a[k2][1]), "r"(b[D - k]), "r"(b1));
        }
    }
}

// c += A B, one mma.sync (16 rows, 8 columns, K = 16) in FP16 with FP32 sums.
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Accumulators start at MAGIC and hold MAGIC + S exactly while |S| <= 2^22 (32 terms of
// 8 digit pairs); their bits minus MAGIC_BITS are S.
constexpr float MAGIC = 12582912.0f;            // 1.5 * 2^23
constexpr unsigned MAGIC_BITS = 0x4b400000u;
constexpr int MAGIC_TERMS = 32;

__device__ __forceinline__ void acc_clear(float (&acc)[DIG_ND][4]) {
#pragma unroll
    for (int D = 0; D < DIG_ND; ++D)
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[D][r] = MAGIC;
}

// sum_D S_D 2^(40 - 8 D) of one output: the part before the binary point, and fr / 2^16 behind it.
__device__ __forceinline__ long long acc_parts(const float (&acc)[8][4], int k, int& fr) {
    constexpr unsigned c = MAGIC_BITS * 257u;
    const unsigned hi = __float_as_uint(acc[0][k]) * 256u + __float_as_uint(acc[1][k]) - c;
    const int mid = (int)(__float_as_uint(acc[2][k]) * 256u + __float_as_uint(acc[3][k]) - c);
    const int lo = (int)(__float_as_uint(acc[4][k]) * 256u + __float_as_uint(acc[5][k]) - c);
    fr = (int)(__float_as_uint(acc[6][k]) * 256u + __float_as_uint(acc[7][k]) - c);
    return (long long)((unsigned long long)hi << 32) + ((long long)mid << 16) + (long long)lo;
}

// One output: sum_D S_D 2^(40 + up - 8 D), the digits below the unit rounded, in units of
// 2^-(56 + up) of the product of the scaled entries (X / 2^64 each); up from up_bits() (units.h).
__device__ __forceinline__ long long acc_value(const float (&acc)[8][4], int k, int up) {
    int fr;
    const long long v = acc_parts(acc, k, fr);
    if (up >= 0) return (long long)((unsigned long long)v << up) + (((fr >> (15 - up)) + 1) >> 1);
    return (v + (fr >> 16) + (1ll << (-up - 1))) >> -up;   // to nearest: sums of floors would drift
}
// v 2^e correctly rounded to FP64 in integer arithmetic (the conversion and the
// multiplication would take the FP64 pipe, which has 1/64 of the integer rate).
__device__ __forceinline__ double from_fixed(long long v, int e) {
    const unsigned long long s = (unsigned long long)v & 0x8000000000000000ull;
    unsigned long long a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
    const int lz = __clzll((long long)a);
    const int ex = 1023 + 63 - lz + e;
    if (ex < 2 || ex > 2045 || a == 0) return a ? ldexp((double)v, e) : 0.0;
    a <<= lz;
    const unsigned long long m = (a >> 11) + ((a >> 10) & 1ull);   // 2^52 <= m <= 2^53
    return __longlong_as_double((long long)(s | (((unsigned long long)(ex - 1) << 52) + m)));
}

// v 2^e rounded to FP64.
__device__ __forceinline__ double int128_double(__int128 v, int e) {
    unsigned __int128 a = v < 0 ? -(unsigned __int128)v : (unsigned __int128)v;
    const unsigned long long hi = (unsigned long long)(a >> 64);
    if (hi != 0 || (long long)a < 0) {   // to 62 bits and a sticky one
        const int s = hi != 0 ? 66 - __clzll((long long)hi) : 2;
        const bool lost = (a & (((unsigned __int128)1 << s) - 1)) != 0;
        a = (a >> s) | (lost ? 1 : 0);
        e += s;
    }
    const long long m = (long long)a;
    return from_fixed(v < 0 ? -m : m, e);
}

}  // namespace cgd
