// The unit in which outputs of digit products (digits.cuh) are kept in 64 bits, from the
// magnitudes of the terms.  Plain C++ on the host, so that the CPU tests compile it.
#pragma once

#ifdef __CUDACC__
#define CGD_HD __host__ __device__ __forceinline__
#else
#define CGD_HD inline
#endif

namespace cgd {

// A magnitude 2^t as a share of the largest, 2^tmax, in 2^-16: integers, so that sums
// of shares do not depend on their order.
CGD_HD unsigned share16(int t, int tmax) {
    const int s = tmax - t;
    return (65536u >> (s < 16 ? s : 16)) + 1u;
}

// The finest unit with room in 63 bits for outputs of at most sum / 2^16 times the
// largest product (0.2481), sum of the shares over the terms times `terms`.  An owner can
// have any number of clusters of a type (a share is up to 65,537, and 65,535 of them pass
// 32 bits), so sums are 64-bit: up to 2^47, of 2^31 terms, times less than 2^16.
CGD_HD int up_bits(unsigned long long sum, int terms) {
    const unsigned long long b = sum * (unsigned)terms;
#ifdef __CUDA_ARCH__
    const int lz = __clzll((long long)b);
#else
    const int lz = b ? __builtin_clzll(b) : 64;
#endif
    const int up = 9 - (64 - lz - 16);   // 2^(9 - up + 16) > sum terms
    return up < -40 ? -40 : (up > 8 ? 8 : up);
}

}  // namespace cgd
