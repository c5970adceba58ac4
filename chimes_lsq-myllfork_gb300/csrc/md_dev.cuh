// Device helpers shared by the MD force kernels (md.cu, md_tensor.cu).
#pragma once
#include "basis.cuh"
#include "md.h"

namespace cgd {

__device__ __forceinline__ int frame_of_atom(const FramesDev& F, int64_t a) {
    int lo = 0, hi = F.nframes - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (F.atom_ofs[mid] <= a) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Sums of N per-lane values over the warp: each step sends half of them away, so N values
// cost about 2 N additions in all, not 5 N (a warp's FP64 addition takes 64 cycles of its SM
// quarter).  Lane l returns the sum of value l / 2 (N > 8) or l / 4 (N <= 8).
template <int N>
__device__ __forceinline__ double warp_sums(const double (&x)[N]) {
    constexpr int P = N > 8 ? 16 : 8;
    static_assert(N <= 16, "values per warp");
    const int lane = threadIdx.x & 31;
    double v[P];
#pragma unroll
    for (int k = 0; k < P; ++k) v[k] = k < N ? x[k < N ? k : 0] : 0.0;
    int o = 16;
#pragma unroll
    for (int h = P / 2; h > 0; h >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const double send = up ? v[k] : v[k + h], keep = up ? v[k + h] : v[k];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return v[0];
}

// Value k of [E, P, Wxx, Wxy, Wxz, Wyy, Wyz, Wzz] into a frame's scalars; tensor slots:
// xx=2 xy=3 xz=4 yx=5 yy=6 yz=7 zx=8 zy=9 zz=10 (symmetric).
__device__ __forceinline__ void scalar_add(double* o, int k, double s) {
    if (k <= 2) atomicAdd(o + k, s);
    else if (k == 3) { atomicAdd(o + 3, s); atomicAdd(o + 5, s); }
    else if (k == 4) { atomicAdd(o + 4, s); atomicAdd(o + 8, s); }
    else if (k == 5) atomicAdd(o + 6, s);
    else if (k == 6) { atomicAdd(o + 7, s); atomicAdd(o + 9, s); }
    else atomicAdd(o + 10, s);
}

// Sum 8 per-thread values over the block and add them to the frame's scalars:
// v = [E, P, Wxx, Wxy, Wxz, Wyy, Wyz, Wzz].
__device__ __forceinline__ void block_scalars_add(const double (&v)[8], double* So, int f) {
    __shared__ double red[8][MDC_TILE / 32];   // of CTAs of MDC_TILE threads
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    const double sum = warp_sums(v);
    if ((lane & 3) == 0) red[lane >> 2][w] = sum;
    __syncthreads();
    if (threadIdx.x < 8) {
        double s = 0.0;
        for (int i = 0; i < nw; ++i) s += red[threadIdx.x][i];
        if (s != 0.0) scalar_add(So + (size_t)f * MD_NSCALAR, threadIdx.x, s);
    }
}

// A warp's sums over one atom's pairs: the force on the atom and the frame's 8 scalars.
__device__ __forceinline__ void pair_sums_add(const double (&x)[11], double* fo, double* so, bool any) {
    const double s = warp_sums(x);
    const int k = (threadIdx.x & 31) >> 1;
    if (!any || (threadIdx.x & 1) || k >= 11) return;
    if (k < 3) atomicAdd(fo + k, s);
    else scalar_add(so, k - 3, s);
}

// Tile -> (key, first grouped cluster); false when the tile is past the last one.
__device__ __forceinline__ bool tile_lookup(const MdBuckets& B, int tile, int& key, int64_t& c0, int64_t& c1) {
    if (tile >= B.tile_ofs[B.nkeys]) return false;
    int lo = 0, hi = B.nkeys - 1;
    if (B.tile_key) lo = hi = B.tile_key[tile];
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (B.tile_ofs[mid] <= tile) lo = mid; else hi = mid - 1;
    }
    key = lo;
    c0 = B.start[key] + (int64_t)(tile - B.tile_ofs[key]) * MDC_TILE;
    c1 = B.start[key] + B.cursor[key];
    return c0 < c1;
}

__device__ __forceinline__ void edge_ab(int NBODY, int e, int& a, int& b) {
    if (NBODY == 3) { a = e == 2 ? 1 : 0; b = e == 0 ? 1 : 2; }
    else {
        a = e < 3 ? 0 : (e < 5 ? 1 : 2);
        b = e == 0 ? 1 : (e == 1 || e == 3) ? 2 : 3;
    }
}

}  // namespace cgd
