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

// Sum 8 per-thread values over the block and add them to the frame's scalars:
// v = [E, P, Wxx, Wxy, Wxz, Wyy, Wyz, Wzz].
__device__ __forceinline__ void block_scalars_add(double* v, double* So, int f) {
    __shared__ double red[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        double s = warp_sum(v[k]);
        if (lane == 0) red[k][w] = s;
    }
    __syncthreads();
    if (threadIdx.x < 8) {
        double s = 0.0;
        for (int i = 0; i < nw; ++i) s += red[threadIdx.x][i];
        // tensor slots: xx=2 xy=3 xz=4 yx=5 yy=6 yz=7 zx=8 zy=9 zz=10 (symmetric)
        const int k = threadIdx.x;
        double* o = So + (size_t)f * MD_NSCALAR;
        if (s != 0.0) {
            if (k == 0) atomicAdd(o + 0, s);
            else if (k == 1) atomicAdd(o + 1, s);
            else if (k == 2) atomicAdd(o + 2, s);
            else if (k == 3) { atomicAdd(o + 3, s); atomicAdd(o + 5, s); }
            else if (k == 4) { atomicAdd(o + 4, s); atomicAdd(o + 8, s); }
            else if (k == 5) atomicAdd(o + 6, s);
            else if (k == 6) { atomicAdd(o + 7, s); atomicAdd(o + 9, s); }
            else atomicAdd(o + 10, s);
        }
    }
}

// Tile -> (key, first grouped cluster); false when the tile is past the last one.
__device__ __forceinline__ bool tile_lookup(const MdBuckets& B, int tile, int& key, int64_t& c0, int64_t& c1) {
    if (tile >= B.tile_ofs[B.nkeys]) return false;
    int lo = 0, hi = B.nkeys - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (B.tile_ofs[mid] <= tile) lo = mid; else hi = mid - 1;
    }
    key = lo;
    c0 = B.start[key] + (int64_t)(tile - B.tile_ofs[key]) * MDC_TILE;
    c1 = B.start[key + 1];
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
