// Normal equations of the fit: G = A^T A and h = A^T b, streamed over row blocks.
//
// The reference solves the least-squares problem with a truncated SVD of the full
// A in numpy (src/chimes_lsq.py:169-214); this library forms the Gram instead, the
// path's only dense contraction and its only tensor-core work:
//  * mixed form: A is split into two BF16 planes (hi = bf16(a), lo = bf16(a - hi)),
//    stored transposed (K = rows contiguous), and G += hi^T hi + hi^T lo + lo^T hi on
//    tcgen05 (kind::f16, FP32 accumulation in TMEM).  A persistent CTA per SM walks
//    the 128 x 256 (or, for small Grams, 128 x 128) tiles that reach the upper
//    triangle: operands arrive by TMA with 128-byte swizzle through a 192 KB mbarrier
//    ring, one thread issues the MMAs into one of two TMEM accumulators, and four
//    epilogue warps drain the other with tcgen05.ld and add it into an FP64 G.
//  * plain form: FP64 G by this library's register-blocked FP64 SYRK (dense64.cu),
//    which runs at the FP64 FMA rate of the GPU.
//  * h = A^T b is an FP64 matrix-vector product (plain form) or is fused into the
//    BF16 split pass (mixed form).
// Every wait on an mbarrier is bounded (about two seconds); on time-out the kernel
// records an error code, skips its stores, frees its TMEM and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <mutex>
#include <stdexcept>
#include <string>
#include <utility>

#include "dense64.h"
#include "digits.cuh"
#include "gram.h"
#include "scratch.h"

namespace cgd {

constexpr int GB_M = 128, GB_K = 64, GB_THREADS = 192;
constexpr uint32_t GB_TILE_A = GB_M * GB_K * 2;             // one 128x64 bf16 row-tile operand (16 KB)
constexpr long long GB_WAIT_CYCLES = 4000000000LL;          // ~2 s at 2 GHz
constexpr int GB_EPI_LD = 33;                               // epilogue staging row (floats)

// ---------------------------------------------------------------- split + transpose
// planes[p][c][k] (bf16, k contiguous) for rows [r0, r0+nr) of A (row-major, lda),
// zero padded to (cpad, kpad), fused with h = A^T b so that A is read once.  A block owns a strip of
// 32 columns and the 128-row K tiles kt = blockIdx.x, blockIdx.x + gridDim.x, ...;
// each thread keeps one column's running sum over the rows it loads.  FP64 input
// sums in FP64.  FP32 input sums in float-float: each product a*b (b split into
// two floats) is formed exactly by an FMA, added by an error-free two-sum, and the
// pair renormalised after every tile, so the sum carries about 44 significant bits
// while the FP64 pipe (a small fraction of the FP32 rate on this GPU) stays idle.
// partial[blockIdx.x][c] = the block's sum, combined in order by k_split_reduce.
constexpr int SPA_K = 128, SPA_C = 32, SPA_THREADS = 256;
struct FloatFloat {
    float hi = 0.f, lo = 0.f;
    __device__ __forceinline__ void add_prod(float a, float bh, float bl) {
        const float p = __fmul_rn(a, bh);
        float e = __fmaf_rn(a, bh, -p);      // a*bh - p exactly
        e = __fmaf_rn(a, bl, e);
        const float s = __fadd_rn(hi, p);    // two-sum(hi, p)
        const float bb = __fsub_rn(s, hi);
        const float t = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), __fsub_rn(p, bb));
        hi = s;
        lo = __fadd_rn(lo, __fadd_rn(t, e));
    }
    __device__ __forceinline__ void renorm() {   // two-sum(hi, lo)
        const float s = __fadd_rn(hi, lo);
        const float bb = __fsub_rn(s, hi);
        lo = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), __fsub_rn(lo, bb));
        hi = s;
    }
    __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};

// b of the rows [r0, r0+nr) as two floats (bh + bl carries 48 bits), zero up to kpad
__global__ void k_split_b(const double* __restrict__ b, int64_t r0, int64_t nr, int64_t kpad, float2* __restrict__ bs) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= kpad) return;
    const double v = k < nr ? b[r0 + k] : 0.0;
    const float bh = __double2float_rn(v);
    bs[k] = make_float2(bh, __double2float_rn(v - (double)bh));
}

// FP64 input reads b (rows r0..); FP32 input reads bsplit (k_split_b of the block).
template <typename T>
__global__ void __launch_bounds__(SPA_THREADS, 4) k_split_atb(const T* __restrict__ A, int64_t lda, int64_t r0,
                                                          int64_t nr, int ncols, const double* __restrict__ b,
                                                          const float2* __restrict__ bsplit,
                                                          __nv_bfloat16* __restrict__ hi, __nv_bfloat16* __restrict__ lo,
                                                          int64_t kpad, double* __restrict__ partial) {
    __shared__ float tile[SPA_K][SPA_C + 1];
    __shared__ double bd[SPA_K];
    __shared__ float2 bs[SPA_K];
    __shared__ double red[SPA_THREADS / 32][SPA_C];
    const int tx = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int c0 = blockIdx.y * SPA_C;
    const int c = c0 + tx;
    const int64_t ntk = (kpad + SPA_K - 1) / SPA_K;   // kpad is a multiple of 64
    double accd = 0.0;
    FloatFloat accf;
    for (int64_t kt = blockIdx.x; kt < ntk; kt += gridDim.x) {
        const int64_t k0 = kt * SPA_K;
        T v[SPA_K / 8];
        const T* p = A + (r0 + k0 + w) * lda + c;
        if (k0 + SPA_K <= nr && c < ncols) {   // interior tile: no per-row checks
#pragma unroll
            for (int i = 0; i < SPA_K / 8; ++i) v[i] = p[(int64_t)i * 8 * lda];
        } else {
#pragma unroll
            for (int i = 0; i < SPA_K / 8; ++i)
                v[i] = (k0 + w + 8 * i < nr && c < ncols) ? p[(int64_t)i * 8 * lda] : T(0);
        }
        if (threadIdx.x < SPA_K) {
            const int64_t k = k0 + threadIdx.x;
            if constexpr (sizeof(T) == 8) bd[threadIdx.x] = k < nr ? b[r0 + k] : 0.0;
            else bs[threadIdx.x] = k < kpad ? bsplit[k] : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < SPA_K / 8; ++i) tile[w + 8 * i][tx] = (float)v[i];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < SPA_K / 8; ++i) {
            if constexpr (sizeof(T) == 8) {
                accd = fma((double)v[i], bd[w + 8 * i], accd);
            } else {
                const float2 bb = bs[w + 8 * i];
                accf.add_prod((float)v[i], bb.x, bb.y);
            }
        }
        if constexpr (sizeof(T) != 8) accf.renorm();
        // planes: column c0+cl gets SPA_K contiguous K values (up to kpad); a warp
        // stores 32 bf16 pairs = 128 bytes per instruction
#pragma unroll
        for (int j = 0; j < SPA_C / 8; ++j) {
            const int cl = w + 8 * j;
#pragma unroll
            for (int hk = 0; hk < SPA_K; hk += 64) {
                if (k0 + hk >= kpad) break;
                const float f0 = tile[hk + 2 * tx][cl], f1 = tile[hk + 2 * tx + 1][cl];
                const __nv_bfloat162 hp = __floats2bfloat162_rn(f0, f1);
                const float2 hf = __bfloat1622float2(hp);
                const __nv_bfloat162 lp = __floats2bfloat162_rn(f0 - hf.x, f1 - hf.y);
                const int64_t o = (int64_t)(c0 + cl) * kpad + k0 + hk + 2 * tx;
                *reinterpret_cast<__nv_bfloat162*>(hi + o) = hp;
                *reinterpret_cast<__nv_bfloat162*>(lo + o) = lp;
            }
        }
        __syncthreads();
    }
    if constexpr (sizeof(T) == 8) red[w][tx] = accd;
    else red[w][tx] = accf.value();
    __syncthreads();
    if (w == 0 && c < ncols) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < SPA_THREADS / 32; ++q) s += red[q][tx];
        partial[(int64_t)blockIdx.x * ncols + c] = s;
    }
}

// h[c] += sum over y of partial[y][c] (the split pass's per-block column sums), in
// a fixed order so that h is reproducible.
__global__ void k_split_reduce(const double* __restrict__ partial, int nslices, int ncols, double* __restrict__ h) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncols) return;
    double s = 0.0;
    for (int y = 0; y < nslices; ++y) s += partial[(int64_t)y * ncols + c];
    h[c] += s;
}

// The strict lower triangle from the upper one, a 64 x 64 tile of the upper triangle per
// CTA, transposed through shared memory with 16 reads in flight per thread.  Reads and
// writes of n^2 / 2 entries each bound it; one thread per entry read column-wise: n = 6,007
// 108 -> 55 us (42 us at the copy rate).
constexpr int SY_B = 64, SY_THREADS = 256;
__global__ void __launch_bounds__(SY_THREADS) k_symmetrize(double* __restrict__ G, int n) {
    __shared__ double t[SY_B][SY_B + 1];
    const int bi = blockIdx.y, bj = blockIdx.x;
    if (bj < bi) return;
    const int c = threadIdx.x % SY_B, r = threadIdx.x / SY_B;
    constexpr int N = SY_B * SY_B / SY_THREADS, RS = SY_THREADS / SY_B;
    const int i0 = bi * SY_B, j0 = bj * SY_B;
    double v[N];
#pragma unroll
    for (int u = 0; u < N; ++u)
        v[u] = i0 + r + RS * u < n && j0 + c < n ? G[(int64_t)(i0 + r + RS * u) * n + j0 + c] : 0.0;
#pragma unroll
    for (int u = 0; u < N; ++u) t[r + RS * u][c] = v[u];
    __syncthreads();
#pragma unroll
    for (int u = 0; u < N; ++u) {
        const int j = j0 + r + RS * u, i = i0 + c;
        if (j < n && i < j) G[(int64_t)j * n + i] = t[c][r + RS * u];
    }
}

// ---------------------------------------------------------------- PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: false (and an error code in *err) when the phase does not complete in time.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* err, int code) {
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - t0 > GB_WAIT_CYCLES) {
            atomicCAS(err, 0, code);
            return false;
        }
    }
    return true;
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}
// K-major operand with 128-byte swizzle: 8-row atoms of 1024 B (SBO), version 1.
__device__ __forceinline__ uint64_t smem_desc(const void* p) {
    const uint64_t addr = smem_u32(p);
    return ((addr >> 4) & 0x3FFFull) | ((uint64_t)(16 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
           (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// Tile pair t of the Gram's upper triangle: ti indexes 128-row tiles, tj column
// tiles of Q x 128 columns, and a pair is kept when its tile reaches the upper
// triangle (tj >= ti / Q).  Pairs are walked in super-tiles of GB_GR row tiles x
// GB_GR / Q column tiles (the same 1536 rows and columns), super-tiles of one
// super-row in column order, tiles inside a super-tile column by column: the ~150
// units in flight at one time read about 12 row tiles and 12 / Q column tiles between
// them, which stay in L2.
constexpr int GB_GR = 12;
template <int Q>
__device__ __forceinline__ void grouped_pair(int t, int nti, int ntj, int& ti, int& tj) {
    constexpr int GB_GC = GB_GR / Q;
    const int nsr = (nti + GB_GR - 1) / GB_GR;
    for (int SI = 0; SI < nsr; ++SI) {
        const int r0 = SI * GB_GR, r1 = min(nti, r0 + GB_GR), r = r1 - r0;
        const int c0 = SI * GB_GC, c1 = min(ntj, c0 + GB_GC);
        if (c0 >= ntj) break;
        int diag = 0;
        for (int i = r0; i < r1; ++i) diag += max(0, c1 - max(c0, i / Q));
        if (t < diag) {   // the diagonal super-tile, by rows
            for (int i = r0; i < r1; ++i) {
                const int lo = max(c0, i / Q), cnt = max(0, c1 - lo);
                if (t < cnt) { ti = i; tj = lo + t; return; }
                t -= cnt;
            }
        }
        t -= diag;
        const int off = r * max(0, ntj - c1);
        if (t < off) {    // full super-tiles to the right, column by column
            const int SJ = SI + 1 + t / (r * GB_GC), tt = t % (r * GB_GC);
            ti = r0 + tt % r;
            tj = SJ * GB_GC + tt / r;
            return;
        }
        t -= off;
    }
    ti = tj = 0;   // not reached for t < the pair count
}

// ---------------------------------------------------------------- tcgen05 Gram tiles
// Persistent kernel, one CTA per SM.  A work unit is a (tile pair i <= j, K slice);
// CTA b takes units b, b + gridDim.x, ... in grouped tile-pair order, so the units in
// flight at one time stay close in the triangle.  Warp roles:
//   warp 0      TMA producer: the hi / lo 128x64 row-tile and BNx64 column-tile
//               operands of each K step into a GB_STAGES-deep ring of stages
//               (full / empty mbarriers);
//   warp 1      MMA issuer: 12 tcgen05.mma (M 128, N BN, K 16) per K step into one
//               of two TMEM accumulators (BN columns each), committed to acc_full[buf];
//   warps 2..5  epilogue: tcgen05.ld of the accumulator (TMEM lane quarter =
//               warp % 4), staged 32 columns at a time through shared memory so that
//               every FP64 atomic instruction adds 32 consecutive columns of a row of
//               G, then acc_empty[buf] frees the accumulator.
// With two accumulators the epilogue of one unit runs under the MMAs of the next, and
// the ring keeps loading across unit boundaries.
// BN: columns of a column tile (256 for large Grams; 128 when the triangle has too
// few tiles to fill the GPU without slicing K, where the wider tile's longer K
// slices lose their L2 reuse).  Both forms hold 192 KB of operand stages.
constexpr int GB_ACC = 2;
template <int BN>
struct GbCfg {
    static constexpr int N = BN;
    static constexpr int Q = BN / GB_M;
    static constexpr int STAGES = BN == 256 ? 2 : 3;
    static constexpr uint32_t TILE_B = BN * GB_K * 2;
    static constexpr uint32_t STAGE_BYTES = 2 * GB_TILE_A + 2 * TILE_B;   // A_hi, A_lo, B_hi, B_lo
    static constexpr uint32_t epi = STAGES * STAGE_BYTES;
    static constexpr uint32_t bars = epi + 4 * 32 * GB_EPI_LD * 4;
    static constexpr uint32_t nbars = 2 * STAGES + 2 * GB_ACC + 1;
    static constexpr uint32_t total = bars + nbars * 8 + 16;
    static_assert(bars % 8 == 0, "mbarrier alignment");
    static_assert(total + 1024 <= 227 * 1024, "shared memory per CTA");
};

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

template <int Q>
__device__ __forceinline__ int gb_unit(int u, int npairs, int nti, int ntj, int64_t kpad, int64_t kslice, int& ti,
                                       int& tj, int64_t& kb) {
    const int slice = u / npairs;
    grouped_pair<Q>(u - slice * npairs, nti, ntj, ti, tj);
    kb = (int64_t)slice * kslice;
    const int64_t ke = min(kpad, kb + kslice);
    return ke > kb ? (int)((ke - kb) / GB_K) : 0;
}

template <int BN>
__global__ void __launch_bounds__(GB_THREADS, 1)
    k_gram_tc(const __grid_constant__ CUtensorMap map_hi_a, const __grid_constant__ CUtensorMap map_lo_a,
              const __grid_constant__ CUtensorMap map_hi_b, const __grid_constant__ CUtensorMap map_lo_b, int nti,
              int ntj, int npairs, int nunits, int64_t kpad, int64_t kslice, int ncols, double* __restrict__ G,
              int* __restrict__ err) {
    using Cfg = GbCfg<BN>;
    constexpr int GB_N = Cfg::N, GB_STAGES = Cfg::STAGES;
    constexpr uint32_t GB_TILE_B = Cfg::TILE_B, GB_STAGE_BYTES = Cfg::STAGE_BYTES;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + Cfg::bars);
    uint64_t* empty = full + GB_STAGES;
    uint64_t* acc_full = empty + GB_STAGES;
    uint64_t* acc_empty = acc_full + GB_ACC;
    uint64_t* done = acc_empty + GB_ACC;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < GB_STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < GB_ACC; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 4); }
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {   // TMEM: 128 lanes x (2 x 128) FP32 columns
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(GB_ACC * GB_N)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {   // producer
            bool ok = true;
            int64_t g = 0;   // K steps issued over all units
            for (int u = blockIdx.x; u < nunits && ok; u += gridDim.x) {
                int ti, tj;
                int64_t kb;
                const int nk = gb_unit<Cfg::Q>(u, npairs, nti, ntj, kpad, kslice, ti, tj, kb);
                for (int it = 0; it < nk; ++it, ++g) {
                    const int s = (int)(g % GB_STAGES);
                    const uint32_t ph = (uint32_t)(g / GB_STAGES) & 1u;
                    if (!mbar_wait(&empty[s], ph ^ 1u, err, 1)) { ok = false; break; }
                    unsigned char* st = smem + s * GB_STAGE_BYTES;
                    // a column tile reaching past the padded column count reads zeros
                    // (out-of-range rows of a TMA load are filled and still counted)
                    mbar_expect_tx(&full[s], GB_STAGE_BYTES);
                    const int x = (int)(kb + (int64_t)it * GB_K);
                    tma_load_2d(st, &map_hi_a, &full[s], x, ti * GB_M);
                    tma_load_2d(st + GB_TILE_A, &map_lo_a, &full[s], x, ti * GB_M);
                    tma_load_2d(st + 2 * GB_TILE_A, &map_hi_b, &full[s], x, tj * GB_N);
                    tma_load_2d(st + 2 * GB_TILE_A + GB_TILE_B, &map_lo_b, &full[s], x, tj * GB_N);
                }
            }
            // drain after a time-out: the last load issued into each stage completes
            // the full-barrier phase (g / GB_STAGES) & 1; wait (bounded) for it so that
            // no copy still writes this CTA's shared memory when it exits
            if (!ok)
                for (int64_t q = g - 1; q >= 0 && q >= g - GB_STAGES; --q)
                    mbar_wait(&full[q % GB_STAGES], (uint32_t)(q / GB_STAGES) & 1u, err, 4);
        }
    } else if (warp == 1) {
        if (lane == 0) {   // MMA issuer
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(GB_N >> 3) << 17) |
                                   ((uint32_t)(GB_M >> 4) << 24);
            bool ok = true;
            int64_t g = 0;
            int j = 0;   // units with K steps, in order (accumulator buffer j & 1)
            for (int u = blockIdx.x; u < nunits && ok; u += gridDim.x) {
                int ti, tj;
                int64_t kb;
                const int nk = gb_unit<Cfg::Q>(u, npairs, nti, ntj, kpad, kslice, ti, tj, kb);
                if (nk == 0) continue;
                const int buf = j & 1;
                if (!mbar_wait(&acc_empty[buf], ((uint32_t)(j >> 1) & 1u) ^ 1u, err, 5)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d = tmem + (uint32_t)(buf * GB_N);
                for (int it = 0; it < nk; ++it, ++g) {
                    const int s = (int)(g % GB_STAGES);
                    const uint32_t ph = (uint32_t)(g / GB_STAGES) & 1u;
                    if (!mbar_wait(&full[s], ph, err, 2)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    unsigned char* st = smem + s * GB_STAGE_BYTES;
                    const uint64_t ahi = smem_desc(st), alo = smem_desc(st + GB_TILE_A);
                    const uint64_t bhi = smem_desc(st + 2 * GB_TILE_A), blo = smem_desc(st + 2 * GB_TILE_A + GB_TILE_B);
#pragma unroll
                    for (int kk = 0; kk < GB_K / 16; ++kk) {
                        const uint64_t adv = (uint64_t)((kk * 32) >> 4);   // 16 bf16 = 32 B along K
                        umma_bf16(d, ahi + adv, bhi + adv, idesc, (it > 0 || kk > 0) ? 1u : 0u);
                        umma_bf16(d, ahi + adv, blo + adv, idesc, 1u);
                        umma_bf16(d, alo + adv, bhi + adv, idesc, 1u);
                    }
                    umma_commit(&empty[s]);
                }
                if (!ok) break;
                umma_commit(&acc_full[buf]);
                ++j;
            }
            // every MMA of this CTA has finished before TMEM is released
            umma_commit(done);
            mbar_wait(done, 0, err, 6);
        }
    } else {   // epilogue warps 2..5
        const int q = warp & 3;   // TMEM lane quarter this warp may read
        float* stile = reinterpret_cast<float*>(smem + Cfg::epi) + (size_t)(warp - 2) * 32 * GB_EPI_LD;
        int j = 0;
        for (int u = blockIdx.x; u < nunits; u += gridDim.x) {
            int ti, tj;
            int64_t kb;
            const int nk = gb_unit<Cfg::Q>(u, npairs, nti, ntj, kpad, kslice, ti, tj, kb);
            if (nk == 0) continue;
            const int buf = j & 1;
            const bool got = mbar_wait(&acc_full[buf], (uint32_t)(j >> 1) & 1u, err, 3);
            if (!__all_sync(0xffffffffu, got)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int c0 = 0; c0 < GB_N; c0 += 32) {
                uint32_t v[32];
                const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * GB_N + c0);
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                    "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                      "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                      "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]),
                      "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]),
                      "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                    : "r"(taddr));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int c = 0; c < 32; ++c) stile[lane * GB_EPI_LD + c] = __uint_as_float(v[c]);
                __syncwarp();
                if (*err == 0) {
                    const int col = tj * GB_N + c0 + lane;
#pragma unroll 4
                    for (int r = 0; r < 32; ++r) {
                        const int row = ti * GB_M + q * 32 + r;
                        if (row < ncols && col < ncols && col >= row)
                            atomicAdd(G + (int64_t)row * ncols + col, (double)stile[r * GB_EPI_LD + lane]);
                    }
                }
                __syncwarp();
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
            ++j;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(GB_ACC * GB_N)
                     : "memory");
    }
}

// ---------------------------------------------------------------- FP64 SYRK update by exact BF16 slices
// C (upper triangle) += alpha X^T X for a panel X of K <= 128 rows, the trailing
// update of the blocked Cholesky, computed with FP64 accuracy on the tensor cores
// (the Ozaki scheme: Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59, 2012).  Each
// column i of X is scaled by a power of two s_i (|X / s_i| < 1) and split into OZ_S
// signed digits, x / s_i = sum_a d_a 128^-(a+1) + r with |d_0| <= 128, |d_a| <= 64,
// |r| <= 2^-57, each an integer that BF16 holds exactly.  A digit product summed over
// K = 128 stays below 2^21 and the sum over the pairs (a, b) of one diagonal a + b = D
// below 2^23 (D < 6: at most 2^22), so the FP32 tensor-core accumulator of each diagonal is exact; the pairs
// with a + b >= OZ_S are dropped (below 2^-56 of the leading term), and the
// epilogue packs sum_D S_D 128^-(D+2) into one 53-bit integer (scaled by s_i s_j).
constexpr int OZ_S = 8;            // digits per element (57 bits)
constexpr int OZ_K = 128;          // panel width (K, zero padded)
constexpr int OZ_M = 128, OZ_N = 64;
constexpr int OZ_EPI = 8;          // epilogue warps: two per TMEM lane quarter
constexpr int OZ_THREADS = 64 + 32 * OZ_EPI;   // warp 0 TMA, warp 1 MMA, warps 2..9 epilogue
constexpr int OZ_W = 16;           // columns per epilogue step
constexpr int OZ_NBARS = 9;        // bfull, bempty, afull[2], aempty[2], tfull, tempty, done
struct OzSmem {
    static constexpr uint32_t b = 0;                                          // OZ_S slices x 2 K halves x 8 KB
    static constexpr uint32_t a = b + OZ_S * 2 * (OZ_N * 128);                // 2 slots x 2 K halves x 16 KB
    static constexpr uint32_t stage = a + 2 * 2 * (OZ_M * 128);               // OZ_EPI warps x 32 x OZ_W doubles
    static constexpr uint32_t bars = stage + OZ_EPI * 32 * OZ_W * 8;
    static constexpr uint32_t total = bars + OZ_NBARS * 8 + 16;
};
static_assert(OzSmem::bars % 8 == 0, "mbarrier alignment");
static_assert(OzSmem::total + 1024 <= 227 * 1024, "shared memory per CTA");

// Digit planes P[a][i][k] (bf16, k contiguous, a < OZ_S, i < mpad, k < OZ_K) and
// scale exponents ex[i] (column i scaled by 2^-ex[i]) of the columns of X (K x m,
// row-major, ldx).  Block: 32 columns.  In integers from the numbers' bits: by FP64
// multiplication and rint the 8 digits of 4,096 elements kept the FP64 pipe (2 per clock)
// busy for 50 us.  A column that holds a NaN or an infinity has zero digits: the update
// leaves its row and column as they are.
__global__ void __launch_bounds__(256) k_oz_slice(const double* __restrict__ X, int64_t ldx, int K, int m, int mpad,
                                                  __nv_bfloat16* __restrict__ P, int* __restrict__ ex) {
    __shared__ double tile[OZ_K][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int i0 = blockIdx.x * 32;
    {
        double v[OZ_K / 8];
#pragma unroll
        for (int u = 0; u < OZ_K / 8; ++u)
            v[u] = (w + 8 * u < K && i0 + lane < m) ? X[(int64_t)(w + 8 * u) * ldx + i0 + lane] : 0.0;
#pragma unroll
        for (int u = 0; u < OZ_K / 8; ++u) tile[w + 8 * u][lane] = v[u];
    }
    __syncthreads();
    for (int c = w; c < 32; c += 8) {
        const int i = i0 + c;
        if (i >= mpad) continue;
        int mx = 0;   // the column's largest high word: its exponent
        for (int k = lane; k < OZ_K; k += 32) mx = max(mx, __double2hiint(tile[k][c]) & 0x7fffffff);
        mx = __reduce_max_sync(0xffffffffu, mx);
        const int emax = max(mx >> 20, 1);   // |x| < 2^(emax - 1022)
        const bool zero = mx == 0 || mx >= 0x7ff00000;
        if (lane == 0) ex[i] = zero ? 0 : emax - 1022;
        auto fixed = [&](double x) {         // x 2^(56 - ex) to nearest, |.| <= 2^56, plus 64 in each lower digit
            const long long bits = __double_as_longlong(x);
            const int ef = (int)((bits >> 52) & 0x7ff), s = max(ef, 1) - emax + 3;
            long long v = (bits & 0xfffffffffffffll) | (ef ? 1ll << 52 : 0ll);
            v = s >= 0 ? v << s : (s < -60 ? 0ll : (v + (1ll << (-s - 1))) >> -s);
            return (zero ? 0ll : (bits < 0 ? -v : v)) + 64ll * (((1ll << 49) - 1) / 127);
        };
        for (int h = 0; h < OZ_K; h += 64) {
            const int k = h + 2 * lane;
            const long long y0 = fixed(tile[k][c]), y1 = fixed(tile[k + 1][c]);
            __nv_bfloat162* out = reinterpret_cast<__nv_bfloat162*>(P + (int64_t)i * OZ_K + k);
            out[0] = __floats2bfloat162_rn((float)(int)(y0 >> 49), (float)(int)(y1 >> 49));
#pragma unroll
            for (int a = 1; a < OZ_S; ++a) {   // 0x4300 | b is the BF16 number 128 + b, b < 128
                const unsigned b0 = (unsigned)(y0 >> (7 * (OZ_S - 1 - a))) & 127u;
                const unsigned b1 = (unsigned)(y1 >> (7 * (OZ_S - 1 - a))) & 127u;
                const unsigned pk = 0x43004300u | b0 | (b1 << 16);
                out[(int64_t)a * mpad * (OZ_K / 2)] =
                    __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&pk), __floats2bfloat162_rn(192.0f, 192.0f));
            }
        }
    }
}

// Tile u of the upper triangle in 128-row x 64-column tiles (ti, tj), kept when
// tj >= 2 ti: row ti holds ntj - 2 ti tiles and f(ti) = ti (ntj + 1 - ti) precede it.
__device__ __forceinline__ void oz_tile(int u, int ntj, int& ti, int& tj) {
    const double b = ntj + 1.0;
    int t = (int)floor((b - sqrt(fmax(0.0, b * b - 4.0 * (double)u))) * 0.5);
    while (t > 0 && (int64_t)t * (ntj + 1 - t) > u) --t;
    while ((int64_t)(t + 1) * (ntj - t) <= u) ++t;
    ti = t;
    tj = 2 * t + (u - t * (ntj + 1 - t));
}

// Persistent: one CTA per SM walks the tiles u = b, b + grid, ...  Warp 0 (TMA) loads a
// tile's OZ_S column-slice operands into one buffer once the previous tile's MMAs have
// read it, and its row-slice operands through two slots; warp 1 issues the digit-pair
// MMAs (M 128, N 64, K 16) into OZ_S TMEM accumulators (diagonal D at columns D x 64:
// all of TMEM) once the epilogue has drained the previous tile; warps 2..9 (TMEM lane
// quarter = warp % 4, half of the columns each) combine the diagonals, add the tile into C and prefetch the next
// tile's rows of C into L2.  The next tile's operands arrive while this tile's
// epilogue runs.
__global__ void __launch_bounds__(OZ_THREADS, 1)
    k_oz_syrk(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
              const int* __restrict__ ex, int m, int mpad, int ntj, int ntiles, double alpha, double* __restrict__ C,
              int64_t ldc, int* __restrict__ err) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bfull = reinterpret_cast<uint64_t*>(smem + OzSmem::bars);
    uint64_t* bempty = bfull + 1;
    uint64_t* afull = bfull + 2;     // [2]
    uint64_t* aempty = bfull + 4;    // [2]
    uint64_t* tfull = bfull + 6;
    uint64_t* tempty = bfull + 7;
    uint64_t* done = bfull + 8;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bfull + OZ_NBARS);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        mbar_init(bfull, 1);
        mbar_init(bempty, 1);
        for (int s = 0; s < 2; ++s) { mbar_init(&afull[s], 1); mbar_init(&aempty[s], 1); }
        mbar_init(tfull, 1);
        mbar_init(tempty, OZ_EPI);
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(OZ_S * OZ_N)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {   // producer
            bool ok = true;
            int64_t g = 0;   // row slices issued over all tiles
            int nb = 0;      // column-slice sets issued
            int64_t last[2] = {-1, -1};
            for (int u = blockIdx.x; u < ntiles && ok; u += gridDim.x) {
                int ti, tj;
                oz_tile(u, ntj, ti, tj);
                if (nb > 0 && !mbar_wait(bempty, (uint32_t)(nb - 1) & 1u, err, 21)) { ok = false; break; }
                mbar_expect_tx(bfull, OZ_S * 2 * OZ_N * 128);
                for (int b = 0; b < OZ_S; ++b)
                    for (int h = 0; h < 2; ++h)
                        tma_load_2d(smem + OzSmem::b + (b * 2 + h) * (OZ_N * 128), &map_b, bfull, h * 64,
                                    b * mpad + tj * OZ_N);
                ++nb;
                for (int a = 0; a < OZ_S; ++a, ++g) {
                    const int s = (int)(g & 1);
                    if (g >= 2 && !mbar_wait(&aempty[s], (uint32_t)((g >> 1) - 1) & 1u, err, 22)) { ok = false; break; }
                    mbar_expect_tx(&afull[s], 2 * OZ_M * 128);
                    for (int h = 0; h < 2; ++h)
                        tma_load_2d(smem + OzSmem::a + (s * 2 + h) * (OZ_M * 128), &map_a, &afull[s], h * 64,
                                    a * mpad + ti * OZ_M);
                    last[s] = g;
                }
            }
            // every issued copy lands before the CTA can exit, on every path (the last
            // copy into a buffer completes that buffer's latest full-barrier phase)
            if (nb > 0) mbar_wait(bfull, (uint32_t)(nb - 1) & 1u, err, 24);
            for (int s = 0; s < 2; ++s)
                if (last[s] >= 0) mbar_wait(&afull[s], (uint32_t)(last[s] >> 1) & 1u, err, 24);
        }
    } else if (warp == 1) {
        if (lane == 0) {   // MMA issuer
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(OZ_N >> 3) << 17) |
                                   ((uint32_t)(OZ_M >> 4) << 24);
            bool ok = true;
            int64_t g = 0;
            int j = 0;
            for (int u = blockIdx.x; u < ntiles && ok; u += gridDim.x, ++j) {
                if (j > 0 && !mbar_wait(tempty, (uint32_t)(j - 1) & 1u, err, 25)) { ok = false; break; }
                if (!mbar_wait(bfull, (uint32_t)j & 1u, err, 26)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int a = 0; a < OZ_S; ++a, ++g) {
                    const int s = (int)(g & 1);
                    if (!mbar_wait(&afull[s], (uint32_t)(g >> 1) & 1u, err, 27)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    for (int b = 0; a + b < OZ_S; ++b) {
                        const uint32_t d = tmem + (uint32_t)((a + b) * OZ_N);
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const uint64_t da = smem_desc(smem + OzSmem::a + (s * 2 + h) * (OZ_M * 128));
                            const uint64_t db = smem_desc(smem + OzSmem::b + (b * 2 + h) * (OZ_N * 128));
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk) {
                                const uint64_t adv = (uint64_t)((kk * 32) >> 4);
                                umma_bf16(d, da + adv, db + adv, idesc, (a > 0 || h > 0 || kk > 0) ? 1u : 0u);
                            }
                        }
                    }
                    umma_commit(&aempty[s]);
                }
                if (!ok) break;
                umma_commit(bempty);
                umma_commit(tfull);
            }
            // every MMA of this CTA has finished before TMEM is released
            umma_commit(done);
            mbar_wait(done, 0, err, 29);
        }
    } else {   // epilogue warps 2..9
        const int q = warp & 3;   // TMEM lane quarter this warp may read
        const int half = (warp - 2) / 4 * 32;   // its columns of the tile
        double* stg = reinterpret_cast<double*>(smem + OzSmem::stage) + (size_t)(warp - 2) * 32 * OZ_W;
        auto prefetch_c = [&](int u) {   // the tile's rows of C into L2: 4 lines of 128 B per row
            int ti, tj;
            oz_tile(u, ntj, ti, tj);
            for (int t = threadIdx.x - 64; t < OZ_M * 4; t += 32 * OZ_EPI) {
                const int row = ti * OZ_M + t / 4, col = tj * OZ_N + (t % 4) * 16;
                if (row < m && col < m) asm volatile("prefetch.global.L2 [%0];" ::"l"(C + (int64_t)row * ldc + col));
            }
        };
        if ((int)blockIdx.x < ntiles) prefetch_c(blockIdx.x);
        int j = 0;
        for (int u = blockIdx.x; u < ntiles; u += gridDim.x, ++j) {
            int ti, tj;
            oz_tile(u, ntj, ti, tj);
            const int row0 = ti * OZ_M + q * 32;
            const int erow = row0 + lane < m ? ex[row0 + lane] : 0;   // row r's exponent from lane r
            const bool got = mbar_wait(tfull, (uint32_t)j & 1u, err, 28);
            if (!__all_sync(0xffffffffu, got)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (*err == 0) {
                // The diagonal sums S_D are exact integers in FP32: |S_D| <= 2^22 for D < 6,
                // read from the bits of S_D + MAGIC, and below 2^23 for the last two.
                // The element is sum_D S_D 2^(-7D-14) = V 2^-54 with the integer
                //   V = sum_{D<6} S_D 2^(40-7D) + round((S_6 2^7 + S_7) / 2^9),   |V| < 2^62,
                // so one rounding to 53 bits (as FP64 arithmetic would) and one FMA per
                // element remain in FP64; the rounded tail moves V by at most 2^-55.
#pragma unroll 1
                for (int c0 = half; c0 < half + 32; c0 += OZ_W) {
                    // lane l < 16: column l of the even rows, l >= 16: of the odd ones
                    const int cl = lane & (OZ_W - 1), col = tj * OZ_N + c0 + cl, rh = lane / OZ_W;
                    const int ecol = col < m ? ex[col] : 0;
                    double cold[OZ_W];   // all reads in flight before the sums are unpacked
#pragma unroll
                    for (int r = 0; r < OZ_W; ++r) {
                        const int row = row0 + 2 * r + rh;
                        cold[r] = (row < m && col < m && col >= row) ? C[(int64_t)row * ldc + col] : 0.0;
                    }
                    uint32_t v[OZ_S][OZ_W];
#pragma unroll
                    for (int D = 0; D < OZ_S; ++D) {
                        const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(D * OZ_N + c0);
                        asm volatile(
                            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,"
                            "%15}, [%16];"
                            : "=r"(v[D][0]), "=r"(v[D][1]), "=r"(v[D][2]), "=r"(v[D][3]), "=r"(v[D][4]),
                              "=r"(v[D][5]), "=r"(v[D][6]), "=r"(v[D][7]), "=r"(v[D][8]), "=r"(v[D][9]),
                              "=r"(v[D][10]), "=r"(v[D][11]), "=r"(v[D][12]), "=r"(v[D][13]), "=r"(v[D][14]),
                              "=r"(v[D][15])
                            : "r"(taddr));
                    }
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int c = 0; c < OZ_W; ++c) {
                        auto bits = [&](int D) { return __float_as_uint(__uint_as_float(v[D][c]) + MAGIC); };
                        constexpr unsigned k0 = MAGIC_BITS * 129u;
                        const int t01 = (int)(bits(0) * 128u + bits(1) - k0);
                        const int t23 = (int)(bits(2) * 128u + bits(3) - k0);
                        const int t45 = (int)(bits(4) * 128u + bits(5) - k0);
                        const int t67 = __float2int_rz(__uint_as_float(v[6][c])) * 128 +
                                        __float2int_rz(__uint_as_float(v[7][c]));
                        const long long V = (((long long)t01 << 28) + ((long long)t23 << 14) + t45) * 32 +
                                            ((t67 + 256) >> 9);
                        // rows of 16, columns rotated by the row: no bank conflicts either way
                        stg[lane * OZ_W + (c ^ (lane & (OZ_W - 1)))] = __longlong_as_double(V);
                    }
                    __syncwarp();
#pragma unroll
                    for (int r = 0; r < OZ_W; ++r) {
                        const int lr = 2 * r + rh, row = row0 + lr;
                        const int e = __shfl_sync(0xffffffffu, erow, lr) + ecol - 54;
                        if (row < m && col < m && col >= row)
                            C[(int64_t)row * ldc + col] =
                                fma(alpha, from_fixed(__double_as_longlong(stg[lr * OZ_W + (cl ^ (lr & (OZ_W - 1)))]), e),
                                    cold[r]);
                    }
                    __syncwarp();
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty);
            if (u + (int)gridDim.x < ntiles) prefetch_c(u + gridDim.x);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(OZ_S * OZ_N)
                     : "memory");
    }
}

}  // namespace cgd

// ================================================================ host side
namespace cg {

static void ck(cudaError_t e, const char* w) {
    if (e != cudaSuccess) throw std::runtime_error(std::string("CUDA error in ") + w + ": " + cudaGetErrorString(e));
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    if (!fn) throw std::runtime_error("cuTensorMapEncodeTiled is not available from the driver");
    return fn;
}

static CUtensorMap plane_map(void* base, int64_t kpad, int64_t cpad, int box_rows) {
    CUtensorMap m;
    cuuint64_t dims[2] = {(cuuint64_t)kpad, (cuuint64_t)cpad};
    cuuint64_t strides[1] = {(cuuint64_t)(kpad * 2)};
    cuuint32_t box[2] = {cgd::GB_K, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw std::runtime_error("cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
    return m;
}

// Streaming multiprocessors of the current device (cached per device).
static int device_sms() {
    static thread_local int dev_cached = -1, cached = 0;
    int dev = 0;
    ck(cudaGetDevice(&dev), "cudaGetDevice");
    if (dev != dev_cached) {
        ck(cudaDeviceGetAttribute(&cached, cudaDevAttrMultiProcessorCount, dev), "SM count");
        cached = std::max(1, cached);
        dev_cached = dev;
    }
    return cached;
}

// Blocks of k_split_atb<T> resident on the current device at once (cached per device).
template <typename T>
static int split_atb_resident() {
    static thread_local int dev_cached = -1, cached = 0;
    int dev = 0;
    ck(cudaGetDevice(&dev), "cudaGetDevice");
    if (dev != dev_cached) {
        int per_sm = 0, sms = 0;
        ck(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cgd::k_split_atb<T>, cgd::SPA_THREADS, 0),
           "occupancy");
        ck(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "SM count");
        cached = std::max(1, per_sm) * std::max(1, sms);
        dev_cached = dev;
    }
    return cached;
}

size_t gram_plane_bytes(int64_t nrows_block, int ncols) {
    const int64_t kpad = (nrows_block + cgd::GB_K - 1) / cgd::GB_K * cgd::GB_K;
    const int64_t cpad = (ncols + cgd::GB_M - 1) / cgd::GB_M * cgd::GB_M;
    return (size_t)(2 * cpad * kpad * 2);
}

void gram_accumulate(int prec_in, const void* A, int64_t lda, int64_t nrows, int ncols, const double* b, int mode,
                     double* G, double* h, void* planes, size_t planes_bytes, int* d_err, cudaStream_t st, const std::function<void(int, bool)>& mark, int ctas_per_sm) {
    if (nrows <= 0) return;
    // stage ids (session.h): ST_GRAM_ATB 11, ST_GRAM_SPLIT 12, ST_GRAM_TC 13, ST_GRAM_SYRK 14
    enum { S_ATB = 11, S_SPLIT = 12, S_TC = 13, S_SYRK = 14 };
    if (mode == 0) {   // h += A^T b (FP64, reproducible), then the FP64 SYRK of the block
        if (prec_in != 0) throw std::runtime_error("the FP64 Gram needs an FP64 A");
        double* partial = scratch_alloc<double>(atb_partial_doubles(nrows, ncols), st);
        mark(S_ATB, true);
        gemv_cols64((const double*)A, lda, nrows, ncols, b, h, partial, st);
        mark(S_ATB, false);
        ck(cudaFreeAsync(partial, st), "atb scratch free");
        mark(S_SYRK, true);
        gram64((const double*)A, lda, nrows, ncols, G, ncols, st);
        mark(S_SYRK, false);
        return;
    }
    // split-BF16 3-term on tcgen05, in row blocks that fit the plane buffer
    const int64_t cpad = (ncols + cgd::GB_M - 1) / cgd::GB_M * cgd::GB_M;
    int64_t rblock = (int64_t)(planes_bytes / (size_t)(2 * cpad * 2)) / cgd::GB_K * cgd::GB_K;
    if (rblock <= 0) throw std::runtime_error("Gram plane buffer too small");
    // column tiles of 256 when the triangle has at least two tiles per SM of those,
    // else of 128 (tiles that reach the upper triangle: tj >= ti / q)
    const int nti = (int)(cpad / cgd::GB_M);   // 128-row tiles
    auto pair_count = [&](int q) {
        const int ntj = (int)((ncols + q * cgd::GB_M - 1) / (q * cgd::GB_M));
        int n = 0;
        for (int tj = 0; tj < ntj; ++tj) n += std::min(nti, q * tj + q);
        return std::make_pair(ntj, n);
    };
    const int q = pair_count(2).second >= 2 * device_sms() ? 2 : 1;
    const int bn = q * cgd::GB_M;
    const int ntj = pair_count(q).first, npairs = pair_count(q).second;
    const size_t smem = (size_t)(q == 2 ? cgd::GbCfg<256>::total : cgd::GbCfg<128>::total) + 1024;
    if (q == 2)
        ck(cudaFuncSetAttribute(cgd::k_gram_tc<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
           "smem attr");
    else
        ck(cudaFuncSetAttribute(cgd::k_gram_tc<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
           "smem attr");
    // split + A^T b: one wave of resident blocks over the column strips (a second,
    // partial wave would double the pass)
    const int nstrip = (int)(cpad / cgd::SPA_C);
    const int64_t ktiles_max = (std::min(rblock, nrows) + cgd::SPA_K - 1) / cgd::SPA_K;
    const int resident = prec_in == 0 ? split_atb_resident<double>() : split_atb_resident<float>();
    const int gx = (int)std::max<int64_t>(1, std::min<int64_t>(ktiles_max, resident / nstrip));
    float2* bsplit = nullptr;
    double* partial = scratch_alloc<double>((size_t)gx * ncols, st);
    const int64_t kpad_max = (std::min(rblock, nrows) + cgd::GB_K - 1) / cgd::GB_K * cgd::GB_K;
    if (prec_in != 0) bsplit = scratch_alloc<float2>(kpad_max, st);
    for (int64_t r0 = 0; r0 < nrows; r0 += rblock) {
        const int64_t nr = std::min(rblock, nrows - r0);
        const int64_t kpad = (nr + cgd::GB_K - 1) / cgd::GB_K * cgd::GB_K;
        __nv_bfloat16* hi = (__nv_bfloat16*)planes;
        __nv_bfloat16* lo = hi + cpad * kpad;
        const int gxb = (int)std::min<int64_t>(gx, (kpad + cgd::SPA_K - 1) / cgd::SPA_K);
        dim3 tg((unsigned)gxb, (unsigned)nstrip);
        mark(S_SPLIT, true);
        if (prec_in == 0) {
            cgd::k_split_atb<double><<<tg, cgd::SPA_THREADS, 0, st>>>((const double*)A, lda, r0, nr, ncols, b, nullptr,
                                                                     hi, lo, kpad, partial);
        } else {
            cgd::k_split_b<<<(unsigned)((kpad + 255) / 256), 256, 0, st>>>(b, r0, nr, kpad, bsplit);
            cgd::k_split_atb<float><<<tg, cgd::SPA_THREADS, 0, st>>>((const float*)A, lda, r0, nr, ncols, nullptr,
                                                                    bsplit, hi, lo, kpad, partial);
        }
        mark(S_SPLIT, false);
        ck(cudaGetLastError(), "k_split_atb");
        mark(S_ATB, true);
        cgd::k_split_reduce<<<(ncols + 127) / 128, 128, 0, st>>>(partial, gxb, ncols, h);
        mark(S_ATB, false);
        ck(cudaGetLastError(), "k_split_reduce");
        CUtensorMap mhi_a = plane_map(hi, kpad, cpad, cgd::GB_M), mlo_a = plane_map(lo, kpad, cpad, cgd::GB_M);
        CUtensorMap mhi_b = plane_map(hi, kpad, cpad, bn), mlo_b = plane_map(lo, kpad, cpad, bn);
        // K slices: the persistent grid (one CTA per SM) runs npairs * nslice units
        // in waves; pick nslice (at most ctas_per_sm units per SM) minimising the K
        // steps on the longest CTA's path, waves * ceil(ksteps / nslice), plus one
        // step per wave for the unit switch.
        // With the wide tile a unit spans at most 128 K steps: over longer ranges the
        // CTAs drift apart along K and the operand tiles they share leave L2.
        const int64_t ksteps = kpad / cgd::GB_K;
        const int64_t sms = device_sms();
        const int64_t smin = q == 2 ? std::max<int64_t>(1, (ksteps + 127) / 128) : 1;
        const int64_t smax = std::max<int64_t>(
            smin, std::min<int64_t>(ksteps, sms * std::max(1, ctas_per_sm) / std::max(1, npairs)));
        int64_t nslice = smin, best = INT64_MAX;
        for (int64_t sl = smin; sl <= smax; ++sl) {
            const int64_t waves = (npairs * sl + sms - 1) / sms;
            const int64_t cost = waves * ((ksteps + sl - 1) / sl + 1);
            if (cost < best) { best = cost; nslice = sl; }
        }
        const int64_t kslice = (ksteps + nslice - 1) / nslice * cgd::GB_K;
        nslice = (kpad + kslice - 1) / kslice;
        const int64_t nunits = (int64_t)npairs * nslice;
        if (nunits > INT32_MAX) throw std::runtime_error("too many Gram tiles");
        const unsigned grid = (unsigned)std::min<int64_t>(nunits, device_sms());
        mark(S_TC, true);
        if (q == 2)
            cgd::k_gram_tc<256><<<grid, cgd::GB_THREADS, smem, st>>>(mhi_a, mlo_a, mhi_b, mlo_b, nti, ntj, npairs,
                                                                     (int)nunits, kpad, kslice, ncols, G, d_err);
        else
            cgd::k_gram_tc<128><<<grid, cgd::GB_THREADS, smem, st>>>(mhi_a, mlo_a, mhi_b, mlo_b, nti, ntj, npairs,
                                                                     (int)nunits, kpad, kslice, ncols, G, d_err);
        mark(S_TC, false);
        ck(cudaGetLastError(), "k_gram_tc");
    }
    ck(cudaFreeAsync(partial, st), "atb scratch free");
    if (bsplit) ck(cudaFreeAsync(bsplit, st), "b split scratch free");
}

size_t ozaki_scratch_bytes(int m_max) {
    const size_t mpad = (size_t)(std::max(m_max, 1) + 127) / 128 * 128;
    return 256 + (mpad * sizeof(double) + 255) / 256 * 256 + (size_t)cgd::OZ_S * mpad * cgd::OZ_K * 2;
}

void syrk_update_ozaki(const double* X, int64_t ldx, int K, int m, double alpha, double* C, int64_t ldc,
                       void* scratch, cudaStream_t st) {
    if (m <= 0 || K <= 0) return;
    if (K > cgd::OZ_K) throw std::runtime_error("syrk_update_ozaki: panel wider than 128");
    const int mpad = (m + 127) / 128 * 128;
    int* d_err = static_cast<int*>(scratch);
    int* ex = reinterpret_cast<int*>(static_cast<char*>(scratch) + 256);
    __nv_bfloat16* P = reinterpret_cast<__nv_bfloat16*>(static_cast<char*>(scratch) + 256 +
                                                        ((size_t)mpad * sizeof(double) + 255) / 256 * 256);
    cgd::k_oz_slice<<<mpad / 32, 256, 0, st>>>(X, ldx, K, m, mpad, P, ex);
    ck(cudaGetLastError(), "k_oz_slice");
    const CUtensorMap ma = plane_map(P, cgd::OZ_K, (int64_t)cgd::OZ_S * mpad, cgd::OZ_M);
    const CUtensorMap mb = plane_map(P, cgd::OZ_K, (int64_t)cgd::OZ_S * mpad, cgd::OZ_N);
    const int ntj = (m + cgd::OZ_N - 1) / cgd::OZ_N, rows = (ntj + 1) / 2;
    const int64_t ntiles = (int64_t)rows * (ntj + 1 - rows);
    const size_t smem = (size_t)cgd::OzSmem::total + 1024;
    static thread_local int attr_dev = -1;
    int dev = 0;
    ck(cudaGetDevice(&dev), "cudaGetDevice");
    if (attr_dev != dev) {
        ck(cudaFuncSetAttribute(cgd::k_oz_syrk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "smem attr");
        attr_dev = dev;
    }
    if (ntiles > INT32_MAX) throw std::runtime_error("syrk_update_ozaki: too many tiles");
    const unsigned grid = (unsigned)std::min<int64_t>(ntiles, device_sms());
    cgd::k_oz_syrk<<<grid, cgd::OZ_THREADS, smem, st>>>(ma, mb, ex, m, mpad, ntj, (int)ntiles, alpha, C, ldc, d_err);
    ck(cudaGetLastError(), "k_oz_syrk");
}

void gram_symmetrize(double* G, int n, bool from_upper, cudaStream_t st) {
    (void)from_upper;
    if (n <= 0) return;
    const unsigned nb = (unsigned)((n + cgd::SY_B - 1) / cgd::SY_B);
    cgd::k_symmetrize<<<dim3(nb, nb), cgd::SY_THREADS, 0, st>>>(G, n);
    ck(cudaGetLastError(), "k_symmetrize");
}

}  // namespace cg
