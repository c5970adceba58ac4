// FP64 dense kernels of the normal-equations solve (see dense64.h).
//
// The reference solves its least-squares problem with numpy's SVD on the CPU
// (src/chimes_lsq.py:169-214).  On this GPU the FP64 pipe delivers about 1/64 of
// the FP32 rate, so every kernel here is shaped around the FP64 FMA rate rather
// than around bytes: register-blocked tiles (16 FMAs per 8 shared-memory loads in
// the SYRK), and enough independent CTAs per SM to keep the pipe issuing.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <stdexcept>
#include <string>

#include "dense64.h"
#include "digits.cuh"
#include "gram.h"
#include "scratch.h"

namespace cgd {

// ---------------------------------------------------------------- SYRK (X^T X)
constexpr int SY_T = 64, SY_KC = 16, SY_THREADS = 256;

// (ti, tj), ti <= tj, of the linear index t over the upper triangle of ntile x ntile
// tiles stored by rows (row ti holds ntile - ti pairs).
__device__ __forceinline__ void upper_pair(int64_t t, int ntile, int& ti, int& tj) {
    const double b = 2.0 * ntile + 1.0;
    int64_t r = (int64_t)floor((b - sqrt(b * b - 8.0 * (double)t)) * 0.5);
    r = max((int64_t)0, min((int64_t)ntile - 1, r));
    auto start = [&](int64_t x) { return x * ntile - x * (x - 1) / 2; };
    while (r > 0 && start(r) > t) --r;
    while (r + 1 < ntile && start(r + 1) <= t) ++r;
    ti = (int)r;
    tj = (int)(r + (t - start(r)));
}

// grid.x: upper tile pair, grid.y: K slice.  Thread (ty, tx) of a 16 x 16 layout owns
// C rows ty + 16u and columns tx + 16v of the 64 x 64 tile (u, v < 4).
template <bool ATOMIC>
__global__ void __launch_bounds__(SY_THREADS) k_syrk_tn(const double* __restrict__ X, int64_t ldx, int64_t K, int m,
                                                        double alpha, double* __restrict__ C, int64_t ldc, int ntile,
                                                        int64_t kslice) {
    __shared__ double As[SY_KC][SY_T];
    __shared__ double Bs[SY_KC][SY_T];
    int ti, tj;
    upper_pair(blockIdx.x, ntile, ti, tj);
    const bool diag = ti == tj;
    const int64_t kb = (int64_t)blockIdx.y * kslice, ke = min(K, kb + kslice);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int ci = ti * SY_T, cj = tj * SY_T;
    double acc[4][4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] = 0.0;
    for (int64_t k0 = kb; k0 < ke; k0 += SY_KC) {
#pragma unroll
        for (int q = 0; q < SY_KC * SY_T / SY_THREADS; ++q) {
            const int idx = threadIdx.x + q * SY_THREADS;
            const int kk = idx / SY_T, c = idx % SY_T;
            const int64_t k = k0 + kk;
            const bool kin = k < ke;
            As[kk][c] = (kin && ci + c < m) ? X[k * ldx + ci + c] : 0.0;
            if (!diag) Bs[kk][c] = (kin && cj + c < m) ? X[k * ldx + cj + c] : 0.0;
        }
        __syncthreads();
        const double(*Bp)[SY_T] = diag ? As : Bs;
#pragma unroll
        for (int kk = 0; kk < SY_KC; ++kk) {
            double a[4], b[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) a[u] = As[kk][ty + 16 * u];
#pragma unroll
            for (int v = 0; v < 4; ++v) b[v] = Bp[kk][tx + 16 * v];
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < 4; ++v) acc[u][v] = fma(a[u], b[v], acc[u][v]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int i = ci + ty + 16 * u;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const int j = cj + tx + 16 * v;
            if (i < m && j < m && j >= i) {
                double* p = C + (int64_t)i * ldc + j;
                if (ATOMIC) atomicAdd(p, alpha * acc[u][v]);
                else *p += alpha * acc[u][v];
            }
        }
    }
}

// ---------------------------------------------------------------- X^T X as digit products
// The same triangle from the tensor cores (digits.cuh) with the accuracy of FP64 sums, entry
// by entry.  Every 32 rows (a block) each column has its own power of two; its entries are
// split into eight base-256 digits, a 64 x 64 tile's 36 digit products per term are summed
// exactly over the block, and the blocks' sums exactly in 128-bit integers, in units of 2^-88 of
// the product of the columns' largest powers of two; one rounding to FP64 at the end.  In units
// of its two powers of two a block loses about 2^-61.6 (32 terms whose dropped diagonals are
// 2^-64.1 each, root mean square), and nothing in rows where either entry is zero.
//
// That is less than FP64 sums lose -- at least 2^-55 of S_ij = sum |x_ki x_kj| -- unless the
// rows of the large entries of one column meet small ones of the other.  So a ninth plane
// holds |x| in FP16 and one more product per 16 rows estimates S: an output whose S is below
// GD_GUARD times the root of its blocks' squared units is summed again in FP64 by the same
// CTA (as are columns that are not finite).  Of a C/H 4-body A of 816 x 3,992 that is 2.5% of
// the outputs, of a water 3-body A of 13,968 x 820 none.
//
// Sixteen warps of 16 rows x 16 columns; the next 16 rows' digits are built while warps that
// have finished theirs run the current products.  The tensor pipe is the bound (36
// products per multiply-add on mma.sync, 606 TFLOP/s measured, or 13.9 TFLOP/s of FP64
// arithmetic).  (Blocks rounded to FP64 and added there took 4.8 ms at 30,001 x 820, at 32 rows a
// block, 4.4 at 64: an addition at 1/64 of the FP32 rate keeps the tensor pipe waiting.)
//
// Whole calls with h, FP64 sums -> this: 30,001 x 820 19.3 -> 4.26 ms, 2,000 x 6,007 60.0 -> 14.0,
// 816 x 3,992 11.5 -> 2.8; entries spread by exp(2 N(0,1)): 19.3 -> 5.6, 60.0 -> 18.0, 11.5 -> 3.5.
// Error over S against long double, root mean square: 30,001 x 820 1.9e-17 -> 1.3e-18, spread
// entries 2.6e-16 -> 2.1e-17.  (One power of two per column over all rows and one 64-bit integer
// over a CTA's rows took 3.51 ms, but lost 7e-13 of S with spread entries.)
constexpr int GD_T = 64, GD_THREADS = 512, GD_ROWS = 16, GD_BLOCK = 32;
constexpr uint32_t GD_CHUNK = 2 * GD_T * DIG_STRIDE;   // 8 rows of K
constexpr uint32_t GD_BUF = 2 * GD_CHUNK;
constexpr uint32_t GD_ABS = 16 * DIG_ND;               // the FP16 plane, in a row's padding
static_assert(GD_ABS + 16 <= DIG_STRIDE, "padding of a row");
constexpr float GD_GUARD = 1.0f / 96.0f;               // 2^-61.6 / GD_GUARD <= 2^-55
constexpr int GD_FRAC = 18;                            // a block's integer sums are kept times 2^GD_FRAC or less
struct GdSmem {
    // [8][threads]: the integer sums; the guard's sum of S and of the squared units
    static constexpr size_t sum = 2 * GD_BUF;
    static constexpr size_t guard = sum + 8 * GD_THREADS * sizeof(__int128);
    static constexpr size_t shift = guard + 8 * GD_THREADS * sizeof(float2);   // [2][2 GD_T] a block's powers of two
    static constexpr size_t total = shift + 2 * 2 * GD_T * sizeof(int);
    static_assert(sum % 16 == 0, "alignment");
    // of the FP64 sums, over the digits: 64 rows of the two column groups, the outputs' list
    static constexpr int frows = 64;
    static constexpr size_t list = 2 * frows * GD_T * sizeof(double);
    static_assert(list + GD_T * GD_T * sizeof(uint16_t) <= sum, "fits over the digits");
};

// The least e with |x| < 0.9942 2^e: the digits' bias adds 0x80..80 / 2^63 = 1.0039, and the
// sum stays below 2.  COL_BAD for infinities and NaN.
constexpr int COL_BAD = 4096;
__device__ __forceinline__ int col_exponent(double x) {
    const int h = __double2hiint(x) & 0x7fffffff;
    return h >= 0x7ff00000 ? COL_BAD : (h >> 20) - 1022 + ((h & 0xfffff) >= 0xfd000 ? 1 : 0);
}
// eb[block][c]: col_exponent of the block's largest entry of column c; ex[c] their largest
// (preset to a very small value).  A warp per (block, 32 columns).
__global__ void __launch_bounds__(256) k_col_exponents(const double* __restrict__ X, int64_t ldx, int64_t K, int m,
                                                int* __restrict__ ex, int16_t* __restrict__ eb) {
    const int c = blockIdx.x * 32 + (threadIdx.x & 31);
    if (c >= m) return;
    int top = -1022;
    for (int64_t b = (int64_t)blockIdx.y * 8 + (threadIdx.x >> 5); b * GD_BLOCK < K; b += (int64_t)gridDim.y * 8) {
        const int64_t k0 = b * GD_BLOCK, k1 = min(K, k0 + GD_BLOCK);
        int lg = -1022;
        int64_t k = k0;
        for (; k + 8 <= k1; k += 8) {   // eight loads in flight
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = X[(k + u) * ldx + c];
#pragma unroll
            for (int u = 0; u < 8; ++u) lg = max(lg, col_exponent(v[u]));
        }
        for (; k < k1; ++k) lg = max(lg, col_exponent(X[k * ldx + c]));
        eb[b * m + c] = (int16_t)lg;
        top = max(top, lg);
    }
    atomicMax(ex + c, top);
}

template <bool ATOMIC>
__global__ void __launch_bounds__(GD_THREADS, 1) k_syrk_digits(const double* __restrict__ X, int64_t ldx, int64_t K,
                                                               int m, double* __restrict__ C, int64_t ldc, int ntile,
                                                               int64_t kslice, const int* __restrict__ ex,
                                                               const int16_t* __restrict__ eb) {
    extern __shared__ __align__(16) unsigned char smem[];
    int ti, tj;
    upper_pair(blockIdx.x, ntile, ti, tj);
    const bool diag = ti == tj;
    const int64_t kb = (int64_t)blockIdx.y * kslice, ke = min(K, kb + kslice);   // kslice: a multiple of GD_BLOCK
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // digits: a warp has 8 columns (of tile ti, then tj), a lane one column and the row pairs
    // p and p + 4 of the 16, so that the 32 stores of a digit fall into different banks
    const int dc = warp * 8 + (lane >> 2), p = lane & 3;
    const int col = (dc < GD_T ? ti * GD_T + dc : tj * GD_T + dc - GD_T);
    const bool builds = !(diag && dc >= GD_T);
    const bool in = builds && col < m;
    const int top = in ? ex[col] : 0;
    double v[4];
    int e = 0;
    int* const sShift = reinterpret_cast<int*>(smem + GdSmem::shift);
    auto fetch = [&](int64_t k0) {
        e = in ? eb[k0 / GD_BLOCK * m + col] : 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t k = k0 + 2 * p + (u & 1) + 8 * (u >> 1);
            v[u] = in && k < ke ? X[k * ldx + col] : 0.0;
        }
    };
    // |x| / 2^e of two entries in FP16; what is not zero stays above zero
    auto sizes = [&](double x0, double x1, long long X0, long long X1) {
        auto f = [](double x, long long Xi) {
            const unsigned hi = (unsigned)((unsigned long long)(Xi < 0 ? -Xi : Xi) >> 32);
            const float y = __uint2float_rn(hi) * 0x1p-31f;
            return (__double_as_longlong(x) & 0x7fffffffffffffffll) == 0 ? 0.0f : fmaxf(y, 0x1p-24f);
        };
        return __floats2half2_rn(f(x0, X0), f(x1, X1));
    };
    auto build = [&](int i) {
        if (!builds) return;
        const int sh = DIG_FIX - e;
        unsigned char* row = smem + (i & 1) * GD_BUF + dc * DIG_STRIDE + 4 * p;
        if ((i & 1) == 0 && p == 0) sShift[(i >> 1 & 1) * 2 * GD_T + dc] = e - top;
#pragma unroll
        for (int c8 = 0; c8 < 2; ++c8) {
            const long long X0 = to_fixed(v[2 * c8], sh), X1 = to_fixed(v[2 * c8 + 1], sh);
            put_digits(row + c8 * GD_CHUNK, X0, X1);
            *reinterpret_cast<__half2*>(row + c8 * GD_CHUNK + GD_ABS) = sizes(v[2 * c8], v[2 * c8 + 1], X0, X1);
        }
    };
    const int mt = warp >> 2, nt = (warp & 3) * 2, g4 = lane >> 2, t4 = lane & 3;
    float acc[2][DIG_ND][4], s[2][4];
    const uint32_t base = smem_addr(smem);
    const int bcol = diag ? 0 : GD_T;   // the second column group's first row of digits
    auto products = [&](int i) {
        const uint32_t t = base + (i & 1) * GD_BUF;
#pragma unroll 1
        for (int c8 = 0; c8 < 2; ++c8) {
            uint32_t fa[DIG_ND][2], fb[DIG_ND];
            load_a(fa, t + c8 * GD_CHUNK + (uint32_t)(16 * mt) * DIG_STRIDE);
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                load_b(fb, t + c8 * GD_CHUNK + (uint32_t)(bcol + 8 * (nt + x)) * DIG_STRIDE);
                mma_digits(acc[x], fa, fb);
            }
        }
        uint32_t a[4], b[4];   // the FP16 plane: both groups of 8 rows in one product
        ldsm4(a, t + (lane >> 4) * GD_CHUNK + (uint32_t)(16 * mt + (lane & 15)) * DIG_STRIDE + GD_ABS);
        ldsm4(b, t + (lane >> 3 & 1) * GD_CHUNK + (uint32_t)(bcol + 8 * (nt + (lane >> 4)) + (lane & 7)) * DIG_STRIDE + GD_ABS);
#pragma unroll
        for (int x = 0; x < 2; ++x) mma_f16(s[x], a, b[2 * x], b[2 * x + 1]);
    };
    __int128* const sSum = reinterpret_cast<__int128*>(smem + GdSmem::sum) + threadIdx.x;
    float2* const sGuard = reinterpret_cast<float2*>(smem + GdSmem::guard) + threadIdx.x;
    // A block's sums to the outputs', in units of 2^(ex_i + ex_j - 70 - GD_FRAC): what a power of
    // two below 2^-GD_FRAC shifts out is below the block's own loss down to 2^-29, so the guard
    // counts a smaller unit as that.
    auto flush = [&](int block) {
        const int* sh = sShift + (block & 1) * 2 * GD_T;
#pragma unroll
        for (int x = 0; x < 2; ++x) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int o = (4 * x + r) * GD_THREADS;
                const int d = sh[16 * mt + g4 + 8 * (r >> 1)] + sh[bcol + 8 * (nt + x) + 2 * t4 + (r & 1)];
                int fr;
                const long long w = acc_parts(acc[x], r, fr);
                const __int128 v = ((__int128)w << 16) + fr;
                sSum[o] += d >= -GD_FRAC ? v << (d + GD_FRAC) : v >> min(-GD_FRAC - d, 127);
                if (s[x][r] > 0.0f) {
                    const float u = __int_as_float((127 + max(d, -29)) << 23);
                    float2 g = sGuard[o];
                    g.x = fmaf(s[x][r], d < -60 ? 0.0f : __int_as_float((127 + d) << 23), g.x);
                    g.y = fmaf(u, u, g.y);
                    sGuard[o] = g;
                }
                s[x][r] = 0.0f;
            }
            acc_clear(acc[x]);
        }
    };
    static_assert(GD_BLOCK <= MAGIC_TERMS && GD_BLOCK == 2 * GD_ROWS, "exact accumulators");
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        acc_clear(acc[x]);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int o = (4 * x + r) * GD_THREADS;
            sSum[o] = 0;
            sGuard[o] = make_float2(0.0f, 0.0f);
            s[x][r] = 0.0f;
        }
    }
    const int nch = ke > kb ? (int)((ke - kb + GD_ROWS - 1) / GD_ROWS) : 0;
    if (nch > 0) {
        fetch(kb);
        build(0);
        if (nch > 1) fetch(kb + GD_ROWS);
        __syncthreads();
    }
    for (int i = 0; i < nch; ++i) {
        if (i + 1 < nch) build(i + 1);
        if (i + 2 < nch) fetch(kb + (int64_t)(i + 2) * GD_ROWS);
        products(i);
        if ((i & 1) || i + 1 == nch) flush(i >> 1);
        __syncthreads();
    }
    __shared__ int nlist;
    uint16_t* const list = reinterpret_cast<uint16_t*>(smem + GdSmem::list);
    if (threadIdx.x == 0) nlist = 0;
    __syncthreads();   // the digits' last readers are done
    auto add = [&](int i, int j, double g) {
        double* o = C + (int64_t)i * ldc + j;
        if (ATOMIC) atomicAdd(o, g);
        else *o += g;
    };
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int li = 16 * mt + g4 + 8 * (r >> 1), lj = 8 * (nt + x) + 2 * t4 + (r & 1);
            const int i = ti * GD_T + li, j = tj * GD_T + lj;
            if (i < m && j < m && j >= i) {
                const int ei = ex[i], ej = ex[j];
                const int o = (4 * x + r) * GD_THREADS;
                if (sGuard[o].x >= GD_GUARD * sqrtf(sGuard[o].y) && ei != COL_BAD && ej != COL_BAD)
                    add(i, j, int128_double(sSum[o], ei + ej - 70 - GD_FRAC));
                else
                    list[atomicAdd(&nlist, 1)] = (uint16_t)(li * GD_T + lj);
            }
        }
    __syncthreads();
    // the outputs that digits do not hold, by FP64 multiply-adds row after row
    const int n = nlist;
    constexpr int FR = GdSmem::frows;
    double* const sA = reinterpret_cast<double*>(smem);
    double* const sB = diag ? sA : sA + FR * GD_T;
    for (int at = 0; at < n; at += GD_THREADS) {
        const bool on = at + (int)threadIdx.x < n;
        const int o = on ? list[at + threadIdx.x] : 0, li = o / GD_T, lj = o % GD_T;
        double g = 0.0;
        for (int64_t k0 = kb; k0 < ke; k0 += FR) {
            __syncthreads();
#pragma unroll 8
            for (int t = threadIdx.x; t < (diag ? 1 : 2) * FR * GD_T; t += GD_THREADS) {
                const int half = t / (FR * GD_T), kk = t / GD_T % FR, c = (half ? tj : ti) * GD_T + t % GD_T;
                sA[t] = k0 + kk < ke && c < m ? X[(k0 + kk) * ldx + c] : 0.0;
            }
            __syncthreads();
            if (on)
#pragma unroll 16
                for (int kk = 0; kk < FR; ++kk) g = fma(sA[kk * GD_T + li], sB[kk * GD_T + lj], g);
        }
        if (on) add(ti * GD_T + li, tj * GD_T + lj, g);
    }
}

// ---------------------------------------------------------------- Cholesky
constexpr int CH_NB = 128;

// A panel of CH_NB columns is factorised as two halves of CH_H.  The FP64 pipe does 2
// multiply-adds a clock per SM, so one SM needs 90 us for a 128 x 128 block and 130 us for 64
// rows of the panel below; with one CTA for the block and 64 rows per CTA a panel of n =
// 5,000 took 535 us, most of the GPU idle.  Here every CTA factorises the 64 x 64 block for
// itself (11 us of multiply-adds) and solves its share of the rows below, one share per SM,
// and the second half's columns are updated from the first's by a third launch.  n = 5,000:
// the panels 21.2 -> 7.3 ms; n = 1,000: the whole factorisation 4.66 -> 1.64 ms.
constexpr int CH_H = 64, CH_B = 16, CH_LD = CH_H + 1, CH_THREADS = 256;

// 16 x 16 diagonal sub-block at b0 of D (bs valid columns), by warp 0: lane r + 16 h holds
// row r, columns 2 i + h, so that one instruction updates two columns (a warp's FP64
// instruction takes 64 cycles of its SM quarter whatever the lanes do).  L D L^T first, one
// reciprocal per column in the chain, and the square roots of all pivots at the end.  A
// pivot that is not positive becomes 1; bad receives its column + 1 (the first).  TINY: pivots
// below 2^-1000 are scaled, as the reciprocal of one below 2^-1024 is not finite.
template <bool TINY>
__device__ __forceinline__ void chol16(double* D, int b0, int bs, double* rdiag, int* bad) {
    const int lane = threadIdx.x & 31, r = lane & 15, h = lane >> 4;
    double a[CH_B / 2], piv = 1.0;
#pragma unroll
    for (int i = 0; i < CH_B / 2; ++i) {
        const int c = 2 * i + h;
        a[i] = r < bs && c <= r ? D[(b0 + r) * CH_LD + b0 + c] : (c == r ? 1.0 : 0.0);
    }
#pragma unroll
    for (int j = 0; j < CH_B; ++j) {
        const double v = __shfl_sync(0xffffffffu, a[j >> 1], r + 16 * (j & 1));   // column j, row r
        double d = __shfl_sync(0xffffffffu, v, j);
        if (!(d > 0.0)) {
            if (lane == 0 && j < bs && *bad == 0) *bad = b0 + j + 1;
            d = 1.0;
        }
        if (r == j) piv = d;
        double w = v;
        if (TINY && d < 0x1p-1000) { d *= 0x1p200; w *= 0x1p200; }
        const double l = w * __drcp_rn(d);
#pragma unroll
        for (int i = j >> 1; i < CH_B / 2; ++i) {
            const int c = 2 * i + h;
            const double vc = __shfl_sync(0xffffffffu, v, c);
            if (c > j && c <= r) a[i] = fma(-l, vc, a[i]);
        }
        if (h == (j & 1)) a[j >> 1] = r == j ? 1.0 : l;
    }
    const double sd = sqrt(piv);
    if (h == 0) rdiag[b0 + r] = 1.0 / sd;
#pragma unroll
    for (int i = 0; i < CH_B / 2; ++i) {
        const int c = 2 * i + h;
        const double x = a[i] * __shfl_sync(0xffffffffu, sd, c);
        if (r < bs && c < bs) D[(b0 + r) * CH_LD + b0 + c] = c <= r ? x : 0.0;
    }
}

// Columns k .. k + kb of the column-major lower matrix (leading dimension n, kb <= 64):
// the diagonal block's factor and the m rows below it, R rows per CTA.  While warp 0
// factorises the next 16 columns' diagonal sub-block, the others finish the update of the
// columns after them.  status: a counter of the launch's CTAs, and a word that becomes 1 if a
// pivot was below 2^-1020 (the factorisation may have failed for want of TINY, which costs 1 to 3%
// of it, in the chain of pivots).
template <bool TINY>
__global__ void __launch_bounds__(CH_THREADS) k_chol_half(double* __restrict__ G, int n, int k, int kb, int m, int R,
                                                          int second, int* info, int* __restrict__ status) {
    extern __shared__ double sm[];
    double* D = sm;                          // rows 0 .. kb: the block, then this CTA's rows
    __shared__ double rdiag[CH_H];
    __shared__ int bad, last;
    const int i0 = blockIdx.x * R, rows = min(R, m - i0), tot = CH_H + max(rows, 0);
    if (threadIdx.x == 0) bad = 0;
    {   // every load of the block in flight at once, then the rows
        double v[CH_H * CH_H / CH_THREADS];
#pragma unroll
        for (int u = 0; u < CH_H * CH_H / CH_THREADS; ++u) {
            const int idx = threadIdx.x + u * CH_THREADS, i = idx % CH_H, j = idx / CH_H;
            v[u] = i < kb && j <= i ? G[(int64_t)(k + j) * n + k + i] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < CH_H * CH_H / CH_THREADS; ++u) {
            const int idx = threadIdx.x + u * CH_THREADS;
            D[(idx % CH_H) * CH_LD + idx / CH_H] = v[u];
        }
        for (int r = threadIdx.x & 31; r < rows; r += 32) {
            const int w = threadIdx.x >> 5;
#pragma unroll
            for (int u = 0; u < CH_H / 8; ++u) {
                const int j = w + 8 * u;
                v[u] = j < kb ? G[(int64_t)(k + j) * n + k + kb + i0 + r] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < CH_H / 8; ++u) D[(CH_H + r) * CH_LD + w + 8 * u] = v[u];
        }
    }
    __syncthreads();
    // columns [c0, c1) of the rows from c0 on minus the product with the sub-block's columns
    // at b0, by threads t0, t0 + step, ...: four columns per item, rows across the lanes
    auto update = [&](int b0, int c0, int c1, int t0, int step) {
        const int ng = (c1 - c0 + 3) >> 2, nr = tot - c0;
        for (int t = t0; t < nr * ng; t += step) {
            const int g = t / nr, r = c0 + t - g * nr, c = c0 + 4 * g;
            if (r < CH_H && (r < c || r >= kb)) continue;
            const double* p = D + r * CH_LD + b0;
            double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int l = 0; l < CH_B; ++l) {
                const double v = p[l];
#pragma unroll
                for (int q = 0; q < 4; ++q) s[q] = fma(v, D[min(c + q, CH_H - 1) * CH_LD + b0 + l], s[q]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) if (c + q < c1) D[r * CH_LD + c + q] -= s[q];
        }
    };
    for (int b0 = 0; b0 < kb; b0 += CH_B) {
        const int bs = min(CH_B, kb - b0);
        if (threadIdx.x < 32) chol16<TINY>(D, b0, bs, rdiag, &bad);
        else if (b0 > 0 && b0 + CH_B < kb) update(b0 - CH_B, b0 + CH_B, kb, threadIdx.x - 32, CH_THREADS - 32);
        __syncthreads();
        // the sub-block's columns of every row below, a row per thread
        for (int r = b0 + CH_B + threadIdx.x; r < tot; r += CH_THREADS) {
            double* p = D + r * CH_LD + b0;
            double x[CH_B];
#pragma unroll
            for (int j = 0; j < CH_B; ++j) {
                double v = j < bs ? p[j] : 0.0;
#pragma unroll
                for (int l = 0; l < j; ++l) v = fma(-x[l], D[(b0 + j) * CH_LD + b0 + l], v);
                x[j] = j < bs ? v * rdiag[b0 + j] : 0.0;
            }
#pragma unroll
            for (int j = 0; j < CH_B; ++j) if (j < bs) p[j] = x[j];
        }
        __syncthreads();
        // the next sub-block's columns now, those after it beside its factorisation
        if (b0 + CH_B < kb) {
            update(b0, b0 + CH_B, min(kb, b0 + 2 * CH_B), threadIdx.x, CH_THREADS);
            __syncthreads();
        }
    }
    for (int j = threadIdx.x >> 5; j < kb; j += CH_THREADS / 32)
        for (int r = threadIdx.x & 31; r < rows; r += 32)
            G[(int64_t)(k + j) * n + k + kb + i0 + r] = D[(CH_H + r) * CH_LD + j];
    // the block's factor, by the last CTA: every other has read the block by then
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(status, 1) == (int)gridDim.x - 1;
        if (last) *status = 0;
    }
    __syncthreads();
    if (!last) return;
    for (int idx = threadIdx.x; idx < kb * kb; idx += blockDim.x) {
        const int i = idx % kb, j = idx / kb;
        G[(int64_t)(k + j) * n + k + i] = i >= j ? D[i * CH_LD + j] : 0.0;
    }
    if (second)   // the block above it, of the 128-wide block's upper triangle
        for (int idx = threadIdx.x; idx < CH_H * kb; idx += blockDim.x)
            G[(int64_t)(k + idx / CH_H) * n + k - CH_H + idx % CH_H] = 0.0;
    if (threadIdx.x == 0 && bad) atomicCAS(info, 0, k + bad);
    if (!TINY && threadIdx.x < kb && rdiag[threadIdx.x] > 0x1p510) status[1] = 1;
}

// The second half's columns, rows k0 + 64 and below: minus the first half's product.
// 16 rows x kb2 columns per CTA (32 rows, 131,000 multiply-adds: 33 us of an SM), four
// columns per thread.
constexpr int ST_R = 16;
__global__ void __launch_bounds__(256) k_chol_strip(double* __restrict__ G, int n, int k0, int kb2) {
    __shared__ double Ls[CH_H][CH_H];    // Ls[l][c] = L(k0 + 64 + c, k0 + l)
    __shared__ double Ps[CH_H][ST_R];
    const int r = threadIdx.x % ST_R, c0 = threadIdx.x / ST_R * 4;
    const int row = k0 + CH_H + blockIdx.x * ST_R + r;
    {
        double v[CH_H * CH_H / 256], p[CH_H * ST_R / 256];
#pragma unroll
        for (int u = 0; u < CH_H * CH_H / 256; ++u) {
            const int idx = threadIdx.x + 256 * u, c = idx % CH_H, l = idx / CH_H;
            v[u] = c < kb2 ? G[(int64_t)(k0 + l) * n + k0 + CH_H + c] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < CH_H * ST_R / 256; ++u)
            p[u] = row < n ? G[(int64_t)(k0 + threadIdx.x / ST_R + 16 * u) * n + row] : 0.0;
#pragma unroll
        for (int u = 0; u < CH_H * CH_H / 256; ++u) (&Ls[0][0])[threadIdx.x + 256 * u] = v[u];
#pragma unroll
        for (int u = 0; u < CH_H * ST_R / 256; ++u) Ps[threadIdx.x / ST_R + 16 * u][r] = p[u];
    }
    __syncthreads();
    double s[4] = {0, 0, 0, 0};
#pragma unroll 8
    for (int l = 0; l < CH_H; ++l) {
        const double p = Ps[l][r];
#pragma unroll
        for (int c = 0; c < 4; ++c) s[c] = fma(p, Ls[l][c0 + c], s[c]);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int col = c0 + c;
        if (col < kb2 && row < n && row >= k0 + CH_H + col) G[(int64_t)(k0 + CH_H + col) * n + row] -= s[c];
    }
}

// ---------------------------------------------------------------- triangular solves
// T(i, j) = M[i*si + j*sj].  One CTA solves the whole system when n fits its shared
// memory: blocks of 32 in solve order, warp 0 substitutes within the block with
// shuffles, then every warp updates the remaining right-hand sides.
constexpr int TS_THREADS = 1024, TS_CHAIN = 128;
__device__ __forceinline__ double tget(const double* M, int64_t si, int64_t sj, int64_t i, int64_t j) {
    return M[i * si + j * sj];
}

// The bl x bl diagonal block at b0 (bl <= 32), staged by every thread of the CTA into
// tb (32 x 33) so that warp 0's substitution below reads shared memory only.
__device__ void trsv_stage_block(const double* M, int64_t si, int64_t sj, int b0, int bl, double (*tb)[33]) {
    for (int t = threadIdx.x; t < 32 * 32; t += blockDim.x) {
        const int i = si == 1 ? t % 32 : t / 32, j = si == 1 ? t / 32 : t % 32;   // contiguous index fastest
        tb[i][j] = (i < bl && j < bl) ? tget(M, si, sj, b0 + i, b0 + j) : 0.0;
    }
}

__device__ void trsv_block_warp(const double (*tb)[33], int b0, int bl, bool lower, double* xs, int lane) {
    double v = lane < bl ? xs[b0 + lane] : 0.0;
    if (lower) {
        for (int k = 0; k < bl; ++k) {
            if (lane == k) v = v / tb[k][k];
            const double xk = __shfl_sync(0xffffffffu, v, k);
            if (lane > k && lane < bl) v = fma(-tb[lane][k], xk, v);
        }
    } else {
        for (int k = bl - 1; k >= 0; --k) {
            if (lane == k) v = v / tb[k][k];
            const double xk = __shfl_sync(0xffffffffu, v, k);
            if (lane < k) v = fma(-tb[lane][k], xk, v);
        }
    }
    if (lane < bl) xs[b0 + lane] = v;
}

// rows [r0, r1) of xs -= T(rows, b0 .. b0+bl) * xs[b0 .. b0+bl)
__device__ void trsv_update_cta(const double* M, int64_t si, int64_t sj, int b0, int bl, int r0, int r1, double* xs) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (sj == 1) {   // rows contiguous along j: a warp per row
        for (int i = r0 + warp; i < r1; i += nw) {
            double p = 0.0;
            for (int c = lane; c < bl; c += 32) p = fma(M[(int64_t)i * si + b0 + c], xs[b0 + c], p);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
            if (lane == 0) xs[i] -= p;
        }
    } else {         // columns contiguous along i (or general): a thread per row
        for (int i = r0 + (int)threadIdx.x; i < r1; i += blockDim.x) {
            double p = 0.0;
#pragma unroll 8   // eight independent loads in flight per thread
            for (int c = 0; c < bl; ++c) p = fma(tget(M, si, sj, i, b0 + c), xs[b0 + c], p);
            xs[i] -= p;
        }
    }
}

__global__ void __launch_bounds__(TS_THREADS) k_trsv_small(const double* __restrict__ M, int64_t si, int64_t sj,
                                                           int n, int lower, double* __restrict__ x) {
    extern __shared__ double xs[];
    __shared__ double tb[32][33];
    for (int i = threadIdx.x; i < n; i += blockDim.x) xs[i] = x[i];
    const int nb = (n + 31) / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int bb = 0; bb < nb; ++bb) {
        const int b = lower ? bb : nb - 1 - bb;
        const int b0 = b * 32, bl = min(32, n - b0);
        trsv_stage_block(M, si, sj, b0, bl, tb);
        __syncthreads();
        if (warp == 0) trsv_block_warp(tb, b0, bl, lower != 0, xs, lane);
        __syncthreads();
        if (lower) trsv_update_cta(M, si, sj, b0, bl, b0 + bl, n, xs);
        else trsv_update_cta(M, si, sj, b0, bl, 0, b0, xs);
        __syncthreads();
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) x[i] = xs[i];
}

// Large systems: one cooperative launch, the CTAs' row blocks of 64 in solve order (block b,
// b + grid, ...).  A CTA subtracts the blocks of x before its own as they are published
// (flag[j] != 0 once block j of x is in place), the next 64 x 64 tile of T on its way
// meanwhile, then solves its diagonal tile and publishes.  A wait that runs out leaves NaN in
// x.  A launch per 128 rows and one per update took 100 us a block: a factor's two solves
// at n = 5,000 7.6 -> 1.9 ms, at n = 24,000 40 -> 9.0 ms.  Below TS_CHAIN one CTA is as fast
// (n = 130: two solves 98 us by the chain; n = 1,000, one CTA -> chain 1,990 -> 410 us).
constexpr int TC_B = 64, TC_THREADS = 256;
__global__ void __launch_bounds__(TC_THREADS) k_trsv_chain(const double* __restrict__ M, int64_t si, int64_t sj, int n,
                                                           int lower, double* __restrict__ x, int* __restrict__ flag) {
    __shared__ double tile[TC_B][TC_B + 1];
    __shared__ double xs[TC_B], red[4][TC_B], rd[TC_B];
    __shared__ int ok;
    const int tid = threadIdx.x;
    const int nb = (n + TC_B - 1) / TC_B;
    const bool along_i = si == 1;   // T(i, j) contiguous along i, else along j
    double pre[TC_B * TC_B / TC_THREADS];
    auto fetch = [&](int bi, int bj) {   // tile of row block bi, column block bj into registers
#pragma unroll
        for (int u = 0; u < TC_B * TC_B / TC_THREADS; ++u) {
            const int t = tid + u * TC_THREADS, p = t % TC_B, q = t / TC_B;
            const int i = bi * TC_B + (along_i ? p : q), j = bj * TC_B + (along_i ? q : p);
            const bool in = i < n && j < n && (bi != bj || (lower ? j <= i : j >= i));
            pre[u] = in ? tget(M, si, sj, i, j) : (i == j ? 1.0 : 0.0);
        }
    };
    auto stage = [&]() {
#pragma unroll
        for (int u = 0; u < TC_B * TC_B / TC_THREADS; ++u) {
            const int t = tid + u * TC_THREADS, p = t % TC_B, q = t / TC_B;
            if (along_i) tile[p][q] = pre[u]; else tile[q][p] = pre[u];
        }
    };
    for (int o = blockIdx.x; o < nb; o += gridDim.x) {
        const int b = lower ? o : nb - 1 - o;
        const int row = tid % TC_B, part = tid / TC_B;
        double s = 0.0;
        fetch(b, o == 0 ? b : (lower ? 0 : nb - 1));
        for (int w = 0; w < o; ++w) {
            const int j = lower ? w : nb - 1 - w;
            __syncthreads();
            stage();
            fetch(b, w + 1 < o ? (lower ? w + 1 : nb - 2 - w) : b);
            if (tid == 0) {
                int v = 0;
                for (int it = 0; it < (1 << 24); ++it) {
                    asm volatile("ld.acquire.gpu.s32 %0, [%1];" : "=r"(v) : "l"(flag + j) : "memory");
                    if (v) break;
                }
                ok = v == 1;
            }
            __syncthreads();
            if (!ok) break;
            if (tid < TC_B) xs[tid] = j * TC_B + tid < n ? __ldcg(x + j * TC_B + tid) : 0.0;
            __syncthreads();
#pragma unroll
            for (int c = 0; c < TC_B / 4; ++c) s = fma(tile[row][part * (TC_B / 4) + c], xs[part * (TC_B / 4) + c], s);
        }
        const bool good = o == 0 || ok;
        __syncthreads();
        stage();
        red[part][row] = s;
        __syncthreads();
        if (tid < TC_B) {
            rd[tid] = 1.0 / tile[tid][tid];
            xs[tid] = (b * TC_B + tid < n ? x[b * TC_B + tid] : 0.0) - ((red[0][tid] + red[1][tid]) + (red[2][tid] + red[3][tid]));
        }
        __syncthreads();
        if (tid < 32) {   // two halves of 32, one row per lane, then the other half's rows
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                const int r0 = (lower ? h : 1 - h) * 32, r1 = 32 - r0;
                double v = xs[r0 + tid];
                for (int q = 0; q < 32; ++q) {
                    const int c = lower ? q : 31 - q;
                    if (tid == c) v *= rd[r0 + c];
                    const double xc = __shfl_sync(0xffffffffu, v, c);
                    if (lower ? tid > c : tid < c) v = fma(-tile[r0 + tid][r0 + c], xc, v);
                }
                xs[r0 + tid] = v;
                __syncwarp();
                if (h == 0) {
                    double u0 = 0.0, u1 = 0.0;
#pragma unroll
                    for (int c = 0; c < 32; c += 2) {
                        u0 = fma(tile[r1 + tid][r0 + c], xs[r0 + c], u0);
                        u1 = fma(tile[r1 + tid][r0 + c + 1], xs[r0 + c + 1], u1);
                    }
                    xs[r1 + tid] -= u0 + u1;
                    __syncwarp();
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = b * TC_B + 32 * h + tid;
                if (i < n) x[i] = good ? xs[32 * h + tid] : nan("");
            }
            __threadfence();
            __syncwarp();
            if (tid == 0) asm volatile("st.release.gpu.s32 [%0], %1;" ::"l"(flag + b), "r"(good ? 1 : 2) : "memory");
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------- matrix-vector
__global__ void __launch_bounds__(256) k_gemv_rows(const double* __restrict__ A, int64_t lda, int64_t nrows, int ncols,
                                                   const double* __restrict__ v, const double* __restrict__ b,
                                                   const double* __restrict__ w, double* __restrict__ t) {
    const int lane = threadIdx.x & 31;
    const int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (r >= nrows) return;
    const double* row = A + r * lda;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int c = lane;
    for (; c + 96 < ncols; c += 128) {
        s0 = fma(row[c], v[c], s0);
        s1 = fma(row[c + 32], v[c + 32], s1);
        s2 = fma(row[c + 64], v[c + 64], s2);
        s3 = fma(row[c + 96], v[c + 96], s3);
    }
    for (; c < ncols; c += 32) s0 = fma(row[c], v[c], s0);
    double s = (s0 + s1) + (s2 + s3);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
        if (b) s = b[r] - s;
        if (w) s *= w[r] * w[r];
        t[r] = s;
    }
}

// partial[y][c] = sum over the rows of slice y of A[r][c] t[r]; a block walks its
// slice's rows with its threads across the columns (four columns per thread, four
// rows per step, whole rows read contiguously).
constexpr int ATB_SLICES = 1024, ATB_THREADS = 256;
__global__ void __launch_bounds__(ATB_THREADS) k_atb_partial(const double* __restrict__ A, int64_t lda, int64_t nr,
                                                             int ncols, const double* __restrict__ b,
                                                             double* __restrict__ partial) {
    const int64_t per = (nr + gridDim.y - 1) / gridDim.y;
    const int64_t r0 = (int64_t)blockIdx.y * per, r1 = min(nr, r0 + per);
    for (int c0 = 0; c0 < ncols; c0 += 4 * ATB_THREADS) {
        double s[4] = {0, 0, 0, 0};
        int cc[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) cc[u] = c0 + u * ATB_THREADS + threadIdx.x;
        int64_t r = r0;
        for (; r + 4 <= r1; r += 4) {   // 16 loads in flight per thread
            double v[4][4];
            double br[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                br[q] = b[r + q];
                const double* row = A + (r + q) * lda;
#pragma unroll
                for (int u = 0; u < 4; ++u) v[q][u] = cc[u] < ncols ? row[cc[u]] : 0.0;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int u = 0; u < 4; ++u) s[u] = fma(v[q][u], br[q], s[u]);
        }
        for (; r < r1; ++r) {
            const double br = b[r];
            const double* row = A + r * lda;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (cc[u] < ncols) s[u] = fma(row[cc[u]], br, s[u]);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (cc[u] < ncols) partial[(int64_t)blockIdx.y * ncols + cc[u]] = s[u];
    }
}
// h[c] += the partials of column c in slice order: eight warps each add a contiguous
// eighth of the slices for 32 columns, then the eighths are added in order.  (One thread
// per column walked all 1,024 slices of a tall block, 80 us of dependent loads.)
__global__ void __launch_bounds__(256) k_atb_reduce(const double* __restrict__ partial, int nslices, int ncols,
                                                    double* __restrict__ h) {
    __shared__ double red[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = blockIdx.x * 32 + lane;
    const int per = (nslices + 7) / 8, y0 = min(nslices, warp * per), y1 = min(nslices, y0 + per);
    double s = 0.0;
    if (c < ncols) {
        int y = y0;
        for (; y + 8 <= y1; y += 8) {   // eight loads in flight
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = partial[(int64_t)(y + u) * ncols + c];
#pragma unroll
            for (int u = 0; u < 8; ++u) s += v[u];
        }
        for (; y < y1; ++y) s += partial[(int64_t)y * ncols + c];
    }
    red[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && c < ncols) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += red[w][lane];
        h[c] += t;
    }
}

// ---------------------------------------------------------------- vectors
__global__ void __launch_bounds__(1024) k_dot(const double* __restrict__ x, const double* __restrict__ y, int n,
                                              double* __restrict__ out) {
    __shared__ double red[32];
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s = fma(x[i], y[i], s);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        s = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) *out = s;
    }
}
__global__ void k_axpby(int n, double a, const double* __restrict__ x, double b, double* __restrict__ y) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = a * x[i] + b * y[i];
}
__global__ void k_add_diag(double* G, int n, double v) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) G[(int64_t)i * n + i] += v;
}

// ---------------------------------------------------------------- FP64 FMA rate
// CH independent FMA chains per thread (enough in flight to cover the FP64 pipe's
// latency at the occupancy the launch gets); the result is stored so that the
// chains are not removed.
template <int CH>
__global__ void __launch_bounds__(256) k_fp64_fma(double* out, int iters, double seed) {
    double x[CH];
#pragma unroll
    for (int k = 0; k < CH; ++k) x[k] = seed + 1e-9 * (threadIdx.x + 37 * k);
    const double mul = 0.9999999999, add = 1e-12;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < CH; ++k) x[k] = fma(x[k], mul, add);
    }
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < CH; ++k) s += x[k];
    out[(int64_t)blockIdx.x * blockDim.x + threadIdx.x] = s;
}

}  // namespace cgd

namespace cg {

static void ckd(cudaError_t e, const char* w) {
    if (e != cudaSuccess) throw std::runtime_error(std::string("CUDA error in ") + w + ": " + cudaGetErrorString(e));
}

static int sm_count() {
    static thread_local int dev_cached = -1, cached = 0;
    int dev = 0;
    ckd(cudaGetDevice(&dev), "cudaGetDevice");
    if (dev != dev_cached) {
        ckd(cudaDeviceGetAttribute(&cached, cudaDevAttrMultiProcessorCount, dev), "SM count");
        cached = std::max(1, cached);
        dev_cached = dev;
    }
    return cached;
}

void syrk_tn(const double* X, int64_t ldx, int64_t K, int m, double alpha, double* C, int64_t ldc, cudaStream_t st) {
    if (K <= 0 || m <= 0) return;
    const int ntile = (m + cgd::SY_T - 1) / cgd::SY_T;
    const int64_t npairs = (int64_t)ntile * (ntile + 1) / 2;
    const int64_t target = (int64_t)sm_count() * 6;   // about six resident CTAs per SM
    const int64_t kchunks = (K + cgd::SY_KC - 1) / cgd::SY_KC;
    int64_t nslice = npairs >= target ? 1 : std::min<int64_t>(kchunks, (target + npairs - 1) / npairs);
    const int64_t kslice = (kchunks + nslice - 1) / nslice * cgd::SY_KC;
    nslice = (K + kslice - 1) / kslice;
    if (npairs > 0x7fffffffLL) throw std::runtime_error("syrk_tn: matrix too large");
    const dim3 grid((unsigned)npairs, (unsigned)nslice);
    if (nslice > 1)
        cgd::k_syrk_tn<true><<<grid, cgd::SY_THREADS, 0, st>>>(X, ldx, K, m, alpha, C, ldc, ntile, kslice);
    else
        cgd::k_syrk_tn<false><<<grid, cgd::SY_THREADS, 0, st>>>(X, ldx, K, m, alpha, C, ldc, ntile, kslice);
    ckd(cudaGetLastError(), "k_syrk_tn");
}

void gram64(const double* X, int64_t ldx, int64_t K, int m, double* C, int64_t ldc, cudaStream_t st) {
    if (K <= 0 || m <= 0) return;
    // Below, the exponent pass and the 512-thread CTAs' start cost what the FP64 products do.
    // Whole calls, FP64 -> digits: 300 x 400 119 -> 79 us, 1,000 x 200 141 -> 91 us; with entries over
    // many powers of two, some outputs summed twice, 117 -> 91 to 121 and 141 -> 118 to 159 us;
    // 1,000 x 100 90 -> 78 and 87 -> 89 to 108 us
    if ((double)K * m * m < 4.0e7) {
        syrk_tn(X, ldx, K, m, 1.0, C, ldc, st);
        return;
    }
    const int ntile = (m + cgd::GD_T - 1) / cgd::GD_T;
    const int64_t npairs = (int64_t)ntile * (ntile + 1) / 2;
    if (npairs > 0x7fffffffLL) throw std::runtime_error("gram64: matrix too large");
    // K slices (FP64 atomics) where the triangle alone leaves SMs idle: the fewest 32-row
    // blocks on the longest CTA's path, two more per slice for its start and end
    const int64_t sms = sm_count(), blocks = (K + cgd::GD_BLOCK - 1) / cgd::GD_BLOCK;
    int64_t nslice = 1, best = -1;
    for (int64_t sl = 1; sl <= std::min<int64_t>(blocks, std::max<int64_t>(1, 8 * sms / npairs)); ++sl) {
        const int64_t cost = (npairs * sl + sms - 1) / sms * ((blocks + sl - 1) / sl + 2);
        if (best < 0 || cost < best) { best = cost; nslice = sl; }
    }
    const int64_t kslice = (blocks + nslice - 1) / nslice * cgd::GD_BLOCK;
    nslice = (K + kslice - 1) / kslice;
    int* ex = scratch_alloc<int>(m, st);
    int16_t* eb = scratch_alloc<int16_t>((size_t)blocks * m, st);   // 1/128 of X
    ckd(cudaMemsetAsync(ex, 0x80, sizeof(int) * m, st), "column exponents");   // a very small value
    const unsigned strips = (unsigned)((m + 31) / 32);
    const unsigned gy = (unsigned)std::max<int64_t>(1, std::min<int64_t>((blocks + 7) / 8, 8 * sms / strips));
    cgd::k_col_exponents<<<dim3(strips, gy), 256, 0, st>>>(X, ldx, K, m, ex, eb);
    const size_t smem = cgd::GdSmem::total;
    const dim3 grid((unsigned)npairs, (unsigned)nslice);
    if (nslice > 1) {
        ckd(cudaFuncSetAttribute(cgd::k_syrk_digits<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "smem");
        cgd::k_syrk_digits<true><<<grid, cgd::GD_THREADS, smem, st>>>(X, ldx, K, m, C, ldc, ntile, kslice, ex, eb);
    } else {
        ckd(cudaFuncSetAttribute(cgd::k_syrk_digits<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "smem");
        cgd::k_syrk_digits<false><<<grid, cgd::GD_THREADS, smem, st>>>(X, ldx, K, m, C, ldc, ntile, kslice, ex, eb);
    }
    ckd(cudaGetLastError(), "k_syrk_digits");
    ckd(cudaFreeAsync(eb, st), "column exponents");
    ckd(cudaFreeAsync(ex, st), "column exponents");
}

bool cholesky64(double* G, int n, int* d_info, cudaStream_t st, bool tensor_updates, bool tiny, bool* tiny_pivot) {
    ckd(cudaMemsetAsync(d_info, 0, sizeof(int), st), "info");
    // trailing updates of full 128-wide panels by exact BF16 digit products on the
    // tensor cores (syrk_update_ozaki); the FP64 SYRK otherwise
    void* oz = nullptr;
    const bool use_oz = tensor_updates && cgd::CH_NB == 128 && n > cgd::CH_NB;
    if (use_oz) {
        oz = scratch_alloc<unsigned char>(ozaki_scratch_bytes(n), st);
        ckd(cudaMemsetAsync(oz, 0, sizeof(int), st), "Ozaki error word");
    }
    int* status = scratch_alloc<int>(2, st);
    ckd(cudaMemsetAsync(status, 0, 2 * sizeof(int), st), "panel status");
    const int sms = sm_count();
    const size_t most = 200 * 1024;
    const auto panel = tiny ? cgd::k_chol_half<true> : cgd::k_chol_half<false>;
    ckd(cudaFuncSetAttribute(panel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most), "panel smem");
    const int rmax = (int)(most / (cgd::CH_LD * sizeof(double))) - cgd::CH_H;
    auto half = [&](int k, int kb, int second) {
        const int m = n - k - kb;
        const int R = std::max(8, std::min(rmax, (m + sms - 1) / sms));   // one share of the rows per SM
        const int grid = std::max(1, (m + R - 1) / R);
        panel<<<grid, cgd::CH_THREADS, (size_t)(cgd::CH_H + R) * cgd::CH_LD * sizeof(double), st>>>(G, n, k, kb, m, R, second,
                                                                                                    d_info, status);
    };
    for (int k = 0; k < n; k += cgd::CH_NB) {
        const int kb = std::min(cgd::CH_NB, n - k), k1 = std::min(cgd::CH_H, kb), k2 = kb - k1;
        half(k, k1, 0);
        if (k2 > 0) {
            cgd::k_chol_strip<<<(n - k - k1 + cgd::ST_R - 1) / cgd::ST_R, 256, 0, st>>>(G, n, k, k2);
            half(k + k1, k2, 1);
        }
        const int m = n - k - kb;
        if (m > 0) {   // trailing update: A22 -= P P^T (P: rows k+kb.., columns k..k+kb, column-major)
            const double* P = G + (int64_t)k * n + (k + kb);
            double* C = G + (int64_t)(k + kb) * n + (k + kb);
            if (use_oz && kb == 128) syrk_update_ozaki(P, n, kb, m, -1.0, C, n, oz, st);
            else syrk_tn(P, n, kb, m, -1.0, C, n, st);
        }
        ckd(cudaGetLastError(), "cholesky step");
    }
    int info = 0, oz_err = 0, small = 0;
    ckd(cudaMemcpyAsync(&info, d_info, sizeof(int), cudaMemcpyDeviceToHost, st), "info");
    if (use_oz) {
        ckd(cudaMemcpyAsync(&oz_err, oz, sizeof(int), cudaMemcpyDeviceToHost, st), "Ozaki error word");
        ckd(cudaFreeAsync(oz, st), "Ozaki scratch");
    }
    ckd(cudaStreamSynchronize(st), "cholesky");
    if (info != 0 && tiny_pivot) ckd(cudaMemcpyAsync(&small, status + 1, sizeof(int), cudaMemcpyDeviceToHost, st), "panel status");
    ckd(cudaFreeAsync(status, st), "panel status");
    if (info != 0) ckd(cudaStreamSynchronize(st), "panel status");
    if (tiny_pivot) *tiny_pivot = small != 0;
    if (oz_err) throw std::runtime_error("Cholesky trailing update timed out on its pipeline (code " +
                                         std::to_string(oz_err) + ")");
    return info == 0;
}

void trsv64(const double* M, int64_t si, int64_t sj, int n, bool lower, double* x, cudaStream_t st) {
    if (n <= 0) return;
    if (n <= cgd::TS_CHAIN) {
        const size_t smem = (size_t)n * sizeof(double);
        ckd(cudaFuncSetAttribute(cgd::k_trsv_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(cgd::TS_CHAIN * sizeof(double))),
            "trsv smem");
        cgd::k_trsv_small<<<1, cgd::TS_THREADS, smem, st>>>(M, si, sj, n, lower ? 1 : 0, x);
        ckd(cudaGetLastError(), "k_trsv_small");
        return;
    }
    const int nb = (n + cgd::TC_B - 1) / cgd::TC_B;
    int* flag = scratch_alloc<int>(nb, st);
    ckd(cudaMemsetAsync(flag, 0, sizeof(int) * nb, st), "trsv flags");
    int lo = lower ? 1 : 0;
    void* args[] = {(void*)&M, (void*)&si, (void*)&sj, (void*)&n, (void*)&lo, (void*)&x, (void*)&flag};
    ckd(cudaLaunchCooperativeKernel((const void*)cgd::k_trsv_chain, dim3((unsigned)std::min(nb, sm_count())),
                                    dim3(cgd::TC_THREADS), args, 0, st),
        "k_trsv_chain");
    ckd(cudaFreeAsync(flag, st), "trsv flags");
}

void cholesky_solve64(const double* L, int n, const double* h, double* x, cudaStream_t st) {
    if (x != h) ckd(cudaMemcpyAsync(x, h, sizeof(double) * n, cudaMemcpyDeviceToDevice, st), "x = h");
    trsv64(L, 1, n, n, true, x, st);    // L y = h:   L(i, j) = L[i + j n]
    trsv64(L, n, 1, n, false, x, st);   // L^T x = y: L^T(i, j) = L[j + i n]
}

void gemv_rows64(const double* A, int64_t lda, int64_t nrows, int ncols, const double* v, const double* b,
                 const double* w, double* t, cudaStream_t st) {
    if (nrows <= 0) return;
    cgd::k_gemv_rows<<<(unsigned)((nrows + 7) / 8), 256, 0, st>>>(A, lda, nrows, ncols, v, b, w, t);
    ckd(cudaGetLastError(), "k_gemv_rows");
}

int64_t atb_partial_doubles(int64_t nrows, int ncols) {
    return std::max<int64_t>(1, std::min<int64_t>(nrows, cgd::ATB_SLICES)) * ncols;
}

void gemv_cols64(const double* A, int64_t lda, int64_t nrows, int ncols, const double* t, double* g, double* partial,
                 cudaStream_t st) {
    if (nrows <= 0) return;
    const int ns = (int)std::min<int64_t>(nrows, cgd::ATB_SLICES);
    cgd::k_atb_partial<<<dim3(1, ns), cgd::ATB_THREADS, 0, st>>>(A, lda, nrows, ncols, t, partial);
    cgd::k_atb_reduce<<<(ncols + 31) / 32, 256, 0, st>>>(partial, ns, ncols, g);
    ckd(cudaGetLastError(), "k_atb");
}

void dot64(const double* x, const double* y, int n, double* out, cudaStream_t st) {
    cgd::k_dot<<<1, 1024, 0, st>>>(x, y, n, out);
    ckd(cudaGetLastError(), "k_dot");
}

void axpby64(int n, double a, const double* x, double b, double* y, cudaStream_t st) {
    if (n <= 0) return;
    cgd::k_axpby<<<(n + 255) / 256, 256, 0, st>>>(n, a, x, b, y);
    ckd(cudaGetLastError(), "k_axpby");
}

void add_diag64(double* G, int n, double v, cudaStream_t st) {
    if (n <= 0 || v == 0.0) return;
    cgd::k_add_diag<<<(n + 255) / 256, 256, 0, st>>>(G, n, v);
    ckd(cudaGetLastError(), "k_add_diag");
}

double fp64_fma_tflops(cudaStream_t st) {
    // the best of a few chain counts and occupancies; flops = 2 per FMA
    const int threads = 256, iters = 1 << 13;
    const int sms = sm_count();
    double* out = nullptr;
    out = scratch_alloc<double>((size_t)sms * 8 * threads, st);
    cudaEvent_t e0, e1;
    ckd(cudaEventCreate(&e0), "event");
    ckd(cudaEventCreate(&e1), "event");
    double best = 0.0;
    auto run = [&](auto kernel, int chains, int blocks_per_sm) {
        const int blocks = sms * blocks_per_sm;
        kernel<<<blocks, threads, 0, st>>>(out, iters, 1.0);   // warm-up (clocks settle)
        for (int rep = 0; rep < 3; ++rep) {
            ckd(cudaEventRecord(e0, st), "record");
            kernel<<<blocks, threads, 0, st>>>(out, iters, 1.0 + rep);
            ckd(cudaEventRecord(e1, st), "record");
            ckd(cudaEventSynchronize(e1), "sync");
            float ms = 0.f;
            ckd(cudaEventElapsedTime(&ms, e0, e1), "elapsed");
            best = std::max(best, 2.0 * chains * iters * (double)blocks * threads / (ms * 1e-3) / 1e12);
        }
        ckd(cudaGetLastError(), "k_fp64_fma");
    };
    run(cgd::k_fp64_fma<8>, 8, 8);
    run(cgd::k_fp64_fma<16>, 16, 4);
    run(cgd::k_fp64_fma<32>, 32, 4);
    run(cgd::k_fp64_fma<32>, 32, 2);
    ckd(cudaFreeAsync(out, st), "peak scratch free");
    {   // and the register-blocked SYRK of this file on a 2048 x 4096 operand (FMA bound)
        const int K = 2048, m = 4096;
        double *X = nullptr, *C = nullptr;
        X = scratch_alloc<double>((size_t)K * m, st);
        C = scratch_alloc<double>((size_t)m * m, st);
        ckd(cudaMemsetAsync(X, 0, sizeof(double) * K * m, st), "peak scratch");   // finite operands
        ckd(cudaMemsetAsync(C, 0, sizeof(double) * m * m, st), "peak scratch");
        syrk_tn(X, m, K, m, 1.0, C, m, st);   // warm-up
        for (int rep = 0; rep < 3; ++rep) {
            ckd(cudaEventRecord(e0, st), "record");
            syrk_tn(X, m, K, m, 1.0, C, m, st);
            ckd(cudaEventRecord(e1, st), "record");
            ckd(cudaEventSynchronize(e1), "sync");
            float ms = 0.f;
            ckd(cudaEventElapsedTime(&ms, e0, e1), "elapsed");
            best = std::max(best, (double)K * m * (m + 1.0) / (ms * 1e-3) / 1e12);
        }
        ckd(cudaFreeAsync(X, st), "peak scratch free");
        ckd(cudaFreeAsync(C, st), "peak scratch free");
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    ckd(cudaStreamSynchronize(st), "sync");
    return best;
}

}  // namespace cg
