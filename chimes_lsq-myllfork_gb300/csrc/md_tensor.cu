// FP64 triplet / quadruplet forces with the coefficient contraction on the tensor cores.
//
// Reference: Cheby::Force_3B / Force_4B (src/Cheby.C:2024-2675); md.cu's formulation.  A
// cluster type's dense coefficients, split at the slots (0 1 2 | 3 4 5) or (0 1 | 2), are a
// matrix C[p_I][p_O].  With U and Q the products of a cluster's u_s[k] = f_s T_k(r_s) over
// the two halves,
//     Y[p_O] = sum C[p_I][p_O] U[p_I],   W[p_I] = sum C[p_I][p_O] Q[p_O],
// dE/du_s comes from W and the other slots of s's half (s in I) or from Y (s in O), E from
// either.  Y and W of the clusters of a type are two matrix products, formed exactly from
// base-256 digits on mma.sync (digits.cuh; the digits of C are tabulated when the
// coefficients are set), so the FP64 pipe is left with the bases and the halves: about
// 1,400 of the 11,000 operations per quadruplet.  One thread per cluster walked the whole
// tensor before: 1,000 C/H/N/O atoms, quadruplets 907 -> 222 us, triplets 285 -> 179 us;
// 64 atoms 500 -> 59 us and 93 -> 36 us (whole force calls took 1.38 and 1.34 ms with that
// form and take 0.66 and 0.60 now, lists and allocation included).  What remains is the FP64 pipe's: the bases, one exp and about 150 operations
// per edge.
#include <algorithm>

#include "digits.cuh"
#include "md.h"
#include "md_dev.cuh"

namespace cgd {

namespace {

template <int NBODY> struct Mt;
// K and columns of Y = U C (K = p_I) and W = Q C^T (K = p_O)
template <> struct Mt<3> { static constexpr int O = 8, NP = 3, NI = 64, NO = 8; };
template <> struct Mt<4> { static constexpr int O = 4, NP = 6, NI = 64, NO = 64; };
constexpr int MT_THREADS = 512;
constexpr int MT_OUT = 65;         // staged outputs per cluster row (doubles)

// bytes of one digit table: K / 8 blocks of `cols` rows
__host__ __device__ constexpr size_t mt_table(int K, int cols) { return (size_t)(K / 8) * cols * DIG_STRIDE; }

// One CTA per cluster type: the digits of C as the columns of Y, then of W, and the
// exponents of their columns (Y's NO, then W's NI; LG_BAD for infinities and NaN).
template <int NBODY>
__global__ void k_md_digit_tables(const double* __restrict__ C, unsigned char* __restrict__ tab, int* __restrict__ ex) {
    using T = Mt<NBODY>;
    const double* c = C + (size_t)blockIdx.x * T::NI * T::NO;
    unsigned char* t = tab + (size_t)blockIdx.x * (mt_table(T::NI, T::NO) + mt_table(T::NO, T::NI));
    int* e = ex + (size_t)blockIdx.x * (T::NO + T::NI);
    __shared__ int se[T::NO + T::NI];
    for (int n = threadIdx.x; n < T::NO + T::NI; n += blockDim.x) {
        const bool w = n >= T::NO;
        int lg = -16384;
        for (int k = 0; k < (w ? T::NO : T::NI); ++k) lg = max(lg, lg_up(w ? c[(n - T::NO) * T::NO + k] : c[k * T::NO + n]));
        se[n] = e[n] = lg == LG_BAD ? LG_BAD : pow2_above(lg);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < T::NI * T::NO; i += blockDim.x) {   // pairs along K
        const bool w = i >= T::NI * T::NO / 2;
        const int j = w ? i - T::NI * T::NO / 2 : i, K = w ? T::NO : T::NI, cols = w ? T::NI : T::NO;
        const int n = j / (K / 2), k = 2 * (j % (K / 2));
        const double x0 = w ? c[n * T::NO + k] : c[k * T::NO + n], x1 = w ? c[n * T::NO + k + 1] : c[(k + 1) * T::NO + n];
        const int en = se[w ? T::NO + n : n];
        unsigned char* row = t + (w ? mt_table(T::NI, T::NO) : 0) + ((size_t)(k >> 3) * cols + n) * DIG_STRIDE + 2 * (k & 7);
        put_digits(row, en == LG_BAD ? 0 : to_fixed(x0, DIG_FIX - en), en == LG_BAD ? 0 : to_fixed(x1, DIG_FIX - en));
    }
}

template <int NBODY>
struct MtSmem {
    using T = Mt<NBODY>;
    // digits of U then Q, digits of C then C^T; both reused by the outputs
    static constexpr size_t a = 0;
    static constexpr size_t a_bytes = mt_table(T::NI, MDC_TILE);
    static constexpr size_t b = a + a_bytes;
    static constexpr size_t b_bytes = mt_table(T::NI, T::NO) > mt_table(T::NO, T::NI) ? mt_table(T::NI, T::NO) : mt_table(T::NO, T::NI);
    static constexpr size_t out = (size_t)MDC_TILE * MT_OUT * 8;
    static constexpr size_t two_out = 2 * out;
    static constexpr size_t u = a + (a_bytes + b_bytes > two_out ? a_bytes + b_bytes : two_out);
    static constexpr size_t h = u + (size_t)MDC_TILE * T::NP * T::O * 8;
    static constexpr size_t r = h + (size_t)MDC_TILE * T::NP * T::O * 8;      // r_ab, r; then the edge force
    static constexpr size_t m = r + (size_t)MDC_TILE * T::NP * 4 * 8;
    static constexpr size_t lg = m + (size_t)MDC_TILE * 16;
    static constexpr size_t ab = lg + (size_t)MDC_TILE * T::NP * 4;
    static constexpr size_t total = ab + (size_t)MDC_TILE * T::NP * 4;
};

__device__ __forceinline__ void cp16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src));
}

template <int NBODY>
__global__ void __launch_bounds__(MT_THREADS, 1)
k_mdt(ModelDev M, FramesDev F, ClusterSet CS, MdBuckets MB, const unsigned char* __restrict__ tab,
      const int* __restrict__ cex, double* Fo, double* So) {
    using T = Mt<NBODY>;
    using S = MtSmem<NBODY>;
    constexpr int NP = T::NP, O = T::O;
    extern __shared__ __align__(16) unsigned char smem[];
    int key;
    int64_t cb, t1;
    if (!tile_lookup(MB, blockIdx.x, key, cb, t1)) return;
    const int f = key / MB.ntypes, type = key % MB.ntypes;
    const int nb = (int)min((int64_t)MDC_TILE, t1 - cb);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned char* tabT = tab + (size_t)type * (mt_table(T::NI, T::NO) + mt_table(T::NO, T::NI));
    const int* exT = cex + (size_t)type * (T::NO + T::NI);
    const uint32_t sm = smem_addr(smem);
    auto fetch = [&](size_t ofs, size_t bytes) {
        for (int i = tid; i < (int)(bytes / 16); i += MT_THREADS) cp16(sm + (uint32_t)S::b + 16 * i, tabT + ofs + 16 * i);
        asm volatile("cp.async.commit_group;");
    };
    fetch(0, mt_table(T::NI, T::NO));
    double* sU = reinterpret_cast<double*>(smem + S::u);
    double* sH = reinterpret_cast<double*>(smem + S::h);
    double* sR = reinterpret_cast<double*>(smem + S::r);
    int4* sM = reinterpret_cast<int4*>(smem + S::m);
    int* sLg = reinterpret_cast<int*>(smem + S::lg);
    int* sAB = reinterpret_cast<int*>(smem + S::ab);
    __shared__ double red[8][MT_THREADS / 32];
    const int N = F.natoms[f];
    const int64_t aofs = F.atom_ofs[f], gb = F.ghost_ofs[f];
    const int* typ = F.type + aofs;
    const BoxDev& B = F.box[f];
    const ClusterTypeDev& CT = (NBODY == 3 ? M.types3 : M.types4)[type];
    if (tid < nb) sM[tid] = CS.m[MB.val[cb + tid]];
    __syncthreads();
    // ---- bases, one (cluster, edge) per thread
    for (int t = tid; t < nb * NP; t += MT_THREADS) {
        const int c = t / NP, e = t - c * NP;
        const int4 mm = sM[c];
        int id = 0, w = 1;
#pragma unroll
        for (int u = 0; u < NBODY; ++u) { id += w * (typ[member(mm, u) % N] + 1); w *= 10; }
        const int s = (NBODY == 3 ? M.pidx3 : M.pidx4)[id * NP + e];
        int a, b;
        edge_ab(NBODY, e, a, b);
        const int ga = member(mm, a), gbm = member(mm, b);
        double R3[3], fc, fd, u[O], h[O];
        const double r = dist_exact(B.h, F.scaled + 3 * (gb + ga), F.scaled + 3 * (gb + gbm), R3);
        const int pt = M.int_pair_map[typ[ga % N] * M.natmtyp + typ[gbm % N]];
        fcut_eval(M, r, CT.smax[s], fc, fd);
        basis_regs<O, true, true>(M, M.pairs[pt].lambda, CT.xavg[s], CT.xdiff[s], CT.smin[s], r, fc, fd, u, h);
        const int o = c * NP + s;
        int lg = -16384;
#pragma unroll
        for (int k = 0; k < O; ++k) { sU[o * O + k] = u[k]; sH[o * O + k] = h[k]; lg = max(lg, lg_up(u[k])); }
        sR[4 * o] = R3[0]; sR[4 * o + 1] = R3[1]; sR[4 * o + 2] = R3[2]; sR[4 * o + 3] = r;
        sLg[o] = lg;
        sAB[o] = a | (b << 2);
    }
    __syncthreads();
    // exponent of a cluster's U or Q; LG_BAD marks infinities and NaN
    auto row_exponent = [&](int c, int s0, int n) {
        int lg = 0;
        bool ok = true;
        for (int s = s0; s < s0 + n; ++s) { lg += sLg[c * NP + s]; ok = ok && sLg[c * NP + s] != LG_BAD; }
        return ok ? pow2_above(lg) : LG_BAD;
    };
    constexpr int SI = NBODY == 3 ? 2 : 3, SO = NP - SI;   // slots of the halves
    // products of the three (one, two) slots from s0: two consecutive entries a pair of digits
    auto digits_of = [&](int s0, int nsl) {
        if (nsl == 3) {          // entries p0 * 16 + p1 * 4 + p2
            for (int t = tid; t < nb * 16; t += MT_THREADS) {
                const int c = t >> 4, p0 = (t >> 2) & 3, p1 = t & 3;
                const double* u = sU + (size_t)(c * NP + s0) * O;
                const int e = row_exponent(c, s0, 3), sh = DIG_FIX - e;
                const double g = u[p0] * u[O + p1];
                unsigned char* row = smem + S::a + (size_t)((2 * p0 + (p1 >> 1)) * MDC_TILE + c) * DIG_STRIDE + 8 * (p1 & 1);
#pragma unroll
                for (int p2 = 0; p2 < 4; p2 += 2)
                    put_digits(row + 2 * p2, to_fixed(g * u[2 * O + p2], sh), to_fixed(g * u[2 * O + p2 + 1], sh));
            }
        } else if (nsl == 2) {   // entries p0 * 8 + p1
            for (int t = tid; t < nb * 16; t += MT_THREADS) {
                const int c = t >> 4, p0 = (t >> 1) & 7, p1 = (t & 1) * 4;
                const double* u = sU + (size_t)(c * NP + s0) * O;
                const int sh = DIG_FIX - row_exponent(c, s0, 2);
                unsigned char* row = smem + S::a + (size_t)(p0 * MDC_TILE + c) * DIG_STRIDE + 2 * p1;
#pragma unroll
                for (int k = 0; k < 4; k += 2)
                    put_digits(row + 2 * k, to_fixed(u[p0] * u[O + p1 + k], sh), to_fixed(u[p0] * u[O + p1 + k + 1], sh));
            }
        } else {                 // one slot's 8 entries
            for (int t = tid; t < nb * 4; t += MT_THREADS) {
                const int c = t >> 2, k = (t & 3) * 2;
                const double* u = sU + (size_t)(c * NP + s0) * O;
                const int sh = DIG_FIX - row_exponent(c, s0, 1);
                put_digits(smem + S::a + (size_t)c * DIG_STRIDE + 2 * k, to_fixed(u[k], sh), to_fixed(u[k + 1], sh));
            }
        }
    };
    // 64 clusters x `cols` outputs over K: a warp has 16 clusters and two column tiles
    const int mt = warp >> 2, g4 = lane >> 2, t4 = lane & 3;
    auto product = [&](long long (&val)[2][4], int K, int cols, int up) {
        const int nt = (warp & 3) * 2;
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int r = 0; r < 4; ++r) val[x][r] = 0;
        if (16 * mt >= nb || 8 * nt >= cols) return;
        const bool two = 8 * (nt + 1) < cols;
        float acc[2][DIG_ND][4];
        for (int k8 = 0; k8 < K / 8; ++k8) {
            if ((k8 & 3) == 0) { acc_clear(acc[0]); acc_clear(acc[1]); }
            uint32_t fa[DIG_ND][2], fb[DIG_ND];
            load_a(fa, sm + (uint32_t)S::a + (uint32_t)(k8 * MDC_TILE + 16 * mt) * DIG_STRIDE);
#pragma unroll
            for (int x = 0; x < 2; ++x)
                if (x == 0 || two) {
                    load_b(fb, sm + (uint32_t)S::b + (uint32_t)(k8 * cols + 8 * (nt + x)) * DIG_STRIDE);
                    mma_digits(acc[x], fa, fb);
                }
            if ((k8 & 3) == 3 || k8 + 1 == K / 8) {   // 32 terms
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int r = 0; r < 4; ++r) val[x][r] += acc_value(acc[x], r, up);
            }
        }
    };
    const int upY = up_bits(65536u, T::NI), upW = up_bits(65536u, T::NO);
    long long vy[2][4], vw[2][4];
    digits_of(0, SI);
    asm volatile("cp.async.wait_all;");
    __syncthreads();
    product(vy, T::NI, T::NO, upY);
    __syncthreads();
    fetch(mt_table(T::NI, T::NO), mt_table(T::NO, T::NI));
    digits_of(SI, SO);
    asm volatile("cp.async.wait_all;");
    __syncthreads();
    product(vw, T::NO, T::NI, upW);
    __syncthreads();
    // ---- Y and W as FP64 over the digit tables
    double* sY = reinterpret_cast<double*>(smem);
    double* sW = reinterpret_cast<double*>(smem + S::out);
    auto store = [&](double* out, const long long (&val)[2][4], int cols, int up, int s0, int nsl, const int* ex) {
        const int nt = (warp & 3) * 2;
        if (16 * mt >= nb) return;
#pragma unroll
        for (int r2 = 0; r2 < 2; ++r2) {
            const int c = 16 * mt + g4 + 8 * r2;
            if (c >= nb) continue;
            const int er = row_exponent(c, s0, nsl);
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const int n = 8 * (nt + x) + 2 * t4 + k;
                    if (n >= cols) continue;
                    const int ec = ex[n];
                    out[c * MT_OUT + n] = er == LG_BAD || ec == LG_BAD ? nan("")
                                                                       : from_fixed(val[x][2 * r2 + k], er + ec + 2 - (56 + up));
                }
        }
    };
    store(sY, vy, T::NO, upY, 0, SI, exT);
    store(sW, vw, T::NI, upW, SI, SO, exT + T::NO);
    __syncthreads();
    // ---- one (cluster, slot) per thread: dE/du, the edge force, energy and virial terms
    const double perm = NBODY == 3 ? B.perm3 : B.perm4;
    double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    static_assert(MDC_TILE * NP <= MT_THREADS, "one pass");
    if (tid < nb * NP) {
        const int c = tid / NP, s = tid - c * NP;
        const double* u = sU + (size_t)c * NP * O;
        const double* h = sH + (size_t)tid * O;
        double G[O];
        bool energy;
        if (NBODY == 4) {
            const int hf = s / 3, l = s - 3 * hf, la = l == 0 ? 1 : 0, lb = l == 2 ? 1 : 2;
            const int sl = 16 >> (2 * l), sa = 16 >> (2 * la), sb = 16 >> (2 * lb);
            const double* t = (hf == 0 ? sW : sY) + c * MT_OUT;
            const double* ua = u + (3 * hf + la) * O;
            const double* ub = u + (3 * hf + lb) * O;
#pragma unroll
            for (int k = 0; k < O; ++k) G[k] = 0.0;
#pragma unroll
            for (int i = 0; i < O; ++i)
#pragma unroll
                for (int j = 0; j < O; ++j) {
                    const double p = ua[i] * ub[j];
#pragma unroll
                    for (int k = 0; k < O; ++k) G[k] = fma(t[k * sl + i * sa + j * sb], p, G[k]);
                }
            energy = s == 0;
        } else {
            if (s == 2) {
#pragma unroll
                for (int k = 0; k < O; ++k) G[k] = sY[c * MT_OUT + k];
            } else {
                const double* uo = u + (1 - s) * O;
                const int sk = s == 0 ? 8 : 1, sj = s == 0 ? 1 : 8;
#pragma unroll
                for (int k = 0; k < O; ++k) G[k] = 0.0;
#pragma unroll
                for (int j = 0; j < O; ++j)
#pragma unroll
                    for (int k = 0; k < O; ++k) G[k] = fma(sW[c * MT_OUT + k * sk + j * sj], uo[j], G[k]);
            }
            energy = s == 2;
        }
        double gs = 0.0, E = 0.0;
#pragma unroll
        for (int k = 0; k < O; ++k) {
            gs = fma(G[k], h[k], gs);
            if (energy) E = fma(G[k], u[s * O + k], E);
        }
        double* R = sR + 4 * (size_t)tid;
        const double r = R[3], ge = perm * gs, wv = ge / r;
        const double x = R[0], y = R[1], z = R[2], fx = wv * x, fy = wv * y, fz = wv * z;
        v[0] = perm * E;
        v[1] = -ge * r;
        v[2] = -fx * x; v[3] = -fx * y; v[4] = -fx * z; v[5] = -fy * y; v[6] = -fy * z; v[7] = -fz * z;
        R[0] = fx; R[1] = fy; R[2] = fz;
    }
    __syncthreads();
    // ---- forces, one (cluster, member) per thread
    if (tid < nb * NBODY) {
        const int c = tid / NBODY, m = tid - c * NBODY;
        double fm[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int s = 0; s < NP; ++s) {
            const int ab = sAB[c * NP + s];
            const double* e = sR + 4 * (size_t)(c * NP + s);
            const double sg = (ab & 3) == m ? 1.0 : -1.0;
            if ((ab & 3) == m || (ab >> 2) == m) {
#pragma unroll
                for (int k = 0; k < 3; ++k) fm[k] = fma(sg, e[k], fm[k]);
            }
        }
        double* fo = Fo + 3 * (aofs + member(sM[c], m) % N);
#pragma unroll
        for (int k = 0; k < 3; ++k) atomicAdd(fo + k, fm[k]);
    }
    // ---- scalars: 8 sums over the CTA, halving the values with every exchange
    {
        double a[4];
        const bool hi16 = lane & 16, hi8 = lane & 8, hi4 = lane & 4;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const double send = hi16 ? v[k] : v[k + 4], keep = hi16 ? v[k + 4] : v[k];
            a[k] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const double send = hi8 ? a[k] : a[k + 2], keep = hi8 ? a[k + 2] : a[k];
            a[k] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
        }
        double w = (hi4 ? a[1] : a[0]) + __shfl_xor_sync(0xffffffffu, hi4 ? a[0] : a[1], 4);
        w += __shfl_xor_sync(0xffffffffu, w, 2);
        w += __shfl_xor_sync(0xffffffffu, w, 1);
        if ((lane & 3) == 0) red[(hi16 ? 4 : 0) + (hi8 ? 2 : 0) + (hi4 ? 1 : 0)][warp] = w;
    }
    __syncthreads();
    if (tid < 8) {
        double s = 0.0;
        for (int i = 0; i < MT_THREADS / 32; ++i) s += red[tid][i];
        // v = E, P, W xx xy xz yy yz zz; tensor slots xx=2 xy=3 xz=4 yx=5 yy=6 yz=7 zx=8 zy=9 zz=10
        const int first[8] = {0, 1, 2, 3, 4, 6, 7, 10}, second[8] = {-1, -1, -1, 5, 8, -1, 9, -1};
        double* o = So + (size_t)f * MD_NSCALAR;
        if (s != 0.0) {
            atomicAdd(o + first[tid], s);
            if (second[tid] >= 0) atomicAdd(o + second[tid], s);
        }
    }
}

}  // namespace

static_assert(Mt<3>::O == mdt_order(3) && Mt<4>::O == mdt_order(4), "orders of the tensor-core form");

size_t md_tensor_bytes(int nbody, int ntypes) {
    return (size_t)ntypes * (nbody == 3 ? mt_table(64, 8) + mt_table(8, 64) : 2 * mt_table(64, 64));
}

int md_tensor_exponents(int nbody) { return nbody == 3 ? 72 : 128; }

void launch_md_tables(int nbody, int ntypes, const double* C, unsigned char* tab, int* ex, cudaStream_t st) {
    if (ntypes <= 0) return;
    if (nbody == 3) k_md_digit_tables<3><<<ntypes, 256, 0, st>>>(C, tab, ex);
    else k_md_digit_tables<4><<<ntypes, 256, 0, st>>>(C, tab, ex);
}

void launch_mdt(int nbody, int64_t max_tiles, const ModelDev& M, const FramesDev& F, const ClusterSet& CS,
                const MdBuckets& B, const unsigned char* tab, const int* ex, double* Fo, double* So, cudaStream_t st) {
    if (max_tiles <= 0) return;
    if (nbody == 3) {
        cudaFuncSetAttribute(k_mdt<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MtSmem<3>::total);
        k_mdt<3><<<(unsigned)max_tiles, MT_THREADS, MtSmem<3>::total, st>>>(M, F, CS, B, tab, ex, Fo, So);
    } else {
        cudaFuncSetAttribute(k_mdt<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MtSmem<4>::total);
        k_mdt<4><<<(unsigned)max_tiles, MT_THREADS, MtSmem<4>::total, st>>>(M, F, CS, B, tab, ex, Fo, So);
    }
}

}  // namespace cgd
