// Many-body A rows as digit products on the tensor cores.
//
// Reference: Cheby::Deriv_3B / Deriv_4B (src/Cheby.C:880-1729).  As in assemble.cu, the
// derivative sum of a power tuple factorises over the slots incident to the owner and
// the rest, F_x[p] = sum_clusters M_x[p_I] Q[p_O], and the stress / energy sums over
// S1 and S2: per (owner, cluster type) and per (frame, cluster type) they are dense
// contractions over clusters.  On the FP64 pipe (1/64 of the FP32 rate) they took 3
// multiply-adds per (cluster, member, power) and 13 per (cluster, power) and kept it
// 88% busy; here only the tables remain on it (about 900 operations per 4-body member
// against 11,600).  The products run on mma.sync: a contraction sums a few to a few
// hundred clusters, far below what fills a tcgen05 pipeline, and its accumulators are
// wanted in registers at once to be packed into integers.  16 frames of 256 C/H/N/O
// atoms (4-body, 7,800 rows x 51,209) 36.5 -> 15.5 ms, 32 frames of 384 water atoms
// (3-body, 820 columns) 22.4 -> 8.95 ms.
//
// A group (an owner's clusters of a type, or a frame's share of them) has one exponent, so the
// digits' loss, 2^-61 of the group's largest product, is the same for all its columns.  The bases
// have errors of 2^-53 of a cluster's largest value themselves: against long double the rows'
// errors are those of the FP64 forms (quadruplets of 90 C/H atoms 2.5e-15 of the column's largest
// entry, both; INVRSE_R 5.2e-16 -> 5.5e-16).  Bases without a bound (CONSTANT_DERIV) are left out.
//
// Column sums: PARAM_INDICES puts powers that permutations of equal atoms exchange
// into one column, so a cluster may be taken with two of its equal atoms exchanged; the
// owner is always given the first canonical position of its atom type, and all of an
// owner's clusters of a type share one contraction.
#include <algorithm>

#include "assemble.h"
#include "basis.cuh"
#include "digits.cuh"

namespace cgd {

namespace {

constexpr int OZ_CH = 16;          // clusters whose tables an owner's CTA holds at a time

__device__ __forceinline__ int slot_id(int nb, int a, int b) {   // slot of canonical positions a, b
    const int lo = min(a, b), hi = max(a, b);
    if (nb == 3) return lo + hi - 1;
    return lo == 0 ? hi - 1 : lo + hi;
}

__device__ __forceinline__ int warp_max(int v) { return __reduce_max_sync(0xffffffffu, v); }

__device__ __forceinline__ int frame_of(const FramesDev& F, int64_t atom) {
    int lo = 0, hi = F.nframes - 1;
    while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (F.atom_ofs[mid] <= atom) lo = mid; else hi = mid - 1; }
    return lo;
}

// ---------------------------------------------------------------- magnitudes
// Exponents of one cluster for its owner: eb, its column entries at most 2^eb; ea, its row
// entries at most 2^ea.  False when a basis value is not finite.
template <int NBODY>
__device__ __forceinline__ bool owner_exponents(const int* __restrict__ lgs, int64_t q, int desc, int& eb, int& ea) {
    constexpr int NP = NBODY == 3 ? 3 : 6;
    int g[NP], h[NP];
    bool ok = true;
#pragma unroll
    for (int j = 0; j < NP; ++j) {
        const int v = lgs[q * NP + ((desc >> (4 * j)) & 7)];
        g[j] = (int)(short)(v & 0xffff); h[j] = v >> 16;
        ok = ok && g[j] != LG_BAD && h[j] != LG_BAD;
    }
    if (NBODY == 4) {
        eb = pow2_above(g[3] + g[4] + g[5]);
        // three terms: log2 3 = 25.4 sixteenths
        ea = pow2_above(max(h[0] + g[1] + g[2], max(g[0] + h[1] + g[2], g[0] + g[1] + h[2])) + 26);
    } else {
        eb = pow2_above(g[2]);
        ea = pow2_above(max(h[0] + g[1], g[0] + h[1]));
    }
    return ok;
}

// ---------------------------------------------------------------- owner incidences by type
// One warp per owner atom: its incidences sorted stably by cluster type, with the slot
// order each cluster is read in.  desc: 4 bits per slot of the owner-first frame,
// incident slots first: the cluster's slot and, in bit 3, whether the owner is the
// edge's second member; bits 24..25 the owner's position.  sexp: the exponents of
// owner_exponents, eb in the lower half.  groups[atom][T]: first entry of type T after
// the owner's first entry, entries, largest ea + eb (GROUP_BAD when a basis value is not
// finite) and the outputs' unit (up_bits).
constexpr int GROUP_BAD = 1 << 20;
template <int NBODY>
__global__ void __launch_bounds__(128) k_oz_sort(ModelDev M, FramesDev F, ClusterSet CS, Buckets inc,
                                                 const int64_t* key_frame_ofs, int nreal,
                                                 const int2* __restrict__ tinfo, const int* __restrict__ lgs,
                                                 int* __restrict__ sq,
                                                 int* __restrict__ sdesc, int* __restrict__ sexp,
                                                 int4* __restrict__ groups) {
    extern __shared__ int sCntAll[];
    const int ntypes = NBODY == 3 ? M.ntypes3 : M.ntypes4;
    const int8_t* revs = NBODY == 3 ? M.rev3 : M.rev4;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gatom = blockIdx.x * 4 + warp;
    if (gatom >= nreal) return;
    int* cnt = sCntAll + warp * 2 * (ntypes + 1);
    int* tmax = cnt + ntypes + 1;
    const int f = frame_of(F, gatom);
    const int a = gatom - (int)F.atom_ofs[f];
    const int N = F.natoms[f];
    const int64_t kb = key_frame_ofs[f];
    const int64_t e0 = inc.key_ofs[kb + a];
    const int n = (int)(inc.key_ofs[kb + a + 1] - e0);
    const int64_t qbase = CS.ofs[F.atom_ofs[f]];
    const int* typ = F.type + F.atom_ofs[f];
    for (int k = lane; k <= ntypes; k += 32) { cnt[k] = 0; tmax[k] = -4000; }
    __syncwarp();
    for (int k = lane; k < n; k += 32) atomicAdd(&cnt[CS.type[qbase + (inc.val[e0 + k] >> 2)] + 1], 1);
    __syncwarp();
    int run = 0;
    for (int b = 0; b <= ntypes; b += 32) {
        int v = b + lane <= ntypes ? cnt[b + lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += u; }
        v += run;
        run = __shfl_sync(0xffffffffu, v, 31);
        if (b + lane <= ntypes) cnt[b + lane] = v;
    }
    __syncwarp();
    for (int b = 0; b < n; b += 32) {
        const int k = b + lane;
        const bool act = k < n;
        int q = 0, T = -1 - lane;
        unsigned d = 0;
        if (act) {
            const int v = inc.val[e0 + k];
            const int m = v & 3;
            q = v >> 2;
            const int4 mm = CS.m[qbase + q];
            T = CS.type[qbase + q];
            int ty[NBODY], id = 0, w = 1;
#pragma unroll
            for (int t = 0; t < NBODY; ++t) { ty[t] = typ[member(mm, t) % N]; id += w * (ty[t] + 1); w *= 10; }
            int pos[NBODY], r0 = NBODY, pi = 0, tm = 0;
#pragma unroll
            for (int t = 0; t < NBODY; ++t) { pos[t] = revs[id * NBODY + t]; if (t == m) { pi = pos[t]; tm = ty[t]; } }
#pragma unroll
            for (int t = 0; t < NBODY; ++t) if (ty[t] == tm) r0 = min(r0, pos[t]);
            auto swap = [&](int x) { return x == pi ? r0 : (x == r0 ? pi : x); };
            int oth[NBODY - 1];   // canonical positions other than r0
#pragma unroll
            for (int t = 0; t < NBODY - 1; ++t) oth[t] = t < r0 ? t : t + 1;
#pragma unroll
            for (int t = 0; t < NBODY - 1; ++t) {   // edge (r0, oth[t]): the owner and the member at swap(oth[t])
                const int px = swap(oth[t]);
                int mx = 0;
#pragma unroll
                for (int u = 0; u < NBODY; ++u) if (pos[u] == px) mx = u;
                d |= (unsigned)(slot_id(NBODY, pi, px) | (mx < m ? 8 : 0)) << (4 * t);
            }
            int j = NBODY - 1;
#pragma unroll
            for (int t = 0; t < NBODY - 1; ++t)
#pragma unroll
                for (int u = t + 1; u < NBODY - 1; ++u)
                    d |= (unsigned)slot_id(NBODY, swap(oth[t]), swap(oth[u])) << (4 * j++);
            d |= (unsigned)r0 << 24;
        }
        const unsigned peers = __match_any_sync(0xffffffffu, T);
        const int leader = __ffs(peers) - 1;
        int st = 0;
        if (act && lane == leader) st = cnt[T];
        st = __shfl_sync(0xffffffffu, st, leader);
        if (act) {
            const int64_t o = e0 + st + __popc(peers & ((1u << lane) - 1u));
            int eb, ea;
            const bool ok = owner_exponents<NBODY>(lgs, qbase + q, (int)d, eb, ea);
            sq[o] = q;
            sdesc[o] = (int)d;
            sexp[o] = (eb & 0xffff) | (ea << 16);
            atomicMax(&tmax[T], ok ? ea + eb : GROUP_BAD);
        }
        if (act && lane == leader) cnt[T] = st + __popc(peers);
        __syncwarp();
    }
    // cnt[T] is now the end of type T's entries
    for (int T = 0; T < ntypes; ++T) {
        const int g0 = T == 0 ? 0 : cnt[T - 1], g1 = cnt[T];
        const int tm = tmax[T];
        unsigned long long s = 0;
        for (int k = g0 + lane; k < g1; k += 32) {
            const int e = sexp[e0 + k];
            s += share16((int)(short)(e & 0xffff) + (e >> 16), tm);
        }
        // 64-bit sum of the lanes': their low 16 bits and the rest each fit 32 bits
        s = ((unsigned long long)__reduce_add_sync(0xffffffffu, (unsigned)(s >> 16)) << 16) +
            __reduce_add_sync(0xffffffffu, (unsigned)(s & 0xffffu));
        if (lane == 0) {
            const int up = g1 > g0 ? up_bits(s, (NBODY == 3 ? 2 : 1) * tinfo[T].x) : 0;
            groups[(int64_t)gatom * ntypes + T] = make_int4(g0, g1 - g0, tm, up);
        }
    }
}

// ---------------------------------------------------------------- force rows
template <int NBODY> struct Oz;
template <> struct Oz<3> {
    static constexpr int BASE = 8, NP = 3, NI = 2, THREADS = 128, MINB = 3, COMPS = 1;
    static constexpr int AROWS = 128, BROWS = 48, STAGE = 64 * 24, ZERO = 24;
};
template <> struct Oz<4> {
    static constexpr int BASE = 4, NP = 6, NI = 3, THREADS = 256, MINB = 2, COMPS = 3;
    static constexpr int AROWS = 64, BROWS = 64, STAGE = 64 * 72, ZERO = 1;
};

template <int NBODY>
struct OzSmem {
    using O = Oz<NBODY>;
    // 8 clusters; 64 bytes on, so that a warp's digit stores into two chunks share no bank
    static constexpr size_t CHUNK = (size_t)(O::AROWS + O::BROWS) * DIG_STRIDE + 64;
    size_t stage, basis, idx, total;
    __host__ __device__ explicit OzSmem(int max_words) {
        stage = (OZ_CH / 8) * CHUNK;
        basis = stage + align16((size_t)(O::STAGE + O::ZERO) * sizeof(long long));
        idx = basis + align16((size_t)OZ_CH * (O::NP + O::NI) * O::BASE * sizeof(double));
        total = idx + align16((size_t)max_words * 4);
    }
};

// One CTA per owner atom and, in the 4-body form, Cartesian component.  Per cluster type
// that holds the owner's atom type, up to 16 clusters at a time: slot bases into shared
// memory, tables and their digits, the products added to the staged outputs; then the
// column sums, each written once.
//   4-body: 64 rows (M_k over the incident-slot tuples) x 64 columns (Q).
//   3-body: rows P_0 = h_0 g_1, P_1 = g_0 h_1 over 64 tuples; columns w_u,k Q for
//     k = x, y, z; F_k = P_0 (w_0k Q) + P_1 (w_1k Q), two terms per cluster and output.
// Two CTAs of 256 threads (4-body) or three of 128 (3-body) per SM, so that one CTA's
// table building and column sums run under another's products.
template <int NBODY>
__global__ void __launch_bounds__(Oz<NBODY>::THREADS, Oz<NBODY>::MINB)
k_force_oz(ModelDev M, FramesDev F, ClusterSet CS, Buckets inc, const int64_t* key_frame_ofs,
           const double* __restrict__ pre, const int* __restrict__ sq, const int* __restrict__ sdesc,
           const int* __restrict__ sexp, const int4* __restrict__ groups, OzTables tab, double* A, int64_t lda) {
    using O = Oz<NBODY>;
    using Sum = long long;
    constexpr int NP = O::NP, NI = O::NI, BASE = O::BASE, NT = O::THREADS;
    constexpr int STRIDE = DIG_STRIDE, FIX = DIG_FIX, ND = DIG_ND;
    constexpr uint32_t CHUNK = (uint32_t)OzSmem<NBODY>::CHUNK;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int ord = NBODY == 3 ? M.order3 : M.order4;
    const int ntypes = NBODY == 3 ? M.ntypes3 : M.ntypes4;
    const ClusterTypeDev* types = NBODY == 3 ? M.types3 : M.types4;
    const OzSmem<NBODY> L(tab.max_words);
    unsigned char* sDig = smem_raw;
    Sum* sStage = reinterpret_cast<Sum*>(smem_raw + L.stage);
    double* sG = reinterpret_cast<double*>(smem_raw + L.basis);                  // [c][slot][BASE]
    double* sH = sG + (size_t)OZ_CH * NP * BASE;                            // [c][incident slot][BASE]: h w_k (4-body), h
    uint32_t* sIdx = reinterpret_cast<uint32_t*>(smem_raw + L.idx);
    __shared__ int sShA[OZ_CH], sShB[OZ_CH];
    __shared__ double sWv[NBODY == 3 ? OZ_CH * 6 : 1];                      // 3-body: w_u,k

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gatom = blockIdx.x / O::COMPS, comp = blockIdx.x % O::COMPS;
    const int f = frame_of(F, gatom);
    const int a = gatom - (int)F.atom_ofs[f];
    const double perm = NBODY == 3 ? F.box[f].perm3 : F.box[f].perm4;
    const int64_t e0 = inc.key_ofs[key_frame_ofs[f] + a];
    const int64_t qbase = CS.ofs[F.atom_ofs[f]];
    const int4* grp = groups + (int64_t)gatom * ntypes;
    const int stride = 2 * ord + 4;
    double* const arow = A + (F.row_ofs[f] + 3 * (int64_t)a + comp) * lda;
    const uint32_t dig = smem_addr(sDig);
    const int g4 = lane >> 2, t4 = lane & 3;
    if (tid < O::ZERO) sStage[O::STAGE + tid] = 0;   // where the places of absent powers point

    for (int T = 0; T < ntypes; ++T) {
        const int4 G = grp[T];
        const int nc = G.y;
        if (nc == 0) continue;
        const ClusterTypeDev& CT = types[T];
        const int2 ti = tab.type[T];
        const int ntrue = CT.n_true, words = (ti.x + 1) >> 1;
        if (ntrue == 0) continue;
        const int64_t ent = e0 + G.x;
        const int et = G.z, up = G.w;
        const bool bad = et == GROUP_BAD;   // infinities and NaN reach the rows as NaN
        for (int ch0 = 0; ch0 < nc; ch0 += OZ_CH) {
            const int nb = min(OZ_CH, nc - ch0), npair = ((nb + 7) & ~7) >> 1;
            // (1) slot bases in the owner-first slot order, one (cluster, slot) per thread; the
            // last warp: the powers of two that bring the columns' entries to at most 1/2 per
            // cluster, the rows taking the cluster's magnitude
            static_assert(OZ_CH * NP <= NT - 32, "one pass, the last warp free");
            if (warp == NT / 32 - 1 && lane < nb) {
                const int eb = (int)(short)(sexp[ent + ch0 + lane] & 0xffff);
                sShB[lane] = FIX - eb;
                sShA[lane] = FIX - et + eb;
            }
            if (tid < nb * NP) {
                const int c = tid / NP, j = tid - c * NP;
                const int d = sdesc[ent + ch0 + c] >> (4 * j);
                const double* src = pre + ((size_t)(qbase + sq[ent + ch0 + c]) * NP + (d & 7)) * stride;
                double gv[BASE], hv[BASE];
#pragma unroll
                for (int n = 0; n < BASE; ++n) {
                    gv[n] = n < ord ? src[n] : 0.0;
                    hv[n] = n < ord && j < NI ? src[ord + n] : 0.0;
                }
#pragma unroll
                for (int n = 0; n < BASE; ++n) sG[(size_t)tid * BASE + n] = gv[n];
                if (j < NI) {
                    double* h = sH + (size_t)(c * NI + j) * BASE;
                    const double ir = ((d & 8) ? -1.0 : 1.0) / src[2 * ord];   // sign / r in the form's type
                    if (NBODY == 4) {
                        const double w = src[2 * ord + 1 + comp] * ir;
#pragma unroll
                        for (int n = 0; n < BASE; ++n) h[n] = hv[n] * w;
                    } else {
#pragma unroll
                        for (int n = 0; n < BASE; ++n) h[n] = hv[n];
#pragma unroll
                        for (int k = 0; k < 3; ++k) sWv[c * 6 + j * 3 + k] = src[2 * ord + 1 + k] * ir;
                    }
                }
            }
            __syncthreads();
            // (2) tables, scaled and split into digits, two clusters at a time; the places of
            // absent clusters get zeros
            if (ch0 == 0) {   // where each column's outputs are staged, for the owner's position
                const uint32_t* src = tab.cix + (size_t)((sdesc[ent] >> 24) & 3) * tab.ncix + ti.y;
                for (int k = tid; k < words * ntrue; k += NT) sIdx[k] = src[k];
            }
            if (NBODY == 4) {
                for (int t = tid; t < 32 * npair; t += NT) {
                    const int p = t % npair, z = t / npair;   // npair is 4 or 8
                    const int q0 = z & 3, q1 = (z >> 2) & 3;
                    long long X[2][4];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int c = 2 * p + i;
                        if (c < nb) {
                            if (z < 16) {   // M_k, 4 entries of one (p0, p1)
                                const double* g = sG + (size_t)c * NP * BASE;
                                const double* h = sH + (size_t)c * NI * BASE;
                                const double g0 = g[q0], g1 = g[BASE + q1], gg = g0 * g1;
                                const double b = h[q0] * g1 + g0 * h[BASE + q1];
#pragma unroll
                                for (int q2 = 0; q2 < 4; ++q2)
                                    X[i][q2] = to_fixed(b * g[2 * BASE + q2] + gg * h[2 * BASE + q2], sShA[c]);
                            } else {        // Q, 4 entries of one (p0, p1)
                                const double* g = sG + ((size_t)c * NP + NI) * BASE;
                                const double gg = g[q0] * g[BASE + q1];
#pragma unroll
                                for (int q2 = 0; q2 < 4; ++q2) X[i][q2] = to_fixed(gg * g[2 * BASE + q2], sShB[c]);
                            }
                        } else {
#pragma unroll
                            for (int q2 = 0; q2 < 4; ++q2) X[i][q2] = 0;
                        }
                    }
                    unsigned char* row = sDig + (p >> 2) * CHUNK + (size_t)((z & 16) * 4 + (z & 15)) * STRIDE + 4 * (p & 3);
#pragma unroll
                    for (int q2 = 0; q2 < 4; ++q2) put_digits(row + (size_t)(16 * q2) * STRIDE, X[0][q2], X[1][q2]);
                }
            } else {
                for (int t = tid; t < 22 * npair; t += NT) {
                    const int p = t % npair, z = t / npair;
                    long long X[2][8];
                    unsigned char* base = sDig + (p >> 2) * CHUNK + 4 * (p & 3);
                    if (z < 16) {   // P_0 or P_1 of one p0
                        const int u = z >> 3, q0 = z & 7;
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const int c = 2 * p + i;
                            const double* x = (u == 0 ? sH : sG) + (size_t)c * (u == 0 ? NI : NP) * BASE;
                            const double* y = (u == 0 ? sG + (size_t)c * NP * BASE : sH + (size_t)c * NI * BASE) + BASE;
                            const double x0 = c < nb ? x[q0] : 0.0;
#pragma unroll
                            for (int q1 = 0; q1 < 8; ++q1) X[i][q1] = c < nb ? to_fixed(x0 * y[q1], sShA[c]) : 0;
                        }
#pragma unroll
                        for (int q1 = 0; q1 < 8; ++q1)
                            put_digits(base + (size_t)(64 * u + 8 * q1 + q0) * STRIDE, X[0][q1], X[1][q1]);
                    } else {        // w_u,k Q
                        const int uk = z - 16;
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const int c = 2 * p + i;
                            const double w = c < nb ? sWv[c * 6 + uk] : 0.0;
                            const double* g = sG + ((size_t)c * NP + 2) * BASE;
#pragma unroll
                            for (int q = 0; q < 8; ++q) X[i][q] = c < nb ? to_fixed(w * g[q], sShB[c]) : 0;
                        }
#pragma unroll
                        for (int q = 0; q < 8; ++q)
                            put_digits(base + (size_t)(O::AROWS + 8 * uk + q) * STRIDE, X[0][q], X[1][q]);
                    }
                }
            }
            __syncthreads();
            // (3) products into the staged outputs (a thread meets the same ones in every chunk)
            const int nch = npair >> 2;
            const bool more = ch0 > 0;
            // a pair of values at a time, 16 bytes: eight lanes cover all banks (two rows of
            // four pairs); as two 8-byte accesses they met two to a bank
            auto stage2 = [&](Sum* at, const float (&acc)[ND][4], int r) {
                longlong2* o = reinterpret_cast<longlong2*>(at);
                longlong2 v = make_longlong2(acc_value(acc, 2 * r, up), acc_value(acc, 2 * r + 1, up));
                if (more) { const longlong2 w = *o; v.x += w.x; v.y += w.y; }
                *o = v;
            };
            if (NBODY == 4) {
                const int mt = warp >> 1;
#pragma unroll 1
                for (int half = 0; half < 2; ++half) {
                    const int n0 = half * 32 + (warp & 1) * 16;
                    float acc[2][ND][4];
                    acc_clear(acc[0]);
                    acc_clear(acc[1]);
                    for (int c8 = 0; c8 < nch; ++c8) {
                        uint32_t fa[ND][2], fb[ND];
                        load_a(fa, dig + c8 * CHUNK + (uint32_t)(16 * mt) * STRIDE);
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
                            load_b(fb, dig + c8 * CHUNK + (uint32_t)(O::AROWS + n0 + 8 * x) * STRIDE);
                            mma_digits(acc[x], fa, fb);
                        }
                    }
#pragma unroll
                    for (int x = 0; x < 2; ++x)
#pragma unroll
                        for (int r = 0; r < 2; ++r)
                            stage2(sStage + (16 * mt + g4 + 8 * r) * 72 + n0 + 8 * x + 2 * t4, acc[x], r);
                }
            } else {
                float acc[3][ND][4];
#pragma unroll
                for (int x = 0; x < 3; ++x) acc_clear(acc[x]);
                for (int c8 = 0; c8 < nch; ++c8) {
#pragma unroll 1
                    for (int u = 0; u < 2; ++u) {
                        uint32_t fa[ND][2], fb[ND];
                        load_a(fa, dig + c8 * CHUNK + (uint32_t)(64 * u + 16 * warp) * STRIDE);
#pragma unroll
                        for (int x = 0; x < 3; ++x) {
                            load_b(fb, dig + c8 * CHUNK + (uint32_t)(O::AROWS + 24 * u + 8 * x) * STRIDE);
                            mma_digits(acc[x], fa, fb);
                        }
                    }
                }
#pragma unroll
                for (int x = 0; x < 3; ++x)
#pragma unroll
                    for (int r = 0; r < 2; ++r)
                        stage2(sStage + (16 * warp + g4 + 8 * r) * 24 + 8 * x + 2 * t4, acc[x], r);
            }
        }
        __syncthreads();
        // (4) column sums; value = sum 2^e
        const int e = et + 2 - (56 + up);
        auto column = [&](Sum s) -> double {
            if (bad) return nan("");
            const double v = from_fixed(s, e);
            return perm == 1.0 ? v : v * perm;
        };
        double* const acol = arow + CT.col_base;
        if (NBODY == 4 && words == 1) {   // at most two powers a column: four columns in flight
            for (int c = tid; c < ntrue; c += 4 * NT) {
                Sum s[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t w = c + k * NT < ntrue ? sIdx[c + k * NT] : O::STAGE | (O::STAGE << 16);
                    s[k] = sStage[w & 0xffff] + sStage[w >> 16];
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) if (c + k * NT < ntrue) acol[c + k * NT] = column(s[k]);
            }
        } else if (NBODY == 4) {
            for (int c = tid; c < ntrue; c += NT) {
                Sum s = 0;
#pragma unroll 2
                for (int k = 0; k < words; ++k) {
                    const uint32_t w = sIdx[k * ntrue + c];
                    s += sStage[w & 0xffff] + sStage[w >> 16];
                }
                acol[c] = column(s);
            }
        } else {
            for (int c = tid; c < ntrue; c += NT) {
                Sum s[3] = {0, 0, 0};
                for (int k = 0; k < words; ++k) {
                    const uint32_t w = sIdx[k * ntrue + c];
                    const Sum *x = sStage + (w & 0xffff), *y = sStage + (w >> 16);
                    s[0] += x[0] + y[0]; s[1] += x[8] + y[8]; s[2] += x[16] + y[16];
                }
#pragma unroll
                for (int k = 0; k < 3; ++k) acol[k * lda + c] = column(s[k]);
            }
        }
    }
}

// ---------------------------------------------------------------- stress / energy rows
// One CTA of 16 warps per (frame, cluster type), up to VIR_CLUSTERS clusters and, in the
// 4-body form, component (0 energy, 1..6 xx yy zz xy xz yz).
//   4-body: W_k = A1_k Q2 + Q1 A2_k over 64 x 64 outputs, two terms per cluster; E = Q1 Q2.
//   3-body: W_k = P_0 (v_0k g_2) + P_1 (v_1k g_2) + Q1 (v_2k h_2) over 64 x 8 outputs, all
//     components in one CTA (a warp pair each); E = Q1 g_2.
// The next chunk's tables are built while warps that have finished theirs run the current
// chunk's products; chunks after that arrive by cp.async.
template <int NBODY> struct Vz;
template <> struct Vz<3> {
    static constexpr int BASE = 8, NP = 3, CH = 8, ROWS = 344, OUT = 7 * 64 * 8, TERMS = 3;
};
template <> struct Vz<4> {
    static constexpr int BASE = 4, NP = 6, CH = 16, ROWS = 256, OUT = 64 * 72, TERMS = 2;
};
constexpr int VZ_THREADS = 512;

template <int NBODY>
struct VzSmem {
    using V = Vz<NBODY>;
    static constexpr size_t CHUNK = (size_t)V::ROWS * DIG_STRIDE + 64;   // 8 clusters, as OzSmem
    static constexpr size_t BUF = CHUNK * (V::CH / 8);
    size_t raw, basis, q, sh, total;
    size_t raw_size;
    __host__ __device__ explicit VzSmem(int ord) {
        const size_t out = align16((size_t)V::OUT * sizeof(double));   // the column sums' stage reuses the tables
        raw_size = align16((size_t)V::CH * V::NP * (2 * ord + 4) * sizeof(double));
        raw = 2 * BUF > out ? 2 * BUF : out;
        basis = raw + 2 * raw_size;
        // slot values of a chunk: g, h (4-body: h v_k; 3-body: and the six v_k)
        q = basis + align16((size_t)V::CH * V::NP * (2 * V::BASE + (NBODY == 3 ? 6 : 0)) * sizeof(double));
        sh = q + VIR_CLUSTERS * 4;
        total = sh + VIR_CLUSTERS * 4;
    }
};

__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src));
}

template <int NBODY>
__global__ void __launch_bounds__(VZ_THREADS, 1)
k_virial_oz(ModelDev M, FramesDev F, ClusterSet CS, Buckets bytype, const int64_t* key_frame_ofs, int ncomp,
            const double* __restrict__ pre, const int* __restrict__ lgs, OzTables tab,
            double* __restrict__ part, int ntrue_max, int nchunks_max) {
    using V = Vz<NBODY>;
    using Sum = long long;
    constexpr int NP = V::NP, BASE = V::BASE, CH = V::CH;
    constexpr int STRIDE = DIG_STRIDE, FIX = DIG_FIX, ND = DIG_ND;
    constexpr uint32_t CHUNK = (uint32_t)VzSmem<NBODY>::CHUNK;
    constexpr uint32_t BUF = (uint32_t)VzSmem<NBODY>::BUF;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int ntypes = NBODY == 3 ? M.ntypes3 : M.ntypes4;
    const int f = blockIdx.x / ntypes;
    const int T = blockIdx.x % ntypes;
    if (F.stress_rows[f] == 0 && F.energy_rows[f] == 0) return;
    const ClusterTypeDev& CT = (NBODY == 3 ? M.types3 : M.types4)[T];
    if (CT.n_allowed == 0) return;
    const int64_t kb = key_frame_ofs[f];
    const int64_t t0 = bytype.key_ofs[kb + T], t1 = bytype.key_ofs[kb + T + 1];
    const int64_t c0 = t0 + (int64_t)blockIdx.z * VIR_CLUSTERS;
    if (c0 >= t1) return;
    const int n = (int)min((int64_t)VIR_CLUSTERS, t1 - c0);
    const int comp = NBODY == 4 ? blockIdx.y : 0;
    const int ord = NBODY == 3 ? M.order3 : M.order4;
    const int stride = 2 * ord + 4;
    const int64_t qbase = CS.ofs[F.atom_ofs[f]];
    const VzSmem<NBODY> L(ord);
    double* sB = reinterpret_cast<double*>(smem_raw + L.basis);
    int* sQ = reinterpret_cast<int*>(smem_raw + L.q);
    int* sE = reinterpret_cast<int*>(smem_raw + L.sh);   // two exponents of each cluster
    __shared__ int sMax[2], sBad;
    __shared__ unsigned sSum[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int lgr = lg_up(NBODY == 3 ? M.maxcut3 : M.maxcut4);   // |r_a r_b / r| <= r < the cut-off
    if (tid == 0) { sMax[0] = sMax[1] = -4000; sBad = 0; sSum[0] = sSum[1] = 0; }
    __syncthreads();
    {   // powers of two: one factor of each term to at most 1/2 per cluster, the other one
        // taking the cluster's magnitude
        int m0 = -4000, m1 = -4000;
        bool ok = true;
        static_assert(VIR_CLUSTERS <= VZ_THREADS, "one cluster per thread");
        if (tid < n) {
            const int c = tid;
            const int q = bytype.val[c0 + c];
            sQ[c] = q;
            int g[NP], h[NP];
#pragma unroll
            for (int s = 0; s < NP; ++s) {
                const int v = lgs[(qbase + q) * NP + s];
                g[s] = (int)(short)(v & 0xffff); h[s] = v >> 16;
                ok = ok && g[s] != LG_BAD && h[s] != LG_BAD;
            }
            if (NBODY == 4) {
                const int e1 = pow2_above(g[0] + g[1] + g[2]), e2 = pow2_above(g[3] + g[4] + g[5]);
                const int a1 = pow2_above(max(h[0] + g[1] + g[2], max(g[0] + h[1] + g[2], g[0] + g[1] + h[2])) + lgr + 26);
                const int a2 = pow2_above(max(h[3] + g[4] + g[5], max(g[3] + h[4] + g[5], g[3] + g[4] + h[5])) + lgr + 26);
                m0 = max(m0, comp == 0 ? e1 + e2 : max(a1 + e2, a2 + e1));
                sE[c] = (e1 & 0xffff) | (e2 << 16);
            } else {
                const int eb = pow2_above(g[2] + lgr), eq = pow2_above(g[0] + g[1]);
                m0 = max(m0, max(pow2_above(max(h[0] + g[1], g[0] + h[1])) + eb, eq + pow2_above(h[2] + lgr)));
                m1 = max(m1, eq + pow2_above(g[2]));
                sE[c] = (eb & 0xffff) | (eq << 16);
            }
        }
        const int w0 = warp_max(m0), w1 = warp_max(m1);
        ok = __all_sync(0xffffffffu, ok);
        if (lane == 0) { atomicMax(&sMax[0], w0); atomicMax(&sMax[1], w1); if (!ok) sBad = 1; }
        __syncthreads();
        const unsigned s0 = __reduce_add_sync(0xffffffffu, tid < n ? share16(m0, sMax[0]) : 0u);
        const unsigned s1 = __reduce_add_sync(0xffffffffu, NBODY == 3 && tid < n ? share16(m1, sMax[1]) : 0u);
        if (lane == 0) { atomicAdd(&sSum[0], s0); atomicAdd(&sSum[1], s1); }
    }
    __syncthreads();
    const int et = sMax[0], ete = sMax[1];
    const int up = up_bits(max(sSum[0], sSum[1]), V::TERMS);
    const int nchunk = (n + CH - 1) / CH;
    const uint32_t rawa = smem_addr(smem_raw + L.raw);
    auto fetch = [&](int ch) {   // chunk ch's slot bases, cluster by cluster as they lie
        if (ch < nchunk) {
            const int words = NP * stride * (int)sizeof(double) / 8, nb = min(CH, n - ch * CH);
            const uint32_t dst = rawa + (ch & 1) * (uint32_t)L.raw_size;
            for (int t = tid; t < nb * words; t += VZ_THREADS) {
                const int c = t / words, w = t - c * words;
                cp_async8(dst + t * 8, reinterpret_cast<const char*>(pre + (size_t)(qbase + sQ[ch * CH + c]) * NP * stride) + 8 * w);
            }
        }
        asm volatile("cp.async.commit_group;");
    };
    // slot values of chunk ch: [c][slot][g | h' | v], h' = h v_k in the 4-body form
    constexpr int SB = 2 * BASE + (NBODY == 3 ? 6 : 0);
    auto slots = [&](int ch) {
        const int nb = min(CH, n - ch * CH);
        const double* raw = reinterpret_cast<const double*>(smem_raw + L.raw + (ch & 1) * L.raw_size);
        if constexpr (NBODY == 3) {
            // one division or one value per thread: six divisions of 24 (cluster, slot) pairs
            // by one warp (an FP64 division is a dozen instructions of 64 cycles) kept the
            // other 15 at the barrier: triplet rows of 32 frames of 384 atoms 3.71 -> 2.81 ms
            for (int t = tid; t < nb * NP * 6; t += VZ_THREADS) {
                const int cs = t / 6, k = t - 6 * cs;
                const double* src = raw + (size_t)cs * stride + 2 * ord;
                const int ka = k < 3 ? k : (k == 5 ? 1 : 0), kc = k < 3 ? k : (k == 3 ? 1 : 2);
                sB[(size_t)cs * SB + 2 * BASE + k] = src[1 + ka] * src[1 + kc] / src[0];
            }
            for (int t = VZ_THREADS - 1 - tid; t < nb * NP * 2 * BASE; t += VZ_THREADS) {
                const int cs = t / (2 * BASE), k = t % (2 * BASE), n = k % BASE;
                sB[(size_t)cs * SB + k] = n < ord ? raw[(size_t)cs * stride + (k < BASE ? n : ord + n)] : 0.0;
            }
        } else {
            for (int t = tid; t < nb * NP; t += VZ_THREADS) {
                const double* src = raw + (size_t)t * stride;
                double* o = sB + (size_t)t * SB;
                const double r = src[2 * ord];
                const double x[3] = {src[2 * ord + 1], src[2 * ord + 2], src[2 * ord + 3]};
                const int ka = comp <= 3 ? comp - 1 : (comp == 6 ? 1 : 0), kc = comp <= 3 ? comp - 1 : (comp == 4 ? 1 : 2);
                const double v = comp == 0 ? 0.0 : (ka == 0 ? x[0] : (ka == 1 ? x[1] : x[2])) *
                                                   (kc == 0 ? x[0] : (kc == 1 ? x[1] : x[2])) / r;
#pragma unroll
                for (int k = 0; k < BASE; ++k) {
                    o[k] = k < ord ? src[k] : 0.0;
                    o[BASE + k] = k < ord ? src[ord + k] * v : 0.0;
                }
            }
        }
    };
    auto build = [&](int ch) {   // tables of chunk ch into buffer ch & 1
        const int nb = min(CH, n - ch * CH);
        unsigned char* buf = smem_raw + (ch & 1) * BUF;
        const int* ex = sE + ch * CH;
        if (NBODY == 4) {
            // rows: A1 (Q1 for the energy) 0.., Q1 64.., Q2 128.., A2 192..; an item is a pair of
            // clusters, a half (S1 or S2), (p0, p1) and two of the p2
            const int p = tid & 7, z = (tid >> 3) & 15, two = (tid >> 7) & 1, hf = tid >> 8;
            const int q0 = z & 3, q1 = z >> 2;
            long long XQ[2][2], XA[2][2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int c = 2 * p + i;
                if (c < nb) {
                    const double* s = sB + ((size_t)c * NP + 3 * hf) * SB;
                    const int e1 = (int)(short)(ex[c] & 0xffff), e2 = ex[c] >> 16;
                    // S1: A1 (or the energy's Q1) carries the magnitude, Q1 is scaled to 1/2; S2: the other way round
                    const int eown = hf == 0 ? e1 : e2, eoth = hf == 0 ? e2 : e1;
                    const int shq = comp == 0 && hf == 0 ? FIX - et + eoth : FIX - eown, sha = FIX - et + eoth;
                    const double g0 = s[q0], g1 = s[SB + q1], gg = g0 * g1;
                    const double b = s[BASE + q0] * g1 + g0 * s[SB + BASE + q1];
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const int q2 = 2 * two + k;
                        XQ[i][k] = to_fixed(gg * s[2 * SB + q2], shq);
                        XA[i][k] = comp == 0 ? 0ll : to_fixed(b * s[2 * SB + q2] + gg * s[2 * SB + BASE + q2], sha);
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < 2; ++k) XQ[i][k] = XA[i][k] = 0;
                }
            }
            unsigned char* row = buf + (p >> 2) * CHUNK + (size_t)(z + 32 * two) * STRIDE + 4 * (p & 3);
            const int rq = comp == 0 ? (hf == 0 ? 0 : 128) : (hf == 0 ? 64 : 128), ra = hf == 0 ? 0 : 192;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                put_digits(row + (size_t)(rq + 16 * k) * STRIDE, XQ[0][k], XQ[1][k]);
                if (comp != 0) put_digits(row + (size_t)(ra + 16 * k) * STRIDE, XA[0][k], XA[1][k]);
            }
        } else {
            // rows: P_0 0.., P_1 64.., Q1 128.., then 24 per component (v_0 g, v_1 g, v_2 h), g
            for (int t = tid; t < 560; t += VZ_THREADS) {
                long long X[2][6];
                if (t < 256) {          // a pair of clusters, one (p0, p1), three tables
                    const int p = t & 3, q0 = (t >> 2) & 7, qq = t >> 5;
                    unsigned char* row = buf + 4 * p + (size_t)(q0 + 8 * qq) * STRIDE;
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int c = 2 * p + i;
                        const bool on = c < nb;
                        const double* s = sB + (size_t)c * NP * SB;
                        const int eb = on ? (int)(short)(ex[c] & 0xffff) : 0, eq = on ? ex[c] >> 16 : 0;
                        X[i][0] = on ? to_fixed(s[BASE + q0] * s[SB + qq], FIX - et + eb) : 0;
                        X[i][1] = on ? to_fixed(s[q0] * s[SB + BASE + qq], FIX - et + eb) : 0;
                        X[i][2] = on ? to_fixed(s[q0] * s[SB + qq], FIX - eq) : 0;
                    }
#pragma unroll
                    for (int k = 0; k < 3; ++k) put_digits(row + (size_t)(64 * k) * STRIDE, X[0][k], X[1][k]);
                } else if (t < 544) {   // a pair of clusters, component k, factor j, two powers
                    const int v = t - 256, p = v & 3, quart = (v >> 2) & 3, kj = v >> 4, k = kj / 3, j = kj - 3 * k;
                    unsigned char* row = buf + 4 * p + (size_t)(192 + 24 * k + 8 * j + 2 * quart) * STRIDE;
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int c = 2 * p + i;
                        const bool on = c < nb;
                        const double* s = sB + (size_t)c * NP * SB;
                        const int eb = on ? (int)(short)(ex[c] & 0xffff) : 0, eq = on ? ex[c] >> 16 : 0;
                        const double w = on ? s[j * SB + 2 * BASE + k] : 0.0;
                        const double* y = s + 2 * SB + (j == 2 ? BASE : 0) + 2 * quart;
                        const int sh = j == 2 ? FIX - et + eq : FIX - eb;
#pragma unroll
                        for (int q = 0; q < 2; ++q) X[i][q] = on ? to_fixed(w * y[q], sh) : 0;
                    }
#pragma unroll
                    for (int q = 0; q < 2; ++q) put_digits(row + (size_t)q * STRIDE, X[0][q], X[1][q]);
                } else {                // the energy's g
                    const int v = t - 544, p = v & 3, quart = v >> 2;
                    unsigned char* row = buf + 4 * p + (size_t)(336 + 2 * quart) * STRIDE;
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int c = 2 * p + i;
                        const bool on = c < nb;
                        const int eq = on ? ex[c] >> 16 : 0;
                        const double* y = sB + ((size_t)c * NP + 2) * SB + 2 * quart;
#pragma unroll
                        for (int q = 0; q < 2; ++q) X[i][q] = on ? to_fixed(y[q], FIX - ete + eq) : 0;
                    }
#pragma unroll
                    for (int q = 0; q < 2; ++q) put_digits(row + (size_t)q * STRIDE, X[0][q], X[1][q]);
                }
            }
        }
    };
    Sum val[2][4];
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int r = 0; r < 4; ++r) val[x][r] = 0;
    // 4-body: a warp has 16 rows, two column tiles; 3-body: one component, two row tiles
    const int wk = warp >> 1;
    const bool works = NBODY == 4 || wk < ncomp;
    auto products = [&](int ch) {
        if (!works) return;
        const uint32_t buf = smem_addr(smem_raw) + (ch & 1) * BUF;
        float acc[2][ND][4];
        acc_clear(acc[0]);
        acc_clear(acc[1]);
        if (NBODY == 4) {
            const int nch = (min(CH, n - ch * CH) + 7) >> 3;
            const int mt = warp >> 2, nt = (warp & 3) * 2;
            for (int c8 = 0; c8 < nch; ++c8)
#pragma unroll 1
                for (int hf = 0; hf < (comp == 0 ? 1 : 2); ++hf) {
                    uint32_t fa[ND][2], fb[ND];
                    load_a(fa, buf + c8 * CHUNK + (uint32_t)(64 * hf + 16 * mt) * STRIDE);
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        load_b(fb, buf + c8 * CHUNK + (uint32_t)(128 + 64 * hf + 8 * (nt + x)) * STRIDE);
                        mma_digits(acc[x], fa, fb);
                    }
                }
        } else {
#pragma unroll 1
            for (int j = wk == 0 ? 2 : 0; j < 3; ++j) {
                uint32_t fa[ND][2], fb[ND];
                load_b(fb, buf + (uint32_t)(wk == 0 ? 336 : 192 + 24 * (wk - 1) + 8 * j) * STRIDE);
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    load_a(fa, buf + (uint32_t)(64 * j + 16 * (2 * (warp & 1) + x)) * STRIDE);
                    mma_digits(acc[x], fa, fb);
                }
            }
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int r = 0; r < 4; ++r) val[x][r] += acc_value(acc[x], r, up);
    };
    static_assert(CH * V::TERMS <= MAGIC_TERMS, "exact accumulators");
    // pipeline: bases of chunk i + 2 on their way, tables of i + 1 built, products of i
    fetch(0);
    fetch(1);
    for (int i = -1; i < nchunk; ++i) {
        asm volatile("cp.async.wait_group 1;");
        __syncthreads();
        if (i + 1 < nchunk) slots(i + 1);
        __syncthreads();
        fetch(i + 3);
        if (i + 1 < nchunk) build(i + 1);
        if (i >= 0) products(i);
    }
    asm volatile("cp.async.wait_group 0;");
    __syncthreads();
    // outputs to shared memory (over the tables), then the column sums
    double* sOut = reinterpret_cast<double*>(smem_raw);
    const bool bad = sBad != 0;   // infinities and NaN reach the rows as NaN
    const int esel = NBODY == 3 && wk == 0 ? ete : et;
    const int e = esel + 2 - (56 + up);
    auto value = [&](Sum s) -> double {
        return bad ? nan("") : from_fixed(s, e);
    };
    if (works) {
        const int g4 = lane >> 2, t4 = lane & 3;
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                double* o;
                if (NBODY == 4)
                    o = sOut + (16 * (warp >> 2) + g4 + 8 * (r >> 1)) * 72 + 8 * ((warp & 3) * 2 + x) + 2 * t4 + (r & 1);
                else
                    o = sOut + (wk * 64 + 16 * (2 * (warp & 1) + x) + g4 + 8 * (r >> 1)) * 8 + 2 * t4 + (r & 1);
                *o = value(val[x][r]);
            }
    }
    __syncthreads();
    const int2 ti = tab.type[T];
    const uint32_t* ix = tab.cix + ti.y;   // the first position's
    const int ntrue = CT.n_true, words = (ti.x + 1) >> 1;
    double* out = part + ((size_t)blockIdx.x * nchunks_max + blockIdx.z) * 7 * ntrue_max;
    for (int col = tid; col < ntrue; col += VZ_THREADS) {
        double s[NBODY == 4 ? 1 : 7];
#pragma unroll
        for (int k = 0; k < (NBODY == 4 ? 1 : 7); ++k) s[k] = 0;
#pragma unroll 2
        for (int w = 0; w < words; ++w) {
            const uint32_t v = ix[w * ntrue + col];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int o = i ? v >> 16 : v & 0xffff;
                if (o == (NBODY == 4 ? Oz<4>::STAGE : Oz<3>::STAGE)) continue;   // an absent power
                if (NBODY == 4) {
                    s[0] += sOut[o];
                } else {
                    const double* x = sOut + (o / 24) * 8 + o % 24;
#pragma unroll
                    for (int k = 0; k < (NBODY == 4 ? 1 : 7); ++k) if (k < ncomp) s[k] += x[k * 512];
                }
            }
        }
#pragma unroll
        for (int k = 0; k < (NBODY == 4 ? 1 : 7); ++k) {
            const int kk = NBODY == 4 ? comp : k;
            if (kk < ncomp) out[(size_t)kk * ntrue_max + col] = kk == 0 ? s[k] : -s[k];
        }
    }
}

}  // namespace

// ---------------------------------------------------------------- rules and launchers
template <int NBODY>
static void force_oz(int nreal, const ModelDev& M, const FramesDev& F, const ClusterSet& CS, const Buckets& inc,
                     const int64_t* kfo, const OzWork& W, double* A, int64_t lda, cudaStream_t st) {
    const int nt = NBODY == 3 ? M.ntypes3 : M.ntypes4;
    k_oz_sort<NBODY><<<(nreal + 3) / 4, 128, (size_t)8 * (nt + 1) * sizeof(int), st>>>(M, F, CS, inc, kfo, nreal,
                                                                                       W.tab.type, W.lgs, W.sq, W.sdesc,
                                                                                       W.sexp, W.groups);
    const size_t smem = OzSmem<NBODY>(W.tab.max_words).total;
    cudaFuncSetAttribute(k_force_oz<NBODY>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_force_oz<NBODY><<<nreal * Oz<NBODY>::COMPS, Oz<NBODY>::THREADS, smem, st>>>(
        M, F, CS, inc, kfo, W.basis, W.sq, W.sdesc, W.sexp, W.groups, W.tab, A, lda);
}

void launch_force_oz(int nbody, int nreal, const ModelDev& M, const FramesDev& F, const ClusterSet& CS,
                     const Buckets& inc, const int64_t* kfo, const OzWork& W, double* A, int64_t lda,
                     cudaStream_t st) {
    if (nreal <= 0) return;
    if (nbody == 3) force_oz<3>(nreal, M, F, CS, inc, kfo, W, A, lda, st);
    else force_oz<4>(nreal, M, F, CS, inc, kfo, W, A, lda, st);
}

template <int NBODY>
static void virial_oz(int nframes, int ncomp, int nchunks_max, int ntrue_max, const ModelDev& M, const FramesDev& F,
                      const ClusterSet& CS, const Buckets& byt, const int64_t* kfo, const OzWork& W, double* part,
                      cudaStream_t st) {
    const int nt = NBODY == 3 ? M.ntypes3 : M.ntypes4;
    const size_t smem = VzSmem<NBODY>(NBODY == 3 ? M.order3 : M.order4).total;
    cudaFuncSetAttribute(k_virial_oz<NBODY>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const dim3 grid((unsigned)(nframes * nt), NBODY == 4 ? (unsigned)ncomp : 1u, (unsigned)nchunks_max);
    k_virial_oz<NBODY><<<grid, VZ_THREADS, smem, st>>>(M, F, CS, byt, kfo, ncomp, W.basis, W.lgs, W.tab, part,
                                                       ntrue_max, nchunks_max);
}

void launch_virial_oz(int nbody, int nframes, int ncomp, int nchunks_max, int ntrue_max, const ModelDev& M,
                      const FramesDev& F, const ClusterSet& CS, const Buckets& byt, const int64_t* kfo,
                      const OzWork& W, double* part, cudaStream_t st) {
    if (nframes <= 0) return;
    if (nbody == 3) virial_oz<3>(nframes, ncomp, nchunks_max, ntrue_max, M, F, CS, byt, kfo, W, part, st);
    else virial_oz<4>(nframes, ncomp, nchunks_max, ntrue_max, M, F, CS, byt, kfo, W, part, st);
}

bool oz_fits(int nbody, int ord, int max_words) {
    // The orders that use at least a quarter of the padded 64 x 64 / 64 x 8 grids: an output
    // costs the same whether its power exists or not, and a 4-body order of 3 would use 729
    // of 4,096.
    if (nbody == 3 ? (ord < 5 || ord > 8) : ord != 4) return false;
    const size_t lim = 226 * 1024;
    return nbody == 3 ? OzSmem<3>(max_words).total <= lim && VzSmem<3>(ord).total <= lim
                      : OzSmem<4>(max_words).total <= lim && VzSmem<4>(ord).total <= lim;
}

}  // namespace cgd
