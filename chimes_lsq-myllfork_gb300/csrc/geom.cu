// Geometry, neighbour lists and cluster enumeration on the device.
//
// Reference behaviour reproduced here (all index sets are bit-exact):
//   FRAME::build_layers / update_ghost  src/ClassDefs.C:2361-2409, 2685-2752
//   BOX::WRAP_ATOM / LAYER_ATOM          src/ClassDefs.C:2064-2164
//   NEIGHBORS::DO_UPDATE_BIG / _SMALL    src/ClassDefs.C:137-393
//   triplet loops of Cheby::Deriv_3B     src/Cheby.C:981-1054
//   quadruplet loops of Cheby::Deriv_4B  src/Cheby.C:1387-1500
//   FCUT::PROCEED                        src/Fcut.C:125-140
// The reference decides membership with FP64 distances.  An FP32 distance decides where it
// differs from the cut-off by more than frame_margin (dev.cuh), which is above the rounding of
// the frame's FP32 positions; nearer, the exact FP64 sequence does.
#include <cooperative_groups.h>

#include "dev.cuh"
#include "kernels.h"

namespace cgd {

// The slots' cut-offs for lists of this skin.
__global__ void k_cuts(const ClusterTypeDev* types, int n, int np, double skin, CutDev* out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * np) return;
    CutDev c;
    c.cut = types[t / np].smax[t % np] + skin;
    c.cutf = (float)c.cut;
    c.pad = 0.0f;
    out[t] = c;
}
void launch_cuts(const ModelDev& M, int nbody, double skin, CutDev* out, cudaStream_t st) {
    const int n = nbody == 3 ? M.ntypes3 : M.ntypes4, np = nbody == 3 ? 3 : 6;
    if (n > 0) k_cuts<<<(n * np + 127) / 128, 128, 0, st>>>(nbody == 3 ? M.types3 : M.types4, n, np, skin, out);
}

// ---------------------------------------------------------------- ghost set-up
__global__ void k_frame_setup(FramesDev F, int64_t total_ghosts) {
    int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= total_ghosts) return;
    // frame lookup: binary search over ghost_ofs
    int lo = 0, hi = F.nframes - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (F.ghost_ofs[mid] <= gid) lo = mid; else hi = mid - 1;
    }
    const int f = lo;
    const int N = F.natoms[f];
    const int g = (int)(gid - F.ghost_ofs[f]);
    const int a = g % N;
    const int k = g / N;   // 0 = real image
    const BoxDev& B = F.box[f];
    const double* x0 = F.xyz + 3 * (F.atom_ofs[f] + a);
    double w[3];
    // WRAP_ATOM (src/ClassDefs.C:2075-2119); with stored shifts (MD list reuse) the
    // shift of the last list build is applied instead of a fresh floor
    int* sh = (F.shift && F.shift_mode) ? F.shift + 3 * (F.atom_ofs[f] + a) : nullptr;
    const bool use_stored = sh && F.shift_mode == 2;
    const bool store = sh && F.shift_mode == 1 && k == 0;
    if (B.is_ortho) {
        double L3[3] = {B.lx, B.ly, B.lz};
        for (int q = 0; q < 3; ++q) {
            int idx = use_stored ? sh[q] : (int)floor(__ddiv_rn(x0[q], L3[q]));
            if (store) sh[q] = idx;
            w[q] = subrn(x0[q], mulrn((double)idx, L3[q]));
        }
    } else {
        double t[3];
        for (int q = 0; q < 3; ++q) t[q] = dot3rn(B.inv[3 * q], B.inv[3 * q + 1], B.inv[3 * q + 2], x0[0], x0[1], x0[2]);
        for (int q = 0; q < 3; ++q) {
            int idx = use_stored ? sh[q] : (int)floor(t[q]);
            if (store) sh[q] = idx;
            t[q] = subrn(t[q], (double)idx);
        }
        for (int q = 0; q < 3; ++q) w[q] = dot3rn(B.h[3 * q], B.h[3 * q + 1], B.h[3 * q + 2], t[0], t[1], t[2]);
    }
    double c[3] = {w[0], w[1], w[2]};
    if (k > 0) {   // LAYER_ATOM (src/ClassDefs.C:2132-2164)
        int n1, n2, n3;
        layer_index(k - 1, F.nlayers, n1, n2, n3);
        if (B.is_ortho) {
            c[0] = addrn(w[0], mulrn((double)n1, B.h[0]));
            c[1] = addrn(w[1], mulrn((double)n2, B.h[4]));
            c[2] = addrn(w[2], mulrn((double)n3, B.h[8]));
        } else {
            double t[3];
            for (int q = 0; q < 3; ++q) t[q] = dot3rn(B.inv[3 * q], B.inv[3 * q + 1], B.inv[3 * q + 2], w[0], w[1], w[2]);
            t[0] = addrn(t[0], (double)n1); t[1] = addrn(t[1], (double)n2); t[2] = addrn(t[2], (double)n3);
            for (int q = 0; q < 3; ++q) c[q] = dot3rn(B.h[3 * q], B.h[3 * q + 1], B.h[3 * q + 2], t[0], t[1], t[2]);
        }
    }
    double* s = F.scaled + 3 * gid;
    for (int q = 0; q < 3; ++q) s[q] = dot3rn(B.inv[3 * q], B.inv[3 * q + 1], B.inv[3 * q + 2], c[0], c[1], c[2]);
    float4 c32 = make_float4((float)c[0], (float)c[1], (float)c[2], 0.f);
    reinterpret_cast<float4*>(F.cart32)[gid] = c32;
}

// ---------------------------------------------------------------- neighbour lists
__device__ __forceinline__ int frame_of_real(const FramesDev& F, int64_t atom) {
    int lo = 0, hi = F.nframes - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (F.atom_ofs[mid] <= atom) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Warps scan the ghosts of the images near a real atom in ghost-index order, 32 at a
// time, nw warps sharing one atom as contiguous slices of that order, so the lists come
// out in ghost-index order and the fill pass is deterministic.
//  * An image of the cell that lies beyond the search radius holds no neighbour: the
//    cell's bounding box, shifted, is tested once per image.  Ordered lists (i <= parent)
//    start each image at the atom's own index.
//  * FP32 distances decide except within frame_margin of a cut-off; the exact FP64 distance,
//    whose pipe has 1/64 of the rate, is formed there and, in the fill pass, once per
//    listed ghost with 32 of them side by side.
// Forming it for every chunk with a candidate in every pass, dividing by the atom count per
// ghost and scanning all atoms of a near image took 1.37 of the 1.96 ms of an MD force
// call on frames of 64, 301, 1111 and 2600 atoms (now 0.16 of 0.66 ms), and 1.38 of 11.3 ms
// of the FP64 rows of 32 frames of 384 (now 8.9 ms in all).
constexpr int NEIGH_IMG = 1024;   // images tested for reach (four layers); every image is scanned above

template <bool FILL>
__global__ void __launch_bounds__(32 * NEIGH_WARPS) k_neigh(ModelDev M, FramesDev F, NeighDev NB, int nw) {
    __shared__ int sc[3][NEIGH_WARPS];
    __shared__ int sHit[NEIGH_WARPS][64];         // ghosts: any number of image layers
    __shared__ uint8_t sLists[NEIGH_WARPS][64];   // and their lists
    __shared__ unsigned sNear[NEIGH_WARPS][NEIGH_IMG / 32];
    __shared__ float2 sPair[55];   // s_max + skin and s_min of the pair types (at most 10 atom types)
    for (int p = threadIdx.x; p < M.npairs; p += 32 * NEIGH_WARPS)
        sPair[p] = make_float2((float)(M.pairs[p].smax + NB.skin), (float)M.pairs[p].smin);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int atom = blockIdx.x * (NEIGH_WARPS / nw) + warp / nw;   // nw divides NEIGH_WARPS
    const int w = warp % nw;
    const bool on = atom < NB.n_real;
    int c2 = 0, c3 = 0, c4 = 0;
    const unsigned lt = (1u << lane) - 1u;
    // ---- the atom, the near images and the warp's slice of their chunks
    const int f = on ? frame_of_real(F, atom) : 0;
    const int N = F.natoms[f];
    const int i = on ? atom - (int)F.atom_ofs[f] : 0;
    const int64_t gbase = F.ghost_ofs[f];
    const BoxDev& B = F.box[f];
    const int* typ = F.type + F.atom_ofs[f];
    const int ti = typ[i];
    const float4* c32 = reinterpret_cast<const float4*>(F.cart32) + gbase;
    const float4 ci = c32[i];
    const double* si = F.scaled + 3 * (gbase + i);
    const bool small = B.small != 0;
    const float maxall = (float)fmax(fmax(M.maxcut2, M.order3 > 0 ? M.maxcut3 : 0.0), M.order4 > 0 ? M.maxcut4 : 0.0);
    const float pre = maxall + MARGIN + (float)NB.skin;
    const float cut3 = M.order3 > 0 ? (float)(M.maxcut3 + NB.skin) : -1.0f;
    const float cut4 = M.order4 > 0 ? (float)(M.maxcut4 + NB.skin) : -1.0f;
    const int a0 = small ? 0 : i & ~31;               // ordered lists hold atoms a >= i
    const int per_image = (N - a0 + 31) >> 5;
    // images of the cell's bounding box (wrapped atoms lie in the cell) within reach of atom i
    const float reach = pre + 0.05f;   // float rounding of the images' positions stays far below 0.05 A
    float bmin[3], bmax[3];
    const float hl = lane < 9 ? (float)B.h[lane] : 0.0f;
    const float mg = frame_margin(B, F.nlayers);
    for (int d = 0; d < 3; ++d) {
        bmin[d] = bmax[d] = 0.0f;
        for (int q = 0; q < 3; ++q) {
            const float h = __shfl_sync(0xffffffffu, hl, 3 * d + q);
            bmin[d] += fminf(h, 0.0f);
            bmax[d] += fmaxf(h, 0.0f);
        }
    }
    const float4 c0 = c32[0];
    unsigned* near = sNear[warp];
    const bool masked = F.nimg <= NEIGH_IMG;
    int nnear = masked ? 0 : F.nimg;
    for (int kb = 0; masked && kb < F.nimg; kb += 32) {
        const int k = kb + lane;
        bool in = false;
        if (k < F.nimg) {
            const float4 ck = c32[(int64_t)k * N];
            const float sh[3] = {ck.x - c0.x, ck.y - c0.y, ck.z - c0.z};
            const float p[3] = {ci.x, ci.y, ci.z};
            float d2 = 0.0f;
            for (int d = 0; d < 3; ++d) {
                const float lo = bmin[d] + sh[d], hi = bmax[d] + sh[d];
                const float e = p[d] < lo ? lo - p[d] : (p[d] > hi ? p[d] - hi : 0.0f);
                d2 += e * e;
            }
            in = d2 <= reach * reach;
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (lane == 0) near[kb >> 5] = m;
        nnear += __popc(m);
    }
    __syncwarp();
    const int total = on ? nnear * per_image : 0;
    const int t0 = (int)((int64_t)total * w / nw), t1 = (int)((int64_t)total * (w + 1) / nw);
    auto next_near = [&](int k) {   // the first near image from k on (one exists)
        if (!masked) return k;
        int wd = k >> 5;
        unsigned m = near[wd] & (0xffffffffu << (k & 31));
        while (m == 0) m = near[++wd];
        return wd * 32 + __ffs(m) - 1;
    };
    auto exact = [&](int g) {
        double rab[3];
        return dist_exact(B.h, si, F.scaled + 3 * (gbase + g), rab);
    };
    // lists of ghost g = k N + a of atom i: bits 0..2
    auto member_of = [&](int g, int a) -> int {
        const float4 cg = c32[g];
        const float dx = cg.x - ci.x, dy = cg.y - ci.y, dz = cg.z - ci.z;
        const float r32 = sqrtf(dx * dx + dy * dy + dz * dz);
        if (!(r32 < pre)) return 0;
        const int pt = M.int_pair_map[ti * M.natmtyp + typ[a]];
        const float smax = sPair[pt].x, smin = sPair[pt].y;
        const bool edge = fabsf(r32 - smax) <= mg || (!NB.md && fabsf(r32 - smin) <= mg) ||
                          fabsf(r32 - cut3) <= mg || fabsf(r32 - cut4) <= mg;
        int fl;
        if (edge) {
            const PairDev& P = M.pairs[pt];
            const double r = exact(g);
            fl = (M.order2 > 0 && r < P.smax + NB.skin && (NB.md || r > P.smin) ? 1 : 0) |
                 (M.order3 > 0 && r < M.maxcut3 + NB.skin ? 2 : 0) | (M.order4 > 0 && r < M.maxcut4 + NB.skin ? 4 : 0);
        } else {
            fl = (M.order2 > 0 && r32 < smax && (NB.md || r32 > smin) ? 1 : 0) | (r32 < cut3 ? 2 : 0) |
                 (r32 < cut4 ? 4 : 0);
        }
        return fl;
    };
    int64_t o2 = 0, o3 = 0, o4 = 0;
    int* hit = sHit[warp];
    uint8_t* lists = sLists[warp];
    auto write = [&](int n) {   // the first n (<= 32) hits: exact distances side by side
        const int g = lane < n ? hit[lane] : 0, fl = lane < n ? lists[lane] : 0;
        const unsigned b2 = __ballot_sync(0xffffffffu, fl & 1);
        const unsigned b3 = __ballot_sync(0xffffffffu, fl & 2);
        const unsigned b4 = __ballot_sync(0xffffffffu, fl & 4);
        if (fl) {
            double rab[3];
            const double r = dist_exact(B.h, si, F.scaled + 3 * (gbase + g), rab);
            if (fl & 1) {
                const int64_t p = o2 + __popc(b2 & lt);
                NB.i2[p] = i; NB.g2[p] = g; NB.pt2[p] = M.int_pair_map[ti * M.natmtyp + typ[g % N]]; NB.r2[p] = r;
                NB.rab2[3 * p] = rab[0]; NB.rab2[3 * p + 1] = rab[1]; NB.rab2[3 * p + 2] = rab[2];
            }
            if (fl & 2) { const int64_t p = o3 + __popc(b3 & lt); NB.g3[p] = g; NB.r3[p] = r; }
            if (fl & 4) { const int64_t p = o4 + __popc(b4 & lt); NB.g4[p] = g; NB.r4[p] = r; }
        }
        o2 += __popc(b2); o3 += __popc(b3); o4 += __popc(b4);
    };
    auto sweep = [&](auto&& each) {   // each(lists, a, k) for every chunk of the slice, all lanes
        if (t0 >= t1) return;
        const int img = t0 / per_image;
        int a = a0 + 32 * (t0 - img * per_image);
        int k = next_near(0);
        for (int n = 0; n < img; ++n) k = next_near(k + 1);
        for (int t = t0; t < t1; ++t) {
            const int al = a + lane, g = k * N + al;
            const bool cand = al < N && (small || al >= i) && g != i;
            each(cand ? member_of(g, al) : 0, al, k);
            a += 32;
            if (a >= N && t + 1 < t1) { a = a0; k = next_near(k + 1); }
        }
    };
    // ---- count (without kept slice counts the fill pass of several warps per atom counts again)
    if (!FILL || (nw > 1 && !NB.slice)) {
        sweep([&](int fl, int, int) {
            c2 += __popc(__ballot_sync(0xffffffffu, fl & 1));
            c3 += __popc(__ballot_sync(0xffffffffu, fl & 2));
            c4 += __popc(__ballot_sync(0xffffffffu, fl & 4));
        });
        if (lane == 0) { sc[0][warp] = c2; sc[1][warp] = c3; sc[2][warp] = c4; }
        if (!FILL && on && NB.slice && lane < 3)
            NB.slice[((int64_t)atom * NEIGH_WARPS + w) * 3 + lane] = lane == 0 ? c2 : (lane == 1 ? c3 : c4);
        __syncthreads();
        if (!FILL) {
            if (on && w == 0 && lane == 0) {
                int t2 = 0, t3 = 0, t4 = 0;
                for (int k = warp; k < warp + nw; ++k) { t2 += sc[0][k]; t3 += sc[1][k]; t4 += sc[2][k]; }
                NB.cnt2[atom] = t2; NB.cnt3[atom] = t3; NB.cnt4[atom] = t4;
            }
            return;
        }
    }
    if (!on) return;
    o2 = NB.ofs2[atom]; o3 = NB.ofs3[atom]; o4 = NB.ofs4[atom];
    if (NB.slice) {
        const int* c = NB.slice + (int64_t)atom * NEIGH_WARPS * 3;
        for (int k = 0; k < w; ++k) { o2 += c[3 * k]; o3 += c[3 * k + 1]; o4 += c[3 * k + 2]; }
    } else {
        for (int k = warp - w; k < warp; ++k) { o2 += sc[0][k]; o3 += sc[1][k]; o4 += sc[2][k]; }
    }
    int pend = 0;
    sweep([&](int fl, int a, int k) {
        const unsigned b = __ballot_sync(0xffffffffu, fl != 0);
        if (fl) {
            const int at = pend + __popc(b & lt);
            hit[at] = k * N + a;
            lists[at] = (uint8_t)fl;
        }
        pend += __popc(b);
        __syncwarp();
        if (pend >= 32) {
            write(32);
            __syncwarp();
            const bool more = lane < pend - 32;
            const int rest = more ? hit[32 + lane] : 0, rest_lists = more ? lists[32 + lane] : 0;
            __syncwarp();
            if (more) { hit[lane] = rest; lists[lane] = (uint8_t)rest_lists; }
            pend -= 32;
            __syncwarp();
        }
    });
    write(pend);
}

// ---------------------------------------------------------------- binned neighbour lists
__device__ __forceinline__ int ghost_frame(const FramesDev& F, int64_t gid) {
    int lo = 0, hi = F.nframes - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (F.ghost_ofs[mid] <= gid) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ int bin_coord(double s, int L, int nb) {
    // s spans [-L, L + 1) over the (2L+1) cell images
    int b = (int)floor((s + L) / (2 * L + 1) * nb);
    return b < 0 ? 0 : (b >= nb ? nb - 1 : b);
}

__device__ __forceinline__ int64_t bin_of(const FramesDev& F, const BinGrid& g, int64_t gid) {
    const double* s = F.scaled + 3 * gid;
    const int L = F.nlayers;
    const int bx = bin_coord(s[0], L, g.nb[0]), by = bin_coord(s[1], L, g.nb[1]), bz = bin_coord(s[2], L, g.nb[2]);
    return g.ofs + ((int64_t)bz * g.nb[1] + by) * g.nb[0] + bx;
}

__global__ void k_bin_count(FramesDev F, int64_t n, Bins B) {
    const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= n) return;
    atomicAdd(B.count + bin_of(F, B.grid[ghost_frame(F, gid)], gid), 1);
}

__global__ void k_bin_fill(FramesDev F, int64_t n, Bins B) {
    const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= n) return;
    const int f = ghost_frame(F, gid);
    const int64_t bin = bin_of(F, B.grid[f], gid);
    const int slot = atomicAdd(B.count + bin, 1);
    B.atoms[B.start[bin] + slot] = (int)(gid - F.ghost_ofs[f]);
}

// One warp per real atom over the ghosts of the 27 bins around it; the per-ghost
// tests are those of k_neigh.
__global__ void __launch_bounds__(256) k_neigh_binned(ModelDev M, FramesDev F, NeighDev NB, Bins BN, int fill) {
    __shared__ float2 sPair[55];   // s_max + skin and s_min of the pair types
    for (int p = threadIdx.x; p < M.npairs; p += blockDim.x)
        sPair[p] = make_float2((float)(M.pairs[p].smax + NB.skin), (float)M.pairs[p].smin);
    __syncthreads();
    const int atom = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (atom >= NB.n_real) return;
    int lo = 0, hi = F.nframes - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (F.atom_ofs[mid] <= atom) lo = mid; else hi = mid - 1;
    }
    const int f = lo;
    const int N = F.natoms[f];
    const int i = atom - (int)F.atom_ofs[f];
    const int64_t gbase = F.ghost_ofs[f];
    const BoxDev& B = F.box[f];
    const int* typ = F.type + F.atom_ofs[f];
    const int ti = typ[i];
    const float4 ci = reinterpret_cast<const float4*>(F.cart32)[gbase + i];
    const double* si = F.scaled + 3 * (gbase + i);
    const float maxall = (float)fmax(fmax(M.maxcut2, M.order3 > 0 ? M.maxcut3 : 0.0), M.order4 > 0 ? M.maxcut4 : 0.0);
    const float pre = maxall + MARGIN + (float)NB.skin;
    const float cut3 = M.order3 > 0 ? (float)(M.maxcut3 + NB.skin) : -1.0f;
    const float cut4 = M.order4 > 0 ? (float)(M.maxcut4 + NB.skin) : -1.0f;
    const float mg = frame_margin(B, F.nlayers);
    const BinGrid g = BN.grid[f];
    const int L = F.nlayers;
    const int cx = bin_coord(si[0], L, g.nb[0]), cy = bin_coord(si[1], L, g.nb[1]), cz = bin_coord(si[2], L, g.nb[2]);
    int64_t o2 = 0, o3 = 0, o4 = 0;
    if (fill) { o2 = NB.ofs2[atom]; o3 = NB.ofs3[atom]; o4 = NB.ofs4[atom]; }
    int c2 = 0, c3 = 0, c4 = 0;
    const unsigned lt = (1u << lane) - 1u;
    for (int dz = -1; dz <= 1; ++dz) {
        const int z = cz + dz;
        if (z < 0 || z >= g.nb[2]) continue;
        for (int dy = -1; dy <= 1; ++dy) {
            const int y = cy + dy;
            if (y < 0 || y >= g.nb[1]) continue;
            for (int dx = -1; dx <= 1; ++dx) {
                const int x = cx + dx;
                if (x < 0 || x >= g.nb[0]) continue;
                const int64_t bin = g.ofs + ((int64_t)z * g.nb[1] + y) * g.nb[0] + x;
                const int64_t b0 = BN.start[bin], b1 = BN.start[bin + 1];
                for (int64_t base = b0; base < b1; base += 32) {
                    const int64_t t = base + lane;
                    bool in2 = false, in3 = false, in4 = false;
                    double r = 0, rab[3] = {0, 0, 0};
                    int pt = 0, gg = -1;
                    if (t < b1) {
                        gg = BN.atoms[t];
                        if (gg != i && (B.small || i <= gg % N)) {
                            const float4 cg = reinterpret_cast<const float4*>(F.cart32)[gbase + gg];
                            const float ddx = cg.x - ci.x, ddy = cg.y - ci.y, ddz = cg.z - ci.z;
                            const float r32 = sqrtf(ddx * ddx + ddy * ddy + ddz * ddz);
                            if (r32 < pre) {
                                pt = M.int_pair_map[ti * M.natmtyp + typ[gg % N]];
                                const float smax = sPair[pt].x, smin = sPair[pt].y;
                                const bool edge = fabsf(r32 - smax) <= mg || (!NB.md && fabsf(r32 - smin) <= mg) ||
                                                  fabsf(r32 - cut3) <= mg || fabsf(r32 - cut4) <= mg;
                                in2 = M.order2 > 0 && r32 < smax && (NB.md || r32 > smin);
                                in3 = r32 < cut3;
                                in4 = r32 < cut4;
                                if (edge || (fill && (in2 || in3 || in4)))
                                    r = dist_exact(B.h, si, F.scaled + 3 * (gbase + gg), rab);
                                if (edge) {
                                    const PairDev& P = M.pairs[pt];
                                    in2 = M.order2 > 0 && r < P.smax + NB.skin && (NB.md || r > P.smin);
                                    in3 = M.order3 > 0 && r < M.maxcut3 + NB.skin;
                                    in4 = M.order4 > 0 && r < M.maxcut4 + NB.skin;
                                }
                            }
                        }
                    }
                    const unsigned b2 = __ballot_sync(0xffffffffu, in2);
                    const unsigned b3 = __ballot_sync(0xffffffffu, in3);
                    const unsigned b4 = __ballot_sync(0xffffffffu, in4);
                    if (fill) {
                        if (in2) {
                            const int64_t p = o2 + c2 + __popc(b2 & lt);
                            NB.i2[p] = i; NB.g2[p] = gg; NB.pt2[p] = pt; NB.r2[p] = r;
                            NB.rab2[3 * p] = rab[0]; NB.rab2[3 * p + 1] = rab[1]; NB.rab2[3 * p + 2] = rab[2];
                        }
                        if (in3) { const int64_t p = o3 + c3 + __popc(b3 & lt); NB.g3[p] = gg; NB.r3[p] = r; }
                        if (in4) { const int64_t p = o4 + c4 + __popc(b4 & lt); NB.g4[p] = gg; NB.r4[p] = r; }
                    }
                    c2 += __popc(b2); c3 += __popc(b3); c4 += __popc(b4);
                }
            }
        }
    }
    if (!fill && lane == 0) { NB.cnt2[atom] = c2; NB.cnt3[atom] = c3; NB.cnt4[atom] = c4; }
}

// ---------------------------------------------------------------- clusters
__device__ __forceinline__ float dist32(const float4* c, int64_t a, int64_t b) {
    float4 x = c[a], y = c[b];
    float dx = y.x - x.x, dy = y.y - x.y, dz = y.z - x.z;
    return sqrtf(dx * dx + dy * dy + dz * dz);
}

// r(a,b) < the cut-off decided exactly; FP32 settles all but the near-boundary cases.
__device__ __forceinline__ bool within(const FramesDev& F, const BoxDev& B, int64_t gbase, int a, int b,
                                       const CutDev& C, float r32, float mg) {
    if (r32 < C.cutf - mg) return true;
    if (r32 > C.cutf + mg) return false;
    double rab[3];
    double r = dist_exact(B.h, F.scaled + 3 * (gbase + a), F.scaled + 3 * (gbase + b), rab);
    return r < C.cut;
}

// Triplets: every pair of an atom's neighbours, 32 at a time.
__global__ void k_triplets(ModelDev M, FramesDev F, NeighDev NB, ClusterSet CS, int fill, int parts) {
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int warp = gw / parts, part = gw - warp * parts;
    if (warp >= NB.n_real) return;
    int lo = 0, hi = F.nframes - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (F.atom_ofs[mid] <= warp) lo = mid; else hi = mid - 1;
    }
    const int f = lo;
    const int N = F.natoms[f];
    const int i = warp - (int)F.atom_ofs[f];
    const int64_t gbase = F.ghost_ofs[f];
    const BoxDev& B = F.box[f];
    const int* typ = F.type + F.atom_ofs[f];
    const float4* c32 = reinterpret_cast<const float4*>(F.cart32);
    const int* lg = NB.g3 + NB.ofs3[warp];
    const double* lr = NB.r3 + NB.ofs3[warp];
    const int n = NB.cnt3[warp];
    const float mg = frame_margin(B, F.nlayers);
    const bool ordered = !B.small;
    const int ti = typ[i];
    int64_t out = fill ? CS.ofs[warp] : 0;
    if (fill)
        for (int q = 0; q < part; ++q) out += CS.pcnt[(int64_t)warp * parts + q];
    int count = 0;
    const int64_t total = (int64_t)n * n;
    const int64_t nbat = (total + 31) / 32;
    const int64_t b0 = nbat * part / parts * 32, b1 = min(total, nbat * (part + 1) / parts * 32);
    for (int64_t base = b0; base < b1; base += 32) {
        const int64_t t = base + lane;
        bool ok = false;
        int j = -1, k = -1, T = -1;
        if (t < total) {
            const int a = n <= 65535 ? (int)((unsigned)t / (unsigned)n) : (int)(t / n), b = (int)(t - (int64_t)a * n);
            j = lg[a]; k = lg[b];
            ok = (j != k) && !(ordered && (j % N) > (k % N));
            if (ok) {
                const int id = (ti + 1) + 10 * (typ[j % N] + 1) + 100 * (typ[k % N] + 1);
                T = M.int_map3[id];
                ok = T >= 0;
                if (ok) {
                    const CutDev* C = NB.cut3 + T * 3;
                    const int8_t* pm = M.pidx3 + id * 3;
                    ok = less_pos(lr[a], C[pm[0]].cut) && less_pos(lr[b], C[pm[1]].cut) &&
                         within(F, B, gbase, j, k, C[pm[2]], dist32(c32, gbase + j, gbase + k), mg);
                }
            }
        }
        const unsigned bal = __ballot_sync(0xffffffffu, ok);
        if (fill && ok) {
            int64_t p = out + count + __popc(bal & ((1u << lane) - 1u));
            CS.m[p] = make_int4(i, j, k, -1);
            CS.type[p] = T;
        }
        count += __popc(bal);
    }
    if (!fill && lane == 0) {
        if (parts == 1) {
            CS.cnt[warp] = count;
        } else {
            CS.pcnt[(int64_t)warp * parts + part] = count;
            atomicAdd(CS.cnt + warp, count);
        }
    }
}

// Quadruplets in two stages (every l against every pair, in a
// fixed order): the lanes first test (j, k) pairs -- distinct, parent-ordered, r_jk under
// the largest 4-body cut-off -- and the surviving pairs of each chunk of 32 are then
// crossed with every l, flattened over the lanes, with the full per-slot tests.
__global__ void k_quads(ModelDev M, FramesDev F, NeighDev NB, ClusterSet CS, int fill, int parts) {
    __shared__ int2 sPair[8][32];
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int wib = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int warp = gw / parts, part = gw - warp * parts;
    if (warp >= NB.n_real) return;
    int lo = 0, hi = F.nframes - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (F.atom_ofs[mid] <= warp) lo = mid; else hi = mid - 1;
    }
    const int f = lo;
    const int N = F.natoms[f];
    const int i = warp - (int)F.atom_ofs[f];
    const int64_t gbase = F.ghost_ofs[f];
    const BoxDev& B = F.box[f];
    const int* typ = F.type + F.atom_ofs[f];
    const float4* c32 = reinterpret_cast<const float4*>(F.cart32);
    const int* lg = NB.g4 + NB.ofs4[warp];
    const double* lr = NB.r4 + NB.ofs4[warp];
    const int n = NB.cnt4[warp];
    const bool ordered = !B.small;
    const int ti = typ[i];
    const float cut = (float)(M.maxcut4 + NB.skin) + MARGIN;
    const float mg = frame_margin(B, F.nlayers);
    int64_t out = fill ? CS.ofs[warp] : 0;
    if (fill)
        for (int q = 0; q < part; ++q) out += CS.pcnt[(int64_t)warp * parts + q];
    int count = 0;
    const int npairs = n * n;
    const unsigned lt = (1u << lane) - 1u;
    const int nbat = (npairs + 31) / 32;
    const int pb0 = nbat * part / parts * 32, pb1 = min(npairs, nbat * (part + 1) / parts * 32);
    for (int pb = pb0; pb < pb1; pb += 32) {
        const int p = pb + lane;
        bool pv = false;
        int a = 0, b = 0;
        if (p < npairs) {
            a = p / n; b = p - a * n;
            const int j = lg[a], k = lg[b];
            pv = (j != k) && !(ordered && (j % N) > (k % N)) && dist32(c32, gbase + j, gbase + k) < cut;
        }
        const unsigned pbal = __ballot_sync(0xffffffffu, pv);
        if (pv) sPair[wib][__popc(pbal & lt)] = make_int2(a, b);
        __syncwarp();
        const int work = __popc(pbal) * n;
        for (int tb = 0; tb < work; tb += 32) {
            const int t = tb + lane;
            bool ok = false;
            int j = -1, k = -1, l = -1, T = -1;
            if (t < work) {
                const int pi = t / n, c = t - pi * n;
                const int2 ab = sPair[wib][pi];
                j = lg[ab.x]; k = lg[ab.y]; l = lg[c];
                ok = (j != l) && (k != l) && !(ordered && (k % N) > (l % N));
                if (ok) {
                    const int id = (ti + 1) + 10 * (typ[j % N] + 1) + 100 * (typ[k % N] + 1) + 1000 * (typ[l % N] + 1);
                    T = M.int_map4[id];
                    ok = T >= 0;
                    if (ok) {
                        const CutDev* C = NB.cut4 + T * 6;
                        const int8_t* pm = M.pidx4 + id * 6;
                        ok = less_pos(lr[ab.x], C[pm[0]].cut) && less_pos(lr[ab.y], C[pm[1]].cut) &&
                             less_pos(lr[c], C[pm[2]].cut) &&
                             within(F, B, gbase, j, k, C[pm[3]], dist32(c32, gbase + j, gbase + k), mg) &&
                             within(F, B, gbase, j, l, C[pm[4]], dist32(c32, gbase + j, gbase + l), mg) &&
                             within(F, B, gbase, k, l, C[pm[5]], dist32(c32, gbase + k, gbase + l), mg);
                    }
                }
            }
            const unsigned bal = __ballot_sync(0xffffffffu, ok);
            if (fill && ok) {
                const int64_t q = out + count + __popc(bal & lt);
                CS.m[q] = make_int4(i, j, k, l);
                CS.type[q] = T;
            }
            count += __popc(bal);
        }
        __syncwarp();
    }
    if (!fill && lane == 0) {
        if (parts == 1) {
            CS.cnt[warp] = count;
        } else {
            CS.pcnt[(int64_t)warp * parts + part] = count;
            atomicAdd(CS.cnt + warp, count);
        }
    }
}

// ---------------------------------------------------------------- bucketing
// Stable counting sort of one frame's items by key, one cluster of up to 8 CTAs per frame.
// The items are split into contiguous ranges, one per warp (as many warps as the per-warp
// key counts fit in shared memory); each warp counts the keys of its range, a scan over the
// cluster's counts (distributed shared memory) gives a start for every (key, warp), and
// each warp then places its range in order, ranking equal keys with __match_any_sync.
// Within a key the items keep their order, so the result depends neither on timing nor on
// the number of CTAs.  A warp's chain of loads and ranks bounds it (32 items a step), so
// warps are what helps: 8 frames of 33 to 1,001 atoms, five sorts, one CTA a frame -> a
// cluster: 919 -> 141 us.
constexpr int BUCKET_THREADS = 512;
constexpr int BUCKET_SMEM_INTS = 24576;   // per-warp key counts + key totals (96 KB)
constexpr int BUCKET_U = 4;               // items in flight per lane

// t < nunits * members of the frame: the values are ints, so 32 bits hold it
__device__ __forceinline__ void bucket_item(const BucketSpec& S, int N, int64_t base, unsigned t, int& key, int& val) {
    if (S.kind == 0) {
        const int64_t p = base + (t >> 1);
        key = (t & 1u) == 0 ? S.i2[p] : S.g2[p] % N;
        val = (int)t;
    } else if (S.kind == 1) {
        const unsigned q = S.nb == 3 ? t / 3u : t / 4u;
        const unsigned e = t - q * (unsigned)S.nb;
        key = reinterpret_cast<const int*>(S.m + base + q)[e] % N;
        val = (int)(q * 4u + e);
    } else {
        key = S.type[base + t];
        val = (int)t;
    }
}

__global__ void __launch_bounds__(BUCKET_THREADS, 2) k_bucket(FramesDev F, BucketSpec S, Buckets out) {
    extern __shared__ int bsm[];
    __shared__ int part[BUCKET_THREADS / 32];
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int f = blockIdx.x / C;
    const int N = F.natoms[f];
    // pair items live in the neighbour CSR, which is indexed by global real atom
    const int64_t base = S.item_frame_ofs[f];
    const int64_t nunits = S.item_frame_ofs[f + 1] - base;
    const int mult = S.kind == 0 ? 2 : (S.kind == 1 ? S.nb : 1);
    const int64_t nitems = nunits * mult;
    const int64_t kbase = S.key_frame_ofs[f];
    const int K = (int)(S.key_frame_ofs[f + 1] - kbase - 1);
    const int64_t vbase = base * mult;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int W = max(1, min((int)(blockDim.x >> 5), (BUCKET_SMEM_INTS - K) / max(K, 1)));
    int* cntw = bsm;            // [W][K]: counts, then starts
    int* tot = bsm + W * K;     // [K]: this CTA's totals, read by the cluster
    for (int k = threadIdx.x; k < W * K; k += blockDim.x) cntw[k] = 0;
    __syncthreads();
    const int64_t chunk = (nitems + W * C - 1) / (W * C);
    const int64_t r0 = min(nitems, (int64_t)(rank * W + warp) * chunk), r1 = min(nitems, r0 + chunk);
    int* cnt = cntw + warp * K;
    // the next BUCKET_U x 32 items from c0 on; items past the range get a key of their own
    auto load = [&](int64_t c0, int (&key)[BUCKET_U], int (&val)[BUCKET_U]) {
#pragma unroll
        for (int u = 0; u < BUCKET_U; ++u) {
            const int64_t t = c0 + 32 * u + lane;
            key[u] = -1 - lane;
            val[u] = 0;
            if (t < r1) bucket_item(S, N, base, (unsigned)t, key[u], val[u]);
        }
    };
    if (warp < W) {
        for (int64_t c0 = r0; c0 < r1; c0 += 32 * BUCKET_U) {
            int key[BUCKET_U], val[BUCKET_U];
            load(c0, key, val);
#pragma unroll
            for (int u = 0; u < BUCKET_U; ++u) if (key[u] >= 0) atomicAdd(&cnt[key[u]], 1);
        }
    }
    __syncthreads();
    // per key: starts of each warp's share relative to the CTA's, and the CTA's total
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
        int run = 0;
        for (int w = 0; w < W; ++w) { const int v = cntw[w * K + k]; cntw[w * K + k] = run; run += v; }
        tot[k] = run;
    }
    cl.sync();
    // exclusive scan of the key totals, by every CTA for itself
    const int per = (K + blockDim.x - 1) / blockDim.x;
    const int k0 = min(K, (int)threadIdx.x * per), k1 = min(K, k0 + per);
    auto totals = [&](int k, int& low) {   // key k's total, and the share of the CTAs before this one
        int t = 0;
        low = 0;
        for (int c = 0; c < C; ++c) {
            const int v = *cl.map_shared_rank(tot + k, c);
            if (c < rank) low += v;
            t += v;
        }
        return t;
    };
    int local = 0, low;
    for (int k = k0; k < k1; ++k) local += totals(k, low);
    int incl = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) part[warp] = incl;
    __syncthreads();
    int run = incl - local;
    for (int w = 0; w < warp; ++w) run += part[w];
    for (int k = k0; k < k1; ++k) {
        const int t = totals(k, low);
        for (int w = 0; w < W; ++w) cntw[w * K + k] += run + low;
        if (rank == 0) out.key_ofs[kbase + k] = vbase + run;
        run += t;
    }
    if (rank == 0 && threadIdx.x == 0) out.key_ofs[kbase + K] = vbase + nitems;
    cl.sync();   // the others have read this CTA's totals; its starts are in place
    if (warp < W) {
        for (int64_t c0 = r0; c0 < r1; c0 += 32 * BUCKET_U) {
            int key[BUCKET_U], val[BUCKET_U];
            load(c0, key, val);
#pragma unroll
            for (int u = 0; u < BUCKET_U; ++u) {
                const unsigned peers = __match_any_sync(0xffffffffu, key[u]);
                const int leader = __ffs(peers) - 1;
                int start = 0;
                if (key[u] >= 0 && lane == leader) {
                    start = cnt[key[u]];
                    cnt[key[u]] = start + __popc(peers);
                }
                start = __shfl_sync(0xffffffffu, start, leader);
                if (key[u] >= 0) out.val[vbase + start + __popc(peers & ((1u << lane) - 1u))] = val[u];
                __syncwarp();   // the next 32 items' leaders see the new starts
            }
        }
    }
}

// ---------------------------------------------------------------- launchers
void launch_frame_setup(const FramesDev& F, int64_t n, cudaStream_t st) {
    if (n > 0) k_frame_setup<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(F, n);
}
void launch_neigh(const ModelDev& M, const FramesDev& F, const NeighDev& NB, int fill, cudaStream_t st) {
    if (NB.n_real <= 0) return;
    // eight warps on an atom of a small batch, one where the atoms alone fill the GPU several
    // times over (frames differ in size: a warp per atom of 2,600 runs 40 times as long as one
    // of 64): 4,076 atoms in frames of 64 to 2,600, count and fill 423 -> 164 us.  Where the
    // fill pass has to count again, no more warps than fill the GPU once.
    int nw = NEIGH_WARPS;
    const int64_t most = NB.slice ? 16 * 2432 : 2 * 2432;
    while (nw > 1 && (int64_t)NB.n_real * nw > most) nw >>= 1;
    const unsigned blocks = (unsigned)((NB.n_real + NEIGH_WARPS / nw - 1) / (NEIGH_WARPS / nw));
    if (fill) k_neigh<true><<<blocks, 32 * NEIGH_WARPS, 0, st>>>(M, F, NB, nw);
    else k_neigh<false><<<blocks, 32 * NEIGH_WARPS, 0, st>>>(M, F, NB, nw);
}
void launch_bins(const FramesDev& F, int64_t n, const Bins& B, cudaStream_t st) {
    if (n <= 0) return;
    cudaMemsetAsync(B.count, 0, sizeof(int) * B.nbins, st);
    k_bin_count<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(F, n, B);
    launch_scan_counts(B.count, (int)B.nbins, B.start, st);
    cudaMemsetAsync(B.count, 0, sizeof(int) * B.nbins, st);
    k_bin_fill<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(F, n, B);
}

void launch_neigh_binned(const ModelDev& M, const FramesDev& F, const NeighDev& NB, const Bins& B, int fill,
                         cudaStream_t st) {
    if (NB.n_real > 0) k_neigh_binned<<<(unsigned)((NB.n_real + 7) / 8), 256, 0, st>>>(M, F, NB, B, fill);
}

int cluster_parts(int n_real) {
    return n_real >= 32768 ? 1 : n_real >= 16384 ? 2 : n_real >= 8192 ? 4 : 8;
}

void launch_clusters(int nbody, const ModelDev& M, const FramesDev& F, const NeighDev& NB, const ClusterSet& CS,
                     int fill, cudaStream_t st) {
    if (NB.n_real <= 0) return;
    const int parts = CS.pcnt ? cluster_parts(NB.n_real) : 1;
    if (parts > 1 && !fill) cudaMemsetAsync(CS.cnt, 0, sizeof(int) * NB.n_real, st);
    const unsigned g = (unsigned)(((int64_t)NB.n_real * parts + 7) / 8);
    if (nbody == 3) k_triplets<<<g, 256, 0, st>>>(M, F, NB, CS, fill, parts);
    else k_quads<<<g, 256, 0, st>>>(M, F, NB, CS, fill, parts);
}
void launch_bucket(int nframes, const FramesDev& F, const BucketSpec& S, const Buckets& out, cudaStream_t st) {
    if (nframes <= 0) return;
    const int smem = BUCKET_SMEM_INTS * (int)sizeof(int);
    cudaFuncSetAttribute(k_bucket, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // two CTAs fit on an SM: no more than the GPU takes at once (with 8 frames, 8 CTAs each are
    // 6.5x as fast as one; 16 would need the non-portable cluster size)
    unsigned c = 8;
    while (c > 1 && (int64_t)nframes * c > 2 * sms) c >>= 1;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = c;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)nframes * c);
    cfg.blockDim = dim3(BUCKET_THREADS);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_bucket, F, S, out);
}

}  // namespace cgd
