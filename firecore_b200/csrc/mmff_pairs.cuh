// mmff_pairs.cuh -- the pair term of one system in 32 x 32 tiles: every unordered
// pair of the central image once, the shifted images from candidate lists as
// tiles or ordered rows.  Shared by the evaluation kernels (mmff_eval.cu) and the
// relaxation kernels (mmff_relax.cu).
#pragma once
#include "mmff_engine.cuh"

namespace mmff {

// T threads, S lanes per atom on the ordered rows; ENERGY: pair energies too;
// COUNT: counts the pair-images; TILES: long candidate lists as tiles (else rows only)
template <int T, int S, bool ENERGY, bool COUNT = false, bool TILES = (T >= kImageTileMinThreads), int G = 1>
struct PairEngine : CtaSystem<T, G> {
    static_assert(32 % S == 0, "bad tile");
    using B = CtaSystem<T, G>;
    using B::P; using B::Y; using B::L; using B::sm; using B::tid; using B::lane; using B::warp;
    using B::natoms; using B::lv; using B::hasH; using B::xrow; using B::nbw;
    using B::ngs; using B::ngc; using B::fix_add;
    template <class X> __device__ __forceinline__ X* at(int off) { return B::template at<X>(off); }
    unsigned long long npair = 0;      // COUNT: pair-images evaluated by this thread

    __device__ PairEngine(const Params& p, const Systems& y, char* smem, const SmemLayout& l) : B(p, y, smem, l) {}

    // pair sum of one atom (already shifted by the image) over j = sub, sub+S, ...
    // Branch-free: excluded and out-of-range pairs get r^2 = 1e30, where every
    // term underflows to zero except the shifted-force constant kq Q / r
    // (< 1e-16 eV/A).  HB: the system has H-bond pseudo-charges (block-uniform).
    // list (nullable): candidate atoms of a shifted image, ascending; else all atoms
    template <bool HB>
    __device__ __forceinline__ void pair_row(const float4* spos, const float4* sREQ, int sub, float4 Ri, float pxs,
                                             float pys, float pzs, int e0, int e1, int e2, int e3, int e4,
                                             const unsigned short* list, int ncand,
                                             float& fx, float& fy, float& fz, float& ei) {
        const bool CUT = P.Rc2 > 0.f;
        const float Rc2 = CUT ? P.Rc2 : 3.0e38f, kq = P.kq_rc2;
        const float rc = CUT ? sqrtf(1.f / kq) : 0.f;
        const int n = list ? ncand : natoms;
        for (int c = sub; c < n; c += S) {
            const int j = list ? (int)list[c] : c;
            const float4 pj = spos[j];
            const float4 Rj = sREQ[j];
            const float dx = pj.x - pxs, dy = pj.y - pys, dz = pj.z - pzs;
            float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            const bool ex = (j == e0) | (j == e1) | (j == e2) | (j == e3) | (j == e4);
            const bool ok = !ex && (r2 < Rc2);
            if (COUNT && ok) npair++;
            r2 = ok ? r2 : 1e30f;
            const float ir = rsq(r2);
            const float ir2 = ir * ir;
            const float R0 = Ri.x + Rj.x;
            const float E0 = Ri.y * Rj.y;
            const float Q = Ri.z * Rj.z;
            const float Eel = Q * ir;
            const float u2 = R0 * R0 * ir2;
            const float u6 = u2 * u2 * u2;
            const float vdW = u6 * E0;
            const float H = HB ? u6 * vdW * fminf(Ri.w * Rj.w, 0.f) : 0.f;
            float F = -fmaf(12.f * ir2, HB ? fmaf(u6 - 1.f, vdW, H) : (u6 - 1.f) * vdW, Eel * ir2);
            F = fmaf(Q * kq, ir, F);
            fx = fmaf(dx, F, fx); fy = fmaf(dy, F, fy); fz = fmaf(dz, F, fz);
            if (ENERGY && ok) {
                float e = fmaf(u6 - 2.f, vdW, Eel + H);
                if (CUT) e += Q * kq * (r2 * ir - 2.f * rc);
                ei += e;
            }
        }
    }

    // atom i (lane sub of its S) against image (ix,iy,iz) of the atoms in list
    // (all atoms if list is null): the exclusions of NBFF::evalLJQs_ng4_PBC_atom
    // (NBFF.h:590-607): i itself, and its bonded neighbours whose cell is ipbc
    __device__ __forceinline__ void pair_image_row(const float4* spos, const float4* sREQ, int i, int sub, float4 pi,
                                                   float4 Ri, int4 ng, int4 ngC, bool pbc, int ipbc, int ix, int iy,
                                                   int iz, const unsigned short* list, int ncand, float& fx, float& fy,
                                                   float& fz, float& ei) {
        const float3 sh = image_shift(lv, ix, iy, iz);
        const float pxs = pi.x - sh.x, pys = pi.y - sh.y, pzs = pi.z - sh.z;
        const int e0 = i;
        const int e1 = (ngC.x == ipbc || !pbc) ? ng.x : -1;
        const int e2 = (ngC.y == ipbc || !pbc) ? ng.y : -1;
        const int e3 = (ngC.z == ipbc || !pbc) ? ng.z : -1;
        const int e4 = (ngC.w == ipbc || !pbc) ? ng.w : -1;
        if (hasH) pair_row<true>(spos, sREQ, sub, Ri, pxs, pys, pzs, e0, e1, e2, e3, e4, list, ncand, fx, fy, fz, ei);
        else pair_row<false>(spos, sREQ, sub, Ri, pxs, pys, pzs, e0, e1, e2, e3, e4, list, ncand, fx, fy, fz, ei);
    }

    // ---- central image, each unordered pair once (Newton's third law) --------
    // 32 x 32 atom tiles: the 32 lanes of a warp own the atoms i of block bi,
    // the atoms j of block bj rotate through the lanes (lane l meets j-slot
    // l + s at step s) and so does the reaction accumulator of the current j,
    // which after 32 steps sits in lane j - 32 bj.  Diagonal tiles take steps
    // 1..16 (s = 16 on lanes < 16 only) and return reactions by shuffle.  Tile
    // sums reach the per-atom totals through 64-bit fixed-point shared-memory
    // adds (2^-32 eV/A resolution): integer addition is associative, so the
    // totals do not depend on which warp finishes first.
#ifndef MMFF_TILE_UNROLL_SMALL
#define MMFF_TILE_UNROLL_SMALL 1
#endif
#ifndef MMFF_TILE_UNROLL_LARGE
#define MMFF_TILE_UNROLL_LARGE 4
#endif
    // tile-step unrolling (build options): none in blocks below
    // MMFF_UNROLL_MIN_T threads, whose fused step is instruction-fetch bound
    // (unrolling by 4 measured -6 % at 64 threads), 4 in the larger blocks
    // (+4.7 %)
    static constexpr int kTileUnroll = T >= MMFF_UNROLL_MIN_T ? MMFF_TILE_UNROLL_LARGE : MMFF_TILE_UNROLL_SMALL;
    // own atom i of a tile: position and parameters; invalid slots exclude everything
    struct TileAtom { float4 p, R; int i; bool v; };
    __device__ __forceinline__ TileAtom tile_atom(int i, const float4* spos, const float4* sREQ) {
        TileAtom t;
        t.v = i < natoms;
        t.i = t.v ? i : 0;
        t.p = spos[t.i]; t.R = sREQ[t.i];
        return t;
    }

    // excluded j-slots of block bj for this lane's atom (the host-built
    // exclusion row: the atom itself, its bonded neighbours in the central
    // cell, the 1-3 pairs the angle terms account for, padding slots of bj);
    // all if the atom is a padding slot
    __device__ __forceinline__ uint32_t tile_mask(const TileAtom& a, int bj) const {
        return a.v ? __ldg(xrow + a.i * nbw + bj) : ~0u;
    }

    template <bool HB>
    __device__ void off_tile(int bi, int bj, const float4* spos, const float4* sREQ, bool pbc, int central,
                             long long* facc, float& ec) {
        const bool CUT = P.Rc2 > 0.f;
        const float Rc2 = CUT ? P.Rc2 : 3.0e38f, kq = P.kq_rc2;
        const float rc = CUT ? sqrtf(1.f / kq) : 0.f;
        const int i = bi * 32 + lane;
        const TileAtom a = tile_atom(i, spos, sREQ);
        const uint32_t xm = tile_mask(a, bj);
        float3 fi = make_float3(0.f, 0.f, 0.f), rj = make_float3(0.f, 0.f, 0.f);
        bool ok;
        float e = 0.f;
#pragma unroll kTileUnroll
        for (int s = 0; s < 32; s++) {
            const int jl = (lane + s) & 31;
            const int j = bj * 32 + jl;
            const int jc = min(j, natoms - 1);
            const float4 pj = spos[jc], Rj = sREQ[jc];
            const bool excl = (xm >> jl) & 1u;
            const float dx = pj.x - a.p.x, dy = pj.y - a.p.y, dz = pj.z - a.p.z;
            const float F = pair_force<ENERGY, HB>(dx, dy, dz, a.R, Rj, excl, Rc2, kq, rc, CUT, ok, e);
            fi.x = fmaf(dx, F, fi.x); fi.y = fmaf(dy, F, fi.y); fi.z = fmaf(dz, F, fi.z);
            rj.x = fmaf(-dx, F, rj.x); rj.y = fmaf(-dy, F, rj.y); rj.z = fmaf(-dz, F, rj.z);
            if (ENERGY) ec += e;
            if (COUNT && ok) npair += 2;
            const int nxt = (lane + 1) & 31;
            rj.x = __shfl_sync(0xffffffffu, rj.x, nxt);
            rj.y = __shfl_sync(0xffffffffu, rj.y, nxt);
            rj.z = __shfl_sync(0xffffffffu, rj.z, nxt);
        }
        if (a.v) fix_add(facc + 3 * i, fi);
        const int jo = bj * 32 + lane;
        if (jo < natoms) fix_add(facc + 3 * jo, rj);
    }

    template <bool HB>
    __device__ void diag_tile(int b, const float4* spos, const float4* sREQ, bool pbc, int central, long long* facc,
                              float& ec) {
        const bool CUT = P.Rc2 > 0.f;
        const float Rc2 = CUT ? P.Rc2 : 3.0e38f, kq = P.kq_rc2;
        const float rc = CUT ? sqrtf(1.f / kq) : 0.f;
        const int i = b * 32 + lane;
        const TileAtom a = tile_atom(i, spos, sREQ);
        const uint32_t xm = tile_mask(a, b);
        float3 fi = make_float3(0.f, 0.f, 0.f);
        bool ok;
        float e = 0.f;
#pragma unroll kTileUnroll
        for (int s = 1; s <= 16; s++) {
            const int jl = (lane + s) & 31;
            const int jc = min(b * 32 + jl, natoms - 1);
            const float4 pj = spos[jc], Rj = sREQ[jc];
            const bool excl = ((xm >> jl) & 1u) || (s == 16 && lane >= 16);
            const float dx = pj.x - a.p.x, dy = pj.y - a.p.y, dz = pj.z - a.p.z;
            const float F = pair_force<ENERGY, HB>(dx, dy, dz, a.R, Rj, excl, Rc2, kq, rc, CUT, ok, e);
            fi.x = fmaf(dx, F, fi.x); fi.y = fmaf(dy, F, fi.y); fi.z = fmaf(dz, F, fi.z);
            if (ENERGY) ec += e;
            if (COUNT && ok) npair += 2;
            const int src = (lane - s) & 31;     // the lane whose partner this lane's atom was
            fi.x += __shfl_sync(0xffffffffu, -dx * F, src);
            fi.y += __shfl_sync(0xffffffffu, -dy * F, src);
            fi.z += __shfl_sync(0xffffffffu, -dz * F, src);
        }
        if (a.v) fix_add(facc + 3 * i, fi);
    }

    // position of atom e in the candidate list of image k, or -1
    __device__ __forceinline__ int cand_slot(int k, int e) {
        if (e < 0) return -1;
        const int w = k * L.nwords + (e >> 5);
        const uint32_t m = at<uint32_t>(L.cwords)[w];
        if (!((m >> (e & 31)) & 1u)) return -1;
        return at<int>(L.cpref)[w] + __popc(m & ((1u << (e & 31)) - 1u));
    }

    // ---- shifted images, each unordered image pair once -----------------------
    // Atom i meets image +k of atom j exactly when atom j meets image -k of
    // atom i, with the opposite force.  So for long candidate lists only the
    // images k < nimg / 2 are visited (image nimg-1-k is the mirror of k), as
    // 32 x 32 tiles of (candidates i of image -k) x (candidates j of image +k),
    // each pair once, the reaction on j rotating through the lanes as in
    // off_tile.  Excluded (NBFF::evalLJQs_ng4_PBC_atom, NBFF.h:590-607): i
    // itself, and the bonded neighbours of i whose cell is this image; both
    // are symmetric under the mirror.  k: image index without the central
    // one (iz, iy, ix order).
    template <bool HB>
    __device__ void image_tile(int k, int ti, int tj, const float4* spos, const float4* sREQ, long long* facc,
                               float& ec) {
        const bool CUT = P.Rc2 > 0.f;
        const float Rc2 = CUT ? P.Rc2 : 3.0e38f, kq = P.kq_rc2;
        const float rc = CUT ? sqrtf(1.f / kq) : 0.f;
        const int nxi = 2 * P.npbc[0] + 1, nyi = 2 * P.npbc[1] + 1;
        const int ipbc = k;                                   // k < central: same index with the central one
        const int ix = ipbc % nxi - P.npbc[0], iy = (ipbc / nxi) % nyi - P.npbc[1], iz = ipbc / (nxi * nyi) - P.npbc[2];
        const int kI = L.nimg - 1 - k;
        const unsigned short* Il = at<unsigned short>(L.clist) + kI * L.maxNA;
        const unsigned short* Jl = at<unsigned short>(L.clist) + k * L.maxNA;
        const int nI = at<int>(L.ccnt)[kI], nJ = at<int>(L.ccnt)[k];
        const int ci = 32 * ti + lane;
        const bool vi = ci < nI;
        const int i = vi ? (int)Il[ci] : 0;
        const float3 sh = image_shift(lv, ix, iy, iz);
        float4 pi = spos[i];
        pi.x -= sh.x; pi.y -= sh.y; pi.z -= sh.z;
        const float4 Ri = sREQ[i];
        // excluded j-slots of this tile
        const int j0 = 32 * tj;
        uint32_t xm = ~0u;
        if (vi) {
            const int nvalid = nJ - j0;
            xm = nvalid >= 32 ? 0u : ~((1u << nvalid) - 1u);
            const int4 ng = ngs(i), ngC = ngc(i);
            const int e[5] = {i, ngC.x == ipbc ? ng.x : -1, ngC.y == ipbc ? ng.y : -1, ngC.z == ipbc ? ng.z : -1,
                              ngC.w == ipbc ? ng.w : -1};
#pragma unroll
            for (int q = 0; q < 5; q++) {
                const int d = cand_slot(k, e[q]) - j0;
                if (d >= 0 && d < 32) xm |= 1u << d;
            }
        }
        float3 fi = make_float3(0.f, 0.f, 0.f), rj = make_float3(0.f, 0.f, 0.f);
        bool ok;
        float e = 0.f;
        const int jlast = nJ - 1;
        // the tile's 32 candidates j into this warp's staging slots (one
        // indirect load per lane instead of one per rotation step)
        float4* stg = at<float4>(L.stage) + 64 * warp;
        {
            const int jj = Jl[min(j0 + lane, jlast)];
            stg[lane] = spos[jj];
            stg[32 + lane] = sREQ[jj];
        }
        __syncwarp();
#pragma unroll kTileUnroll
        for (int s = 0; s < 32; s++) {
            const int jl = (lane + s) & 31;
            const float4 pj = stg[jl], Rj = stg[32 + jl];
            const bool excl = (xm >> jl) & 1u;
            const float dx = pj.x - pi.x, dy = pj.y - pi.y, dz = pj.z - pi.z;
            const float F = pair_force<ENERGY, HB>(dx, dy, dz, Ri, Rj, excl, Rc2, kq, rc, CUT, ok, e);
            fi.x = fmaf(dx, F, fi.x); fi.y = fmaf(dy, F, fi.y); fi.z = fmaf(dz, F, fi.z);
            rj.x = fmaf(-dx, F, rj.x); rj.y = fmaf(-dy, F, rj.y); rj.z = fmaf(-dz, F, rj.z);
            if (ENERGY) ec += e;
            if (COUNT && ok) npair += 2;
            const int nxt = (lane + 1) & 31;
            rj.x = __shfl_sync(0xffffffffu, rj.x, nxt);
            rj.y = __shfl_sync(0xffffffffu, rj.y, nxt);
            rj.z = __shfl_sync(0xffffffffu, rj.z, nxt);
        }
        __syncwarp();                                         // staging slots free for the next tile
        if (vi) fix_add(facc + 3 * i, fi);
        if (j0 + lane < nJ) fix_add(facc + 3 * (int)Jl[j0 + lane], rj);
    }

    // mirror pair (k, nimg-1-k): tiles (true) or ordered rows of both images.
    // Cost in pair evaluations: a tile evaluates 32 x 32 pairs at ~1.2 times
    // the cost of an ordered pair (the reaction and its rotation); the rows
    // evaluate the nI x nJ pairs of each image.
    __device__ __forceinline__ bool image_tiled(int nI, int nJ, int& units) const {
        const int nti = (nI + 31) >> 5, ntj = (nJ + 31) >> 5;
        if (TILES && 6 * 1024 * nti * ntj <= 5 * 2 * nI * nJ) { units = nti * ntj; return true; }
        units = 0;
        return false;
    }

    // Shifted images from this step's candidate lists, in tiles: 32 x 32 tiles of
    // the mirror pairs with long lists (their number; all of equal cost, 1024
    // pair evaluations) ...
    __device__ int image_tile_count() const {
        const int* ccnt = reinterpret_cast<const int*>(sm + L.ccnt);
        int total = 0;
        for (int k = 0; k < L.nimg / 2; k++) {
            int n;
            if (image_tiled(ccnt[L.nimg - 1 - k], ccnt[k], n)) total += n;
        }
        return total;
    }
    // ... one of them ...
    template <bool HB>
    __device__ void image_tile_unit(int rem, const float4* spos, const float4* sREQ, long long* facc, float& ec) {
        const int* ccnt = at<int>(L.ccnt);
        int k = 0, n = 0;
        for (;; k++) {
            if (image_tiled(ccnt[L.nimg - 1 - k], ccnt[k], n) && rem < n) break;
            rem -= n;
        }
        const int ntj = (ccnt[k] + 31) >> 5;
        image_tile<HB>(k, rem / ntj, rem % ntj, spos, sREQ, facc, ec);
    }
    // ... and the mirror pairs with short lists as ordered rows of both images, S
    // lanes per candidate atom i (the images that reach a few edge atoms of a small
    // molecule); thread t0 of nt.
    template <bool HB>
    __device__ void image_rows(int t0, int nt, const float4* spos, const float4* sREQ, bool pbc, long long* facc,
                               float& ec) {
        const int* ccnt = at<int>(L.ccnt);
        int nrows = 0;
        for (int k = 0; k < L.nimg / 2; k++) {
            int n;
            if (!image_tiled(ccnt[L.nimg - 1 - k], ccnt[k], n)) nrows += ccnt[L.nimg - 1 - k] + ccnt[k];
        }
        const int nxi = 2 * P.npbc[0] + 1, nyi = 2 * P.npbc[1] + 1;
        const unsigned short* clist = at<unsigned short>(L.clist);
        for (int u0 = 0; u0 < nrows * S; u0 += nt) {
            const int u = u0 + t0;
            int c = u / S;
            const int sub = u % S;
            float fx = 0.f, fy = 0.f, fz = 0.f, ei = 0.f;
            int i = -1;
            if (c < nrows) {
                // row c -> image kk (k, then its mirror) and candidate position
                int kk = -1;
                for (int k = 0; k < L.nimg / 2; k++) {
                    int n;
                    if (image_tiled(ccnt[L.nimg - 1 - k], ccnt[k], n)) continue;
                    const int nI = ccnt[L.nimg - 1 - k], nJ = ccnt[k];
                    if (c < nI) { kk = k; break; }
                    c -= nI;
                    if (c < nJ) { kk = L.nimg - 1 - k; break; }
                    c -= nJ;
                }
                const int ipbc = kk < L.nimg / 2 ? kk : kk + 1;
                const int ix = ipbc % nxi - P.npbc[0], iy = (ipbc / nxi) % nyi - P.npbc[1];
                const int iz = ipbc / (nxi * nyi) - P.npbc[2];
                i = clist[(L.nimg - 1 - kk) * L.maxNA + c];
                pair_image_row(spos, sREQ, i, sub, spos[i], sREQ[i], ngs(i), ngc(i), pbc, ipbc, ix, iy, iz,
                               clist + kk * L.maxNA, ccnt[kk], fx, fy, fz, ei);
            }
#pragma unroll
            for (int o = S / 2; o > 0; o >>= 1) {
                fx += __shfl_xor_sync(0xffffffffu, fx, o);
                fy += __shfl_xor_sync(0xffffffffu, fy, o);
                fz += __shfl_xor_sync(0xffffffffu, fz, o);
            }
            if (i >= 0 && sub == 0) fix_add(facc + 3 * i, make_float3(fx, fy, fz));
            if (ENERGY) ec += 0.5f * ei;
        }
    }

    // LISTS: the candidate lists of this step exist (block-uniform; the
    // central-only form keeps the image code out of the tile loop).
    // Warp units: each off-diagonal tile and pairs of diagonal tiles of the
    // central image, then the image tiles, dealt round-robin to the warps; then the
    // rows.  No barrier anywhere: every sum goes to the fixed-point accumulators.
    template <bool HB, bool LISTS>
    __device__ void pair_tiles(const float4* spos, const float4* sREQ, bool pbc, int central, long long* facc,
                               float& ec) {
        const int B = (natoms + 31) >> 5;
        const int noff = B * (B - 1) / 2;
        const int ncen = noff + ((B + 1) >> 1);
        const int nunits = ncen + (LISTS && TILES ? image_tile_count() : 0);
        for (int u = warp; u < nunits; u += L.nwarps) {
            if (u < noff) {
                int bi = 0, rem = u;
                while (rem >= B - 1 - bi) { rem -= B - 1 - bi; bi++; }
                off_tile<HB>(bi, bi + 1 + rem, spos, sREQ, pbc, central, facc, ec);
            } else if (u < ncen) {
                const int d = 2 * (u - noff);
                diag_tile<HB>(d, spos, sREQ, pbc, central, facc, ec);
                if (d + 1 < B) diag_tile<HB>(d + 1, spos, sREQ, pbc, central, facc, ec);
            } else if (LISTS && TILES) {
                image_tile_unit<HB>(u - ncen, spos, sREQ, facc, ec);
            }
        }
        if (LISTS) image_rows<HB>(tid, T, spos, sREQ, pbc, facc, ec);
    }
};

}  // namespace mmff
