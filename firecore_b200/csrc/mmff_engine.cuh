// mmff_engine.cuh -- one system held by one CTA: what the evaluation kernels
// (mmff_eval.cu) and the relaxation kernels (mmff_relax.cu) share -- loading
// into shared memory, the bounding box and the candidate lists of the shifted
// images, the bonded terms, the GridFF samples and the fixed-point force sums.
#pragma once
#include "mmff_device.cuh"
#include <cfloat>

// blocks of at least this many threads unroll the pair tiles and the GridFF
// columns; smaller ones (four or eight per SM, instruction-fetch bound) do
// not: measured +5-7 % at 64 threads, +1.7 % at 128 threads (C2 class of
// 65-128 atoms), while the 256-thread blocks gain 5 % from unrolling
#ifndef MMFF_UNROLL_MIN_T
#define MMFF_UNROLL_MIN_T 256
#endif

namespace mmff {

// warp-level sums / extrema
__device__ __forceinline__ double wsum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float wmax(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float wmin(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Image shift for cell index (ix, iy, iz)
__device__ __forceinline__ float3 image_shift(const float* lv, int ix, int iy, int iz) {
    return make_float3(lv[0] * ix + lv[3] * iy + lv[6] * iz, lv[1] * ix + lv[4] * iy + lv[7] * iz,
                       lv[2] * ix + lv[5] * iy + lv[8] * iz);
}

// G: systems of a CTA, T threads each, with barriers of their own
template <int T, int G = 1>
struct CtaSystem {
    static_assert(T % 32 == 0, "whole warps");
    static __device__ __forceinline__ int group() { return G == 1 ? 0 : threadIdx.x / T; }
    static __device__ __forceinline__ void sync() {
        if (G == 1) __syncthreads();
        else if (T == 32) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(1 + group()), "n"(T) : "memory");
    }
    static __device__ __forceinline__ bool sync_or(int p) {
        if (G == 1) return __syncthreads_or(p) != 0;
        if (T == 32) return __any_sync(0xffffffffu, p) != 0;
        int r;
        asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.or.pred q, %2, %3, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
                     : "=r"(r) : "r"(p), "r"(1 + group()), "n"(T) : "memory");
        return r != 0;
    }
    const Params& P;
    const Systems& Y;
    const SmemLayout& L;        // kernel parameter: its offsets come from the constant bank
    char* sm;
    int tid, lane, warp;
    // current system
    int isys, natoms, nnode, nvecs, aoff, noff, voff;
    float* lv;                  // shared memory: lattice vectors [9], grid offset of the local frame [3]
    // per-step image culling
    float bbmin[3], bbmax[3];
    bool hasH = false;          // any H-bond pseudo-charge in the system (block-uniform)
    bool hasX = false;          // any bond into a shifted cell (block-uniform)
    const uint32_t* xrow;       // central-image exclusion rows (ceil(natoms/32) words per atom)
    int nbw;                    // words per row
    bool pairbad = false;       // a non-finite pair force reached the fixed-point sums

    __device__ CtaSystem(const Params& p, const Systems& y, char* smem, const SmemLayout& l)
        : P(p), Y(y), L(l), sm(smem) {
        tid = G == 1 ? threadIdx.x : threadIdx.x % T; lane = tid & 31; warp = tid >> 5;
        lv = at<float>(L.sysc);
    }
    template <class X> __device__ __forceinline__ X* at(int off) { return reinterpret_cast<X*>(sm + off); }
    // per-atom / per-node arrays that a compact layout leaves in global memory
    static constexpr bool kMayCompact = T >= kCompactMinThreads;
    __device__ __forceinline__ bool compact() const { return kMayCompact && L.ng < 0; }
    __device__ __forceinline__ int4 ngs(int a) { return compact() ? __ldg(Y.neighs + aoff + a) : at<int4>(L.ng)[a]; }
    __device__ __forceinline__ int4 ngc(int a) { return compact() ? __ldg(Y.neighCell + aoff + a) : at<int4>(L.ngC)[a]; }
    __device__ __forceinline__ int4 bks(int a) { return compact() ? __ldg(Y.bkneighs + aoff + a) : at<int4>(L.bk)[a]; }
    __device__ __forceinline__ float4 plq(int a) { return compact() ? __ldg(Y.PLQ + aoff + a) : at<float4>(L.PLQ)[a]; }
    // velocities (read and written by the owner of a vector only)
    __device__ __forceinline__ float4* vels() { return kMayCompact && L.vel < 0 ? Y.vel + voff : at<float4>(L.vel); }
    __device__ __forceinline__ float4 npar(int off, const float4* g, int n) {
        return compact() ? __ldg(g + noff + n) : at<float4>(off)[n];
    }

    // stage system s; contains a barrier, and the caller's next one makes all of it visible
    __device__ void load(int s) {
        isys = s;
        const int4 d = Y.desc[s];
        aoff = d.x; noff = d.y; voff = d.z; natoms = d.w;
        nnode = Y.nnode[s];
        nvecs = natoms + nnode;
        xrow = Y.xmask + Y.moff[s];
        nbw = (natoms + 31) >> 5;
        pairbad = false;
        if (tid < 9) lv[tid] = Y.lvec[9 * s + tid];
        if (tid >= 9 && tid < 12) lv[tid] = comp(Y.gorg[s], tid - 9);
        float4* spos = at<float4>(L.pos);
        for (int v = tid; v < nvecs; v += T) spos[v] = Y.pos[voff + v];
        if (L.vel >= 0)
            for (int v = tid; v < nvecs; v += T) at<float4>(L.vel)[v] = Y.vel[voff + v];
        float4* sREQ = at<float4>(L.REQ);
        const bool full = !compact();         // else topology stays in global memory
        const int npx = P.npbc[0], npy = P.npbc[1], npz = P.npbc[2];
        const int central = (npz * (2 * npy + 1) + npy) * (2 * npx + 1) + npx;
        int h = 0;
        for (int a = tid; a < natoms; a += T) {
            const float4 r = Y.REQ[aoff + a];
            const int4 g = Y.neighs[aoff + a], c = Y.neighCell[aoff + a];
            sREQ[a] = r;
            h |= (r.w != 0.f);
            h |= ((g.x >= 0 && c.x != central) || (g.y >= 0 && c.y != central) || (g.z >= 0 && c.z != central) ||
                  (g.w >= 0 && c.w != central)) ? 2 : 0;
            if (L.key >= 0 && Y.gkey) at<unsigned>(L.key)[a] = Y.gkey[aoff + a];
            if (full) {
                at<float4>(L.PLQ)[a] = Y.PLQ[aoff + a];
                at<int4>(L.ng)[a] = g;
                at<int4>(L.ngC)[a] = c;
                at<int4>(L.bk)[a] = Y.bkneighs[aoff + a];
            }
        }
        hasH = sync_or(h & 1);
        hasX = sync_or(h & 2);
        if (full)
            for (int n = tid; n < nnode; n += T) {
                at<float4>(L.apar)[n] = Y.apars[noff + n]; at<float4>(L.bL)[n] = Y.bLs[noff + n];
                at<float4>(L.bK)[n] = Y.bKs[noff + n]; at<float4>(L.ksp)[n] = Y.Ksp[noff + n];
                at<float4>(L.kpp)[n] = Y.Kpp[noff + n];
            }
    }

    // bounding box of the atoms (all threads end with the same box); needs a barrier inside
    __device__ void bbox_from_smem() {
        const float4* spos = at<float4>(L.pos);
        float mn[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, mx[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        for (int a = tid; a < natoms; a += T) {
            const float4 p = spos[a];
            mn[0] = fminf(mn[0], p.x); mn[1] = fminf(mn[1], p.y); mn[2] = fminf(mn[2], p.z);
            mx[0] = fmaxf(mx[0], p.x); mx[1] = fmaxf(mx[1], p.y); mx[2] = fmaxf(mx[2], p.z);
        }
        bbox_reduce(mn, mx);
    }
    // reduce per-thread boxes: warp shuffle, warp partials in smem, barrier, redundant final
    __device__ void bbox_reduce(float* mn, float* mx) {
        float* red = at<float>(L.red) + 8 * 2 * L.nwarps;   // after the 4 doubles per warp
#pragma unroll
        for (int k = 0; k < 3; k++) { mn[k] = wmin(mn[k]); mx[k] = wmax(mx[k]); }
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < 3; k++) { red[6 * warp + k] = mn[k]; red[6 * warp + 3 + k] = mx[k]; }
        }
        sync();
        float a[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, b[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        for (int w = 0; w < L.nwarps; w++) {
#pragma unroll
            for (int k = 0; k < 3; k++) { a[k] = fminf(a[k], red[6 * w + k]); b[k] = fmaxf(b[k], red[6 * w + 3 + k]); }
        }
#pragma unroll
        for (int k = 0; k < 3; k++) { bbmin[k] = a[k]; bbmax[k] = b[k]; }
    }

    // is image (ix,iy,iz) within the cutoff of the molecule's own box?
    __device__ __forceinline__ bool image_active(int ix, int iy, int iz) const { return image_within(ix, iy, iz, P.Rc2); }
    // ... within sqrt(R2) (the cutoff, or the cutoff plus the list skin)
    __device__ __forceinline__ bool image_within(int ix, int iy, int iz, float R2) const {
        if (P.Rc2 <= 0.f) return true;
        if (ix == 0 && iy == 0 && iz == 0) return true;
        const float3 sh = image_shift(lv, ix, iy, iz);
        // gap between [bbmin,bbmax] and [bbmin+sh, bbmax+sh] per axis
        const float gx = fmaxf(0.f, fabsf(sh.x) - (bbmax[0] - bbmin[0]));
        const float gy = fmaxf(0.f, fabsf(sh.y) - (bbmax[1] - bbmin[1]));
        const float gz = fmaxf(0.f, fabsf(sh.z) - (bbmax[2] - bbmin[2]));
        return gx * gx + gy * gy + gz * gz < R2;
    }

    // Candidate lists of the shifted images: atom j is a candidate of image
    // (ix,iy,iz) when its shifted position lies within sqrt(R2) (the cutoff,
    // or the cutoff plus the list skin) of this system's own bounding box (no
    // atom i can reach the others).  Lists are
    // ascending in j (ballot words, per-image prefix sums), so the pair sums
    // keep a fixed order.  All threads; contains barriers.
    __device__ void build_candidates(float R2) {
        const float4* spos = at<float4>(L.pos);
        uint32_t* words = at<uint32_t>(L.cwords);
        int* pref = at<int>(L.cpref);
        int* cnt = at<int>(L.ccnt);
        unsigned short* list = at<unsigned short>(L.clist);
        const int npx = P.npbc[0], npy = P.npbc[1], npz = P.npbc[2];
        const int nw = L.nwords;
        for (int base = warp * 32; base < natoms; base += T) {
            const int j = base + lane;
            const float4 p = (j < natoms) ? spos[j] : make_float4(0, 0, 0, 0);
            int k = 0;
            for (int iz = -npz; iz <= npz; iz++)
                for (int iy = -npy; iy <= npy; iy++)
                    for (int ix = -npx; ix <= npx; ix++) {
                        if ((ix | iy | iz) == 0) continue;
                        bool c = false;
                        if (j < natoms && image_within(ix, iy, iz, R2)) {
                            const float3 sh = image_shift(lv, ix, iy, iz);
                            const float qx = p.x + sh.x, qy = p.y + sh.y, qz = p.z + sh.z;
                            const float gx = fmaxf(0.f, fmaxf(bbmin[0] - qx, qx - bbmax[0]));
                            const float gy = fmaxf(0.f, fmaxf(bbmin[1] - qy, qy - bbmax[1]));
                            const float gz = fmaxf(0.f, fmaxf(bbmin[2] - qz, qz - bbmax[2]));
                            c = gx * gx + gy * gy + gz * gz < R2;
                        }
                        const uint32_t bal = __ballot_sync(0xffffffffu, c);
                        if (lane == 0) words[k * nw + (base >> 5)] = bal;
                        k++;
                    }
        }
        sync();
        for (int k = warp; k < L.nimg; k += L.nwarps) {
            int run = 0;
            for (int w0 = 0; w0 < nw; w0 += 32) {
                const int w = w0 + lane;
                const uint32_t m = (w < nw && 32 * w < natoms) ? words[k * nw + w] : 0u;
                const int c = __popc(m);
                int incl = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += t;
                }
                if (w < nw) pref[k * nw + w] = run + incl - c;
                run += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (lane == 0) cnt[k] = run;
        }
        sync();
        for (int j = tid; j < natoms; j += T) {
            const int w = j >> 5;
            const uint32_t below = (1u << (j & 31)) - 1u;
            for (int k = 0; k < L.nimg; k++) {
                const uint32_t m = words[k * nw + w];
                if ((m >> (j & 31)) & 1u) list[k * L.maxNA + pref[k * nw + w] + __popc(m & below)] = (unsigned short)j;
            }
        }
        sync();
    }

    // excluded pair of the shifted image ipbc (NBFF::evalLJQs_ng4_PBC_atom,
    // NBFF.h:590-607): i itself, and the bonded neighbours of i whose cell is this image
    __device__ __forceinline__ bool image_excluded(int i, int j, int ipbc) {
        if (j == i) return true;
        if (!hasX) return false;
        const int4 ng = ngs(i), ngC = ngc(i);
        return (ngC.x == ipbc && ng.x == j) || (ngC.y == ipbc && ng.y == j) || (ngC.z == ipbc && ng.z == j) ||
               (ngC.w == ipbc && ng.w == j);
    }

    // 64-bit fixed-point force sums in shared memory (2^-32 eV/A resolution):
    // integer addition is associative, so the totals do not depend on which
    // warp adds first.  Each add is clamped to |f| <= 2^20 eV/A, so the sums
    // (2^31 units of range per eV/A) cannot wrap for any system that fits a
    // block; a non-finite force (atoms on top of each other) would convert to
    // an arbitrary integer, so it marks the system bad instead (assemble).
    static constexpr float kFix = 4294967296.f;
    static constexpr float kFixMax = 1048576.f;
    __device__ __forceinline__ void fix_add(long long* a, float3 f) {
        pairbad |= !isfinite(f.x + f.y + f.z);
        const float x = fminf(fmaxf(f.x, -kFixMax), kFixMax), y = fminf(fmaxf(f.y, -kFixMax), kFixMax);
        const float z = fminf(fmaxf(f.z, -kFixMax), kFixMax);
        add64(a + 0, __float2ll_rn(x * kFix));
        add64(a + 1, __float2ll_rn(y * kFix));
        add64(a + 2, __float2ll_rn(z * kFix));
    }
    // 64-bit add in shared memory by two 32-bit ones (the hardware's; a 64-bit one is a
    // compare-and-swap loop): whoever makes the low word wrap carries
    static __device__ __forceinline__ void add64(long long* a, long long v) {
        unsigned* w = reinterpret_cast<unsigned*>(a);
        const unsigned lo = (unsigned)v, old = atomicAdd(w, lo);
        atomicAdd(w + 1, (unsigned)((unsigned long long)v >> 32) + (old + lo < old ? 1u : 0u));
    }

    // bonded terms of nodes tid, tid + nt, ... by threads tid < nt; caps get a zero own-force
    template <bool ENERGY>
    __device__ __forceinline__ void bonded_phase(int nt, double& Eb, double& e13) {
        const float4* spos = at<float4>(L.pos);
        const float4* sREQ = at<float4>(L.REQ);
        float4* fasm = at<float4>(L.fasm);
        float4* fng = at<float4>(L.fng);
        if (tid >= nt) return;
        for (int ia = tid; ia < natoms; ia += nt) {
            if (ia >= nnode) { fasm[ia] = make_float4(0, 0, 0, 0); continue; }
            BondedOut o;
            eval_atom<ENERGY>(ia, natoms, nnode, P.flags, P.Fmax2NB, spos, sREQ, ngs(ia), ngc(ia),
                              npar(L.apar, Y.apars, ia), npar(L.bL, Y.bLs, ia), npar(L.bK, Y.bKs, ia),
                              npar(L.ksp, Y.Ksp, ia), npar(L.kpp, Y.Kpp, ia), lv, P.npbc[0], P.npbc[1], P.npbc[2],
                              __ldg(Y.a13 + noff + ia), Cut13(P), o);
            fasm[ia] = make_float4(o.fa.x, o.fa.y, o.fa.z, 0.f);
            fasm[natoms + ia] = make_float4(o.fpi.x, o.fpi.y, o.fpi.z, 0.f);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                fng[ia * 4 + k] = make_float4(o.fbs[k].x, o.fbs[k].y, o.fbs[k].z, 0.f);
                fng[4 * L.maxNN + ia * 4 + k] = make_float4(o.fps[k].x, o.fps[k].y, o.fps[k].z, 0.f);
            }
            if (ENERGY) { Eb += (double)o.E; e13 += (double)o.E13; }
        }
    }

    // GridFF B-spline of every atom, 4 lanes per atom (x-slices), by the
    // threads t0 = 0 .. nt-1 of the caller (whole warps); zero without a grid
    template <bool ENERGY>
    __device__ void grid_phase(int t0, int nt, float4* fgr, double& Eg) {
        const float4* spos = at<float4>(L.pos);
        if (!(P.flags & F_GRID)) {
            for (int a = t0; a < natoms; a += nt) fgr[a] = make_float4(0, 0, 0, 0);
            return;
        }
        const int nunits = natoms * 4;
        const bool cached = Y.gkey != nullptr;      // launch-uniform
        for (int u0 = 0; u0 < nunits; u0 += nt) {
            const int u = u0 + t0;
            const int i = u >> 2, a = u & 3;
            const bool ok = i < natoms;
            const int ic = ok ? i : natoms - 1;
            const float4 p = spos[ic];
            const float3 uu = make_float3((p.x + lv[9]) * P.ginv[0], (p.y + lv[10]) * P.ginv[1],
                                          (p.z + lv[11]) * P.ginv[2]);
            float3 e = make_float3(0, 0, 0);
            float4 bx = make_float4(0, 0, 0, 0), dx = bx;
            if (cached)
                e = grid_slice_cached(P.grid, P.gn[0], P.gn[1], P.gn[2], uu, plq(ic), a, ok, Y.gkey + aoff + ic,
                                      Y.gkey + aoff + ic, Y.gcs + (size_t)(aoff + ic) * 16, bx, dx);
            else if (ok)
                e = grid_slice<(T >= MMFF_UNROLL_MIN_T) ? 4 : 1>(P.grid, P.gn[0], P.gn[1], P.gn[2], uu, plq(ic), a, bx, dx);
            float4 r = slice_force(e, bx, dx, a);
#pragma unroll
            for (int o = 2; o > 0; o >>= 1) {
                r.x += __shfl_xor_sync(0xffffffffu, r.x, o);
                r.y += __shfl_xor_sync(0xffffffffu, r.y, o);
                r.z += __shfl_xor_sync(0xffffffffu, r.z, o);
                if (ENERGY) r.w += __shfl_xor_sync(0xffffffffu, r.w, o);
            }
            if (ok && a == 0) {
                fgr[i] = make_float4(r.x * P.gmi[0], r.y * P.gmi[1], r.z * P.gmi[2], 0.f);
                if (ENERGY) Eg += (double)r.w;
            }
        }
    }
};

}  // namespace mmff
