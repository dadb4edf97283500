// mmff_relax.cu -- persistent relaxation kernels for sm_100a, one CTA per system.
//
// The system's whole state (positions, velocities, topology, force-field
// parameters, recoil slots) is staged in shared memory, and every FIRE step
// runs inside the CTA with three block barriers:
//   forces   bonded terms (4 lanes per node), GridFF samples (4 lanes per atom),
//            ordered pairs of the central image (and, without a cutoff, of
//            every image), the listed pairs of the shifted images
//   | barrier |
//   assemble recoil slots, clamp, FP64 sums of (f.v, v.v, f.f) and max |f|^2
//   | barrier |
//   move     FIRE_update_params in FP64 (every thread computes the same
//            scalars), move_atom_FIRE, displacement since the lists' build
//   | barrier |
// A CTA claims systems from a device work queue (atomic counter): one that
// finishes a system (converged, failed or out of steps) writes it back and
// claims the next one, so converged systems retire and their slots refill
// without a host round trip.
//
// Bound: FP32 issue, with 16 warps per SM (128 registers, shared memory) and, in
// the small blocks, instruction fetch.  Hence few instructions per pair (two
// pairs per packed operation), loops instead of straight-line code (bonded
// terms by neighbour), three barriers, and shared-memory offsets as a kernel
// parameter (constant bank) instead of registers.  Time per system-step with
// the chip full, the kernel before (ordered thread-per-node bonded terms,
// 32 x 32 Newton-3 tiles with shuffled reactions, lists in runs per thread) and
// this one: 28 atoms 0.0087 -> 0.0056 us, 60: 0.0224 -> 0.0155, 100: 0.0566 ->
// 0.0291, 200: 0.136 -> 0.088, 330: 0.286 -> 0.212; 127 atoms without a cutoff
// (9 images), 300 systems: 0.380 -> 0.278 us.
#include "mmff_engine.cuh"

#include <cooperative_groups.h>

namespace mmff {

// ---- packed FP32 pairs (sm_100: one instruction, two IEEE operations)
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) { f32x2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { f32x2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) { f32x2 d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ float hsum2(f32x2 v) { float a, b; unpack2(v, a, b); return a + b; }

// two atoms j at a time, as the arrays of SmemLayout::soa hold them
struct PairJ { f32x2 x, y, z, R, E, Q, H; };
// one atom i (shift - position, so that d = p_j + shift - p_i is one addition), in both halves
struct PairI { f32x2 x, y, z, R, E, Q, H; };
struct PairC { f32x2 kq, p12, m12; float Rc2; };

// Two ordered pairs: force on i into (fx, fy, fz).  getLJQH (Forces.h:341-360)
// plus the shifted-force Coulomb part, as
//   F = 12 E0 u6 (1 - u6 (1 + H)) / r^2 + Q (kq - 1/r^2) / r,  f_i += d F
// taken as (12 E0 u6 (...) + g) / r^2 + (-kq) g with g = -Q / r (i.Q and c.kq hold
// the negatives): 23 packed operations a pair instead of 24 and a shorter chain
// (4096 x 60 atoms 159.9 -> 153.4 ms; errors against FP64 unchanged).
// Excluded and out-of-range pairs are evaluated
// at r^2 = 1e30, where every term underflows to zero except kq Q / r
// (< 1e-16 eV/A).  bits 0, 1 of m: pair excluded.
template <bool HB, bool COUNT>
__device__ __forceinline__ void pair2(const PairJ& j, const PairI& i, const PairC& c, bool ex0, bool ex1, f32x2& fx,
                                      f32x2& fy, f32x2& fz, unsigned long long& np) {
    const f32x2 dx = add2(j.x, i.x), dy = add2(j.y, i.y), dz = add2(j.z, i.z);
    const f32x2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
    float a, b;
    unpack2(r2, a, b);
    const bool ok0 = !ex0 && a < c.Rc2, ok1 = !ex1 && b < c.Rc2;
    if (COUNT) np += (ok0 ? 1 : 0) + (ok1 ? 1 : 0);
    a = ok0 ? a : 1e30f;
    b = ok1 ? b : 1e30f;
    const f32x2 ir = pack2(rsq(a), rsq(b));
    const f32x2 ir2 = mul2(ir, ir);
    const f32x2 w = mul2(add2(j.R, i.R), ir);
    const f32x2 u2 = mul2(w, w);
    const f32x2 u6 = mul2(mul2(u2, u2), u2);
    f32x2 h = c.m12;
    if (HB) {
        float h0, h1;
        unpack2(mul2(j.H, i.H), h0, h1);
        h = pack2(fmaf(-12.f, fminf(h0, 0.f), -12.f), fmaf(-12.f, fminf(h1, 0.f), -12.f));
    }
    const f32x2 t = mul2(u6, fma2(u6, h, c.p12));
    const f32x2 g = mul2(mul2(i.Q, j.Q), ir);
    const f32x2 F = fma2(ir2, fma2(t, mul2(i.E, j.E), g), mul2(c.kq, g));
    fx = fma2(dx, F, fx); fy = fma2(dy, F, fy); fz = fma2(dz, F, fz);
}

// sqrt(vv) / (sqrt(ff) + 1e-32) in FP64 without the library's roots and division (four
// times the instructions, for every thread of a step) where both arguments are in
// range and the 1e-32 is below the last place
__device__ __forceinline__ double length_ratio(double vv, double ff) {
    if (vv > 1e-30 && ff > 1e-30 && vv < 1e30 && ff < 1e30) return vv * inv_sqrt64(vv) * inv_sqrt64(ff);
    return vv > 0.0 ? sqrt(vv) / (sqrt(ff) + 1e-32) : 0.0;
}

// CL: a cluster of CTAs relaxes one system (batches with fewer systems than half
// the SMs).  Every CTA holds the whole system and runs every step; each takes a
// share of the pairs, list rows and GridFF samples into its own fixed-point
// sums, and assemble adds the sums of all of them through distributed shared
// memory.  Integer sums are exact, so all CTAs get the same bits, and with the
// same code on the same bits they take every decision alike: the cluster barrier
// after the forces is the only one of a step.  Two sets of sums alternate, so
// that the next step's adds never meet a neighbour that still reads.  Whatever
// one CTA alone could see (a non-finite pair force, a full list slot) is
// exchanged before it decides anything.
template <int T, bool COUNT, bool CL = false>
struct RelaxEngine : CtaSystem<T> {
    using B = CtaSystem<T>;
    using B::P; using B::Y; using B::L; using B::tid; using B::lane; using B::warp;
    using B::isys; using B::natoms; using B::nnode; using B::nvecs; using B::aoff; using B::noff; using B::voff;
    using B::lv; using B::hasH; using B::hasX; using B::xrow; using B::nbw; using B::pairbad; using B::kFix;
    using B::ngs; using B::ngc; using B::bks; using B::image_within; using B::build_candidates; using B::fix_add;
    using B::image_excluded; using B::bbox_from_smem;
    template <class X> __device__ __forceinline__ X* at(int off) { return B::template at<X>(off); }
    static constexpr int NW = T / 32;
    unsigned long long npair = 0;      // COUNT: pair-images evaluated by this thread
    // shifted-image pair lists of the current system (block-uniform): usable
    // (a scratch slot, no overflow so far), built and valid, entries
    bool listok = false, listed = false;
    int nlist = 0, nrows = 0;
    int cr = 0, cn = 1, par = 0;       // CL: rank in the cluster, its size, which set of sums this step uses

    __device__ RelaxEngine(const Params& p, const Systems& y, char* smem, const SmemLayout& l) : B(p, y, smem, l) {
        if constexpr (CL) {
            cr = (int)cooperative_groups::this_cluster().block_rank();
            cn = (int)cooperative_groups::this_cluster().num_blocks();
        }
    }
    // barrier of everything that works on the system
    static __device__ __forceinline__ void csync() {
        if constexpr (CL) cooperative_groups::this_cluster().sync();
        else __syncthreads();
    }
    // this step's force sums
    __device__ __forceinline__ long long* sums() { return at<long long>(L.facc) + (CL ? par * 3 * L.maxNA : 0); }
    // flags of this CTA that the others read: [0, 1] non-finite pair force (per set of sums), [2] list slot full
    __device__ __forceinline__ int* flags_cl() const {
        __shared__ int f[4];
        return f;
    }
    // some CTA of the cluster set flag k
    __device__ __forceinline__ bool any_cl(int k) const {
        int a = 0;
        if constexpr (CL)
            for (int c = 0; c < cn; c++) a |= cooperative_groups::this_cluster().map_shared_rank(flags_cl(), c)[k];
        return a != 0;
    }

    // arrays of the pair loops, NP atoms each
    __device__ __forceinline__ int np() const { return 32 * L.nwords; }
    __device__ __forceinline__ float* soa(int k) { return at<float>(L.soa) + k * np(); }

    __device__ void load(int s) {
        B::load(s);
        listok = P.vlist != nullptr && natoms <= 4096 && P.Rc2 > 0.f && L.nimg > 0 && L.nimg <= kListMaxImages &&
                 (P.flags & F_NONBONDED);
        listed = false;
        nlist = 0;
        __syncthreads();
        if (L.shf >= 0 && tid < L.nimg) {
            const float3 s = image_of(image_index(tid));
            at<float4>(L.shf)[tid] = make_float4(s.x, s.y, s.z, 0.f);
        }
        split_pairs((P.flags & F_PBC) && !(P.Rc2 > 0.f));
        // padding atoms up to whole 8-atom chunks: no charge, no LJ, far away
        const float4* spos = at<float4>(L.pos);
        const float4* sREQ = at<float4>(L.REQ);
        for (int a = tid; a < np(); a += T) {
            const bool v = a < natoms;
            const float4 p = v ? spos[a] : make_float4(1e6f, 1e6f, 1e6f, 0.f);
            const float4 r = v ? sREQ[a] : make_float4(0.f, 0.f, 0.f, 0.f);
            soa(0)[a] = p.x; soa(1)[a] = p.y; soa(2)[a] = p.z;
            soa(3)[a] = r.x; soa(4)[a] = r.y; soa(5)[a] = r.z; soa(6)[a] = r.w;
        }
        long long* facc = at<long long>(L.facc);
        for (int a = tid; a < 3 * natoms; a += T) facc[a] = 0;
        if constexpr (CL) {
            par = 0;
            for (int a = tid; a < 3 * natoms; a += T) facc[3 * L.maxNA + a] = 0;
            if (tid < 4) flags_cl()[tid] = 0;
        }
    }

    // ---- ordered pairs (i, j + shift), every atom i of the central image -----
    // Lanes own 32 atoms i and walk the atoms j together (shared-memory
    // broadcasts, no shuffles, no reactions), two j per packed instruction.
    // Work: i-blocks x images x chunks of 8 j, one flat range cut into equal
    // parts, one per warp; a warp's sum for a block goes to the fixed-point
    // accumulators when its range leaves the block.  In the last block, when
    // at most 16 atoms are left, 2, 4, ... lanes share an atom and take every
    // 2nd, 4th, ... chunk.
    int pb0, pr0, plen;          // this warp's part of the range: first block, position in it, length
    __device__ __forceinline__ int last_lg() const {      // last block: 2^lg lanes per atom
        const int rem = natoms - 32 * (nbw - 1);
        return rem > 16 ? 0 : rem > 8 ? 1 : rem > 4 ? 2 : rem > 2 ? 3 : rem > 1 ? 4 : 5;
    }
    __device__ void split_pairs(bool all_images) {        // once per system
        const int nim = all_images ? (2 * P.npbc[0] + 1) * (2 * P.npbc[1] + 1) * (2 * P.npbc[2] + 1) : 1;
        const int c8 = (natoms + 7) >> 3, lg = last_lg(), cl = (c8 + (1 << lg) - 1) >> lg;
        const int total = ((nbw - 1) * c8 + cl) * nim;
        const int w = cr * NW + warp, nw = cn * NW;
        const int q = (int)((long long)total * w / nw);
        plen = (int)((long long)total * (w + 1) / nw) - q;
        pb0 = min(q / (c8 * nim), nbw - 1);
        pr0 = q - pb0 * c8 * nim;
    }

    template <bool HB>
    __device__ void ordered_pairs(bool all_images, long long* facc) {
        const int npx = all_images ? P.npbc[0] : 0, npy = all_images ? P.npbc[1] : 0, npz = all_images ? P.npbc[2] : 0;
        const int nxi = 2 * npx + 1, nyi = 2 * npy + 1, nim = nxi * nyi * (2 * npz + 1);
        const int central = (npz * nyi + npy) * nxi + npx;
        const int c8 = (natoms + 7) >> 3, lg = last_lg(), cl = (c8 + (1 << lg) - 1) >> lg;
        PairC C;
        const bool cut = P.Rc2 > 0.f;
        C.Rc2 = cut ? P.Rc2 : 3.0e38f;
        C.kq = pack2(-P.kq_rc2, -P.kq_rc2); C.p12 = pack2(12.f, 12.f); C.m12 = pack2(-12.f, -12.f);
        const float *X = soa(0), *Yy = soa(1), *Z = soa(2), *R = soa(3), *E = soa(4), *Q = soa(5), *H = soa(6);
        int b = pb0, r = pr0, left = plen;                   // r: position inside the block's images x chunks
        while (left > 0) {
            const bool last = b == nbw - 1;
            const int sh = last ? lg : 0, cs = last ? cl : c8;
            const int rend = min(cs * nim, r + left);
            left -= rend - r;
            const int i = 32 * b + (lane & ((32 >> sh) - 1)), sub = lane >> (5 - sh);
            const bool vi = i < natoms;
            const int ic = vi ? i : natoms - 1;
            const float ix = X[ic], iy = Yy[ic], iz = Z[ic];
            PairI I;
            I.R = pack2(R[ic], R[ic]); I.E = pack2(E[ic], E[ic]); I.Q = pack2(-Q[ic], -Q[ic]); I.H = HB ? pack2(H[ic], H[ic]) : 0;
            const uint8_t* row = reinterpret_cast<const uint8_t*>(xrow + ic * nbw);     // byte c: chunk c of 8 atoms j
            f32x2 fx = 0, fy = 0, fz = 0;
            while (r < rend) {
                const int im = all_images ? r / cs : 0;
                int t = r - im * cs;
                const int tend = min(cs, t + (rend - r));
                r += tend - t;
                float3 s = make_float3(0.f, 0.f, 0.f);
                if (im != central) s = image_shift(lv, im % nxi - npx, (im / nxi) % nyi - npy, im / (nxi * nyi) - npz);
                I.x = pack2(s.x - ix, s.x - ix); I.y = pack2(s.y - iy, s.y - iy); I.z = pack2(s.z - iz, s.z - iz);
                // excluded j of chunk c (bits 0..7): the host-built rows in the
                // central image; else i itself and its bonded neighbours there
                auto excl = [&](int c) -> uint32_t {
                    if (!vi || c >= c8) return 0xFFu;
                    if (im == central) return __ldg(row + c);
                    uint32_t m = (i >> 3) == c ? 1u << (i & 7) : 0u;
                    if (8 * c + 8 > natoms) m |= 0xFFu << (natoms - 8 * c);
                    if (hasX) {
                        const int4 g = ngs(i), gc = ngc(i);
                        if (gc.x == im && g.x >= 0 && (g.x >> 3) == c) m |= 1u << (g.x & 7);
                        if (gc.y == im && g.y >= 0 && (g.y >> 3) == c) m |= 1u << (g.y & 7);
                        if (gc.z == im && g.z >= 0 && (g.z >> 3) == c) m |= 1u << (g.z & 7);
                        if (gc.w == im && g.w >= 0 && (g.w >> 3) == c) m |= 1u << (g.w & 7);
                    }
                    return m;
                };
                uint32_t mn = excl((t << sh) + sub);
                for (; t < tend; t++) {
                    const uint32_t m = mn;
                    const int j0 = 8 * min((t << sh) + sub, c8 - 1);
                    if (t + 1 < tend) mn = excl(((t + 1) << sh) + sub);
#pragma unroll
                    for (int k = 0; k < 8; k += 4) {
                        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(X + j0 + k);
                        const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(Yy + j0 + k);
                        const ulonglong2 z = *reinterpret_cast<const ulonglong2*>(Z + j0 + k);
                        const ulonglong2 rr = *reinterpret_cast<const ulonglong2*>(R + j0 + k);
                        const ulonglong2 e = *reinterpret_cast<const ulonglong2*>(E + j0 + k);
                        const ulonglong2 qq = *reinterpret_cast<const ulonglong2*>(Q + j0 + k);
                        ulonglong2 h = make_ulonglong2(0, 0);
                        if (HB) h = *reinterpret_cast<const ulonglong2*>(H + j0 + k);
                        const PairJ ja = {x.x, y.x, z.x, rr.x, e.x, qq.x, h.x}, jb = {x.y, y.y, z.y, rr.y, e.y, qq.y, h.y};
                        pair2<HB, COUNT>(ja, I, C, m & (1u << k), m & (2u << k), fx, fy, fz, npair);
                        pair2<HB, COUNT>(jb, I, C, m & (4u << k), m & (8u << k), fx, fy, fz, npair);
                    }
                }
            }
            float3 f = make_float3(hsum2(fx), hsum2(fy), hsum2(fz));
            for (int o = 32 >> sh; o < 32; o <<= 1) {        // lanes that share an atom
                f.x += __shfl_xor_sync(0xffffffffu, f.x, o);
                f.y += __shfl_xor_sync(0xffffffffu, f.y, o);
                f.z += __shfl_xor_sync(0xffffffffu, f.z, o);
            }
            if (all_images) {
                // an atom on top of an image: the force is scaled to the
                // accumulators' range as a vector, so that its direction stays
                const float m = fmaxf(fabsf(f.x), fmaxf(fabsf(f.y), fabsf(f.z)));
                if (m > B::kFixMax && isfinite(m)) f = f * (B::kFixMax / m);
            }
            if (vi && sub == 0) fix_add(facc + 3 * i, f);
            b++;
            r = 0;
        }
    }

    // ---- shifted images under a cutoff ---------------------------------------
    // one ordered pair (scalar form of pair2)
    template <bool HB>
    __device__ __forceinline__ void pair1(float dx, float dy, float dz, float4 Ri, float4 Rj, bool excl, float3& f) {
        bool ok;
        float e;
        const float F = pair_force<false, HB>(dx, dy, dz, Ri, Rj, excl, P.Rc2, P.kq_rc2, 0.f, true, ok, e);
        if (COUNT && ok) npair++;
        f.x = fmaf(dx, F, f.x); f.y = fmaf(dy, F, f.y); f.z = fmaf(dz, F, f.z);
    }
    // shifted image k (0 .. nimg-1, without the central one) -> image index with it, and its shift
    __device__ __forceinline__ int image_index(int k) const { return k < L.nimg / 2 ? k : k + 1; }
    __device__ __forceinline__ float3 image_of(int ipbc) const {
        const int nxi = 2 * P.npbc[0] + 1, nyi = 2 * P.npbc[1] + 1;
        return image_shift(lv, ipbc % nxi - P.npbc[0], (ipbc / nxi) % nyi - P.npbc[1], ipbc / (nxi * nyi) - P.npbc[2]);
    }

    // Per-step candidate rows: every ordered pair (i, j + shift) with i a
    // candidate of the mirror image and j one of the image (build_candidates),
    // one thread per row.  The path of systems without pair lists (lists
    // switched off, more than kListMaxImages images, a list that overflowed).
    template <bool HB>
    __device__ void candidate_rows(const float4* spos, const float4* sREQ, long long* facc) {
        const int* ccnt = at<int>(L.ccnt);
        const unsigned short* clist = at<unsigned short>(L.clist);
        int nrows = 0;
        for (int k = 0; k < L.nimg; k++) nrows += ccnt[L.nimg - 1 - k];
        for (int u = cr * T + tid; u < nrows; u += cn * T) {
            int c = u, k = 0;
            while (c >= ccnt[L.nimg - 1 - k]) { c -= ccnt[L.nimg - 1 - k]; k++; }
            const int i = clist[(L.nimg - 1 - k) * L.maxNA + c];
            const int ipbc = image_index(k);
            const float3 s = image_of(ipbc);
            const float4 pi = spos[i], Ri = sREQ[i];
            const unsigned short* Jl = clist + k * L.maxNA;
            float3 f = make_float3(0.f, 0.f, 0.f);
            for (int q = 0; q < ccnt[k]; q++) {
                const int j = Jl[q];
                const float4 pj = spos[j];
                pair1<HB>(pj.x + s.x - pi.x, pj.y + s.y - pi.y, pj.z + s.z - pi.z, Ri, sREQ[j], image_excluded(i, j, ipbc), f);
            }
            fix_add(facc + 3 * i, f);
        }
    }

    // Shifted-image pair lists (Verlet lists with a skin, P.vskin, 1 A by
    // default).  Of the pairs the candidate rows of the shifted images
    // evaluate, only a few percent lie inside the cutoff: for a large molecule
    // the candidates of an image span its whole cross-section.  With lists,
    // the ordered pairs (i, j + shift of image k) over every shifted image k
    // closer than Rc + skin are collected once and evaluated every step (both
    // orders of a pair are listed, so no reaction is needed) until some atom
    // has moved more than skin/2 since the build (move() checks); then they are
    // rebuilt.  One row per atom i over all images, entry j | k << 12, in the
    // CTA's slot of global scratch; row starts in shared memory.
    __device__ __forceinline__ unsigned short* vslot() const { return P.vlist + (size_t)blockIdx.x * P.vcap; }

    // pass over the listed pairs of atom i by one warp: f(pair listed here, entry) per 32 candidates
    template <class F>
    __device__ __forceinline__ void row_pass(int i, const float4* spos, float Rv2, F&& f) {
        const int* ccnt = at<int>(L.ccnt);
        const unsigned short* clist = at<unsigned short>(L.clist);
        const uint32_t* words = at<uint32_t>(L.cwords);
        const float4 pi = spos[i];
        for (int k = 0; k < L.nimg; k++) {
            if (!((words[(L.nimg - 1 - k) * L.nwords + (i >> 5)] >> (i & 31)) & 1u)) continue;   // i cannot reach image k
            const int ipbc = image_index(k);
            const float4 s = at<float4>(L.shf)[k];
            const float qx = pi.x - s.x, qy = pi.y - s.y, qz = pi.z - s.z;
            const unsigned short* Jl = clist + k * L.maxNA;
            const int nJ = ccnt[k];
            for (int j0 = 0; j0 < nJ; j0 += 32) {
                const int j = Jl[min(j0 + lane, nJ - 1)];
                const float4 pj = spos[j];
                const float dx = pj.x - qx, dy = pj.y - qy, dz = pj.z - qz;
                f(j0 + lane < nJ && fmaf(dx, dx, fmaf(dy, dy, dz * dz)) < Rv2 && !image_excluded(i, j, ipbc), j | (k << 12));
            }
        }
    }

    // rebuild this system's lists from the current positions; false
    // (block-uniform) when they do not fit in the slot.  All threads; barriers.
    __device__ bool list_build(const float4* spos) {
        const float Rv = sqrtf(P.Rc2) + P.vskin, Rv2 = Rv * Rv;
        bbox_from_smem();
        bool any = false;
        for (int k = 0; k < L.nimg; k++) {
            const int ipbc = image_index(k), nxi = 2 * P.npbc[0] + 1, nyi = 2 * P.npbc[1] + 1;
            any |= image_within(ipbc % nxi - P.npbc[0], (ipbc / nxi) % nyi - P.npbc[1], ipbc / (nxi * nyi) - P.npbc[2], Rv2);
        }
        float* vp = at<float>(L.vp);
        for (int a = tid; a < natoms; a += T) {
            const float4 p = spos[a];
            vp[a] = p.x; vp[L.maxNA + a] = p.y; vp[2 * L.maxNA + a] = p.z;
        }
        nlist = 0;
        if (!any) return true;
        build_candidates(Rv2);
        int* rst = at<int>(L.rst);
        for (int i = warp; i < natoms; i += NW) {            // count (CL: the rows of atoms i = cr mod cn)
            int c = 0;
            if (!CL || i % cn == cr) row_pass(i, spos, Rv2, [&](bool in, int) { c += __popc(__ballot_sync(0xffffffffu, in)); });
            if (lane == 0) rst[i] = c;
        }
        __syncthreads();
        if (warp == 0) {                                     // row starts
            int run = 0;
            for (int a0 = 0; a0 < natoms; a0 += 32) {
                const int a = a0 + lane, ce = a < natoms ? rst[a] : 0;
                const int c = (ce + 1) & ~1;                 // rows start at whole words
                int incl = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += t;
                }
                if (a < natoms) rst[a] = 2 * (run + incl - c) + (ce & 1);
                run += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (lane == 0) rst[natoms] = 2 * run;
        }
        __syncthreads();
        const int total = rst[natoms] >> 1;
        bool full = total > P.vcap;
        if constexpr (CL) {
            if (tid == 0) flags_cl()[2] = full;
            csync();
            full = any_cl(2);
            csync();
        }
        if (full) return false;
        // rows by falling length: the rows a warp evaluates at a time are
        // alike (their longest sets the time), atoms without a row drop out
        unsigned short* perm = at<unsigned short>(L.perm);
        float4* flist = at<float4>(L.flist);
        for (int a = tid; a < natoms; a += T) {
            const int n = (rst[a + 1] >> 2) - (rst[a] >> 2);
            flist[a] = make_float4(0.f, 0.f, 0.f, 0.f);
            int rank = 0;
            for (int o = 0, p0 = 0; o < natoms; o++) {
                const int p1 = rst[o + 1] >> 2, m = p1 - p0;
                rank += (m > n) || (m == n && o < a);
                p0 = p1;
            }
            perm[rank] = (unsigned short)a;
        }
        unsigned short* ent = vslot();
        for (int i = warp; i < natoms; i += NW) {            // write
            int at0 = rst[i] >> 1;
            if ((rst[i + 1] >> 1) == at0) continue;
            row_pass(i, spos, Rv2, [&](bool in, int w) {
                const uint32_t bal = __ballot_sync(0xffffffffu, in);
                if (in) ent[at0 + __popc(bal & ((1u << lane) - 1u))] = (unsigned short)w;
                at0 += __popc(bal);
            });
        }
        nlist = total;
        __syncthreads();
        int lo = 0, hi = natoms;                             // rows that are not empty
        while (lo < hi) {
            const int mid = (lo + hi) >> 1, a = perm[mid];
            if ((rst[a + 1] >> 2) > (rst[a] >> 2)) lo = mid + 1; else hi = mid;
        }
        nrows = lo;
        return true;
    }

    // the listed pairs: kRowLanes lanes per atom, two entries (one word) per lane
    // and packed operation; each atom's sum goes to flist (no atomics: the row is
    // all of the atom's listed pairs).  The entries come from L2, several hundred
    // cycles away: four words per lane are in flight ahead of the one evaluated,
    // and a group's next row is fetched before it evaluates this one.  Rows hold
    // 5 to 30 entries: with four lanes fewer of them idle at the row's end and
    // each warp closes eight rows at once (time per system-step, eight -> four
    // lanes: 100 atoms 0.0317 -> 0.0299 us, 200: 0.0942 -> 0.0906, 330: 0.2223 ->
    // 0.2163, 395: 0.3008 -> 0.2933); a cluster's CTA has too few rows for that
    // (350 atoms x 37: 0.604 with eight, 0.634 with four).
    static constexpr int kRowLanes = CL ? 8 : 4;
    template <bool HB>
    __device__ void list_pairs(const float4* spos, const float4* sREQ, long long* facc) {
        constexpr int G = kRowLanes, NG = T / G, RW = 32 / G;      // lanes per row, rows of the block, of a warp
        const int* rst = at<int>(L.rst);
        float4* flist = at<float4>(L.flist);
        const float4* shf = at<float4>(L.shf);
        const uint32_t* ent = reinterpret_cast<const uint32_t*>(vslot());       // two entries a word
        const unsigned short* perm = at<unsigned short>(L.perm);
        const int gl = lane & (G - 1);
        PairC C;
        C.Rc2 = P.Rc2;
        C.kq = pack2(-P.kq_rc2, -P.kq_rc2); C.p12 = pack2(12.f, 12.f); C.m12 = pack2(-12.f, -12.f);
        // row: atom, words, whether the last word holds one entry, first word, and
        // this lane's first four words
        struct Row { int i, nw, odd; const uint32_t* p; uint32_t u[4]; };
        auto fetch = [&](int row, Row& x) {
            x.i = row < nrows ? (int)perm[row] : 0;
            const int a = rst[x.i];
            x.odd = a & 1;
            x.nw = row < nrows ? (rst[x.i + 1] >> 2) - (a >> 2) : 0;
            x.p = ent + (a >> 2) + gl;
#pragma unroll
            for (int t = 0; t < 4; t++) x.u[t] = G * t + gl < x.nw ? x.p[G * t] : 0u;
        };
        Row nx;
        fetch(tid / G, nx);
        for (int i0 = 0, k = 0; i0 < nrows; i0 += NG, k++) {
            Row w = nx;
            // every other round the warps take their rows in reverse order
            if (i0 + NG < nrows) fetch(i0 + NG + ((k & 1) ? tid / G : (NG - RW) - RW * warp + (lane / G)), nx);
            const int i = w.i, n = w.nw;
            f32x2 fx = 0, fy = 0, fz = 0;
            if (gl < n) {
                const float4 pi = spos[i], Ri = sREQ[i];
                PairI I;
                I.x = I.y = I.z = 0;
                I.R = pack2(Ri.x, Ri.x); I.E = pack2(Ri.y, Ri.y); I.Q = pack2(-Ri.z, -Ri.z); I.H = HB ? pack2(Ri.w, Ri.w) : 0;
#pragma unroll 1
                for (int t = gl; t < n; t += G) {
                    const bool one = w.odd && t + 1 == n;                  // the word's second half is no entry
                    const unsigned c0 = w.u[0] & 0xFFFFu, c1 = one ? c0 : w.u[0] >> 16;
                    w.u[0] = w.u[1]; w.u[1] = w.u[2]; w.u[2] = w.u[3];
                    w.p += G;
                    if (t + 4 * G < n) w.u[3] = w.p[3 * G];
                    const float4 s0 = shf[c0 >> 12], s1 = shf[c1 >> 12];
                    const float4 p0 = spos[c0 & 0xFFFu], p1 = spos[c1 & 0xFFFu], R0 = sREQ[c0 & 0xFFFu], R1 = sREQ[c1 & 0xFFFu];
                    PairJ J;
                    J.x = pack2(p0.x + s0.x - pi.x, p1.x + s1.x - pi.x);
                    J.y = pack2(p0.y + s0.y - pi.y, p1.y + s1.y - pi.y);
                    J.z = pack2(p0.z + s0.z - pi.z, p1.z + s1.z - pi.z);
                    J.R = pack2(R0.x, R1.x); J.E = pack2(R0.y, R1.y); J.Q = pack2(R0.z, R1.z); J.H = HB ? pack2(R0.w, R1.w) : 0;
                    pair2<HB, COUNT>(J, I, C, false, one, fx, fy, fz, npair);
                }
            }
            float3 f = make_float3(hsum2(fx), hsum2(fy), hsum2(fz));
#pragma unroll
            for (int o = G / 2; o > 0; o >>= 1) {
                f.x += __shfl_xor_sync(0xffffffffu, f.x, o);
                f.y += __shfl_xor_sync(0xffffffffu, f.y, o);
                f.z += __shfl_xor_sync(0xffffffffu, f.z, o);
            }
            if (CL) {
                if (gl == 0 && n > 0) fix_add(facc + 3 * i, f);
            } else if (gl == 0 && n > 0) {
                auto lim = [](float x) { return fminf(fmaxf(x, -B::kFixMax), B::kFixMax) + 0.f * x; };   // as fix_add; NaN stays
                flist[i] = make_float4(lim(f.x), lim(f.y), lim(f.z), 0.f);
            }
        }
    }

    // ---- bonded terms of one node, four lanes (one per neighbour slot q) ------
    // MMFFsp3_loc::eval_atom (MMFFsp3_loc.h:250-575), the terms of eval_atom in
    // mmff_device.cuh.  A lane evaluates the bond, pi-pi and pi-sigma terms of its
    // neighbour and its own end of the three angles it is part of (the other
    // end's bond vector comes by shuffle), so no force has to travel back; the
    // force on the node is minus the sum of the four ends' (without the 1-3
    // pair part, which acts between the ends).  A thread per node instead is
    // some 1000 instructions of straight-line code, which the small blocks
    // (eight per SM in different phases) mostly wait for the instruction
    // cache to deliver, with the lanes beyond the node count idle.
    // All lanes of the warp call it; ia: node (ok: a real one).
    __device__ __forceinline__ float node_par(int off, const float4* g, int n4) {
        return B::compact() ? __ldg(reinterpret_cast<const float*>(g + noff) + n4) : at<float>(off)[n4];
    }
    __device__ void bonded_node(int ia, bool ok) {
        const float4* spos = at<float4>(L.pos);
        const float4* sREQ = at<float4>(L.REQ);
        const int flags = P.flags, q = lane & 3, n4 = 4 * ia + q;
        int ing = -1, cell = 0;
        if (ok) {
            ing = B::compact() ? __ldg(reinterpret_cast<const int*>(Y.neighs + aoff) + n4) : at<int>(L.ng)[n4];
            cell = B::compact() ? __ldg(reinterpret_cast<const int*>(Y.neighCell + aoff) + n4) : at<int>(L.ngC)[n4];
        }
        // neighbour slots end at the first empty one
        const unsigned neg = (__ballot_sync(0xffffffffu, ing < 0) >> (lane & 28)) & 0xFu;
        const int nbn = neg ? __ffs(neg) - 1 : 4;
        const bool v = q < nbn;
        const float4 apar = B::npar(L.apar, Y.apars, ia);
        const float3 pa = f3(spos[ia]), hpi = f3(spos[natoms + ia]);
        float3 h = make_float3(0.f, 0.f, 1.f), fb = make_float3(0.f, 0.f, 0.f), f13 = fb, fpi = fb, fps = fb;
        float il = 1.f, l = 1.f;
        if (v) {
            h = f3(spos[ing]) - pa;
            // most bonds stay in the central cell: no shift, and none of the integer
            // divisions that name the cell (with the assembly's loads side by side:
            // 24 atoms x 16 systems 0.337 -> 0.324 us per system-step, 60 atoms
            // 0.0159 -> 0.0155, 330: 0.214 -> 0.212)
            if ((flags & F_PBC) && cell != ((2 * P.npbc[1] + 1) * P.npbc[2] + P.npbc[1]) * (2 * P.npbc[0] + 1) + P.npbc[0]) {
                const float3 c = image_cell(cell, P.npbc[0], P.npbc[1], P.npbc[2]);
                h.x += lv[0] * c.x + lv[3] * c.y + lv[6] * c.z;
                h.y += lv[1] * c.x + lv[4] * c.y + lv[7] * c.z;
                h.z += lv[2] * c.x + lv[5] * c.y + lv[8] * c.z;
            }
            const float l2 = dot3(h, h);
            il = rsq_nr(l2);
            l = sqrt_from(l2, il);
            h = h * il;
            if (ia < ing) {
                if (flags & F_BONDS) {
                    float fr = (l - node_par(L.bL, Y.bLs, n4)) * node_par(L.bK, Y.bKs, n4);
                    if (flags & F_SUB_BOND_NB) {
                        const float4 Ri = sREQ[ia], Rj = sREQ[ing];
                        float e, F = l * ljqh<false>(l * l, Ri.x + Rj.x, Ri.y * Rj.y, Ri.z * Rj.z, fminf(Ri.w * Rj.w, 0.f), e);
                        if ((flags & F_CLAMP_NB) && F * F > P.Fmax2NB) F = copysignf(sqrtf(P.Fmax2NB), F);
                        fr -= F;
                    }
                    fb = h * -fr;
                }
                const float kk = node_par(L.kpp, Y.Kpp, n4);
                if ((flags & F_PIPI) && (ing < nnode) && (kk > 1e-6f)) {
                    const float3 h2 = f3(spos[natoms + ing]);             // evalPiAling
                    const float c = dot3(hpi, h2), g = c < 0.f ? -kk : kk, cc = fabsf(c);
                    fpi = fma3(hpi, -cc, h2) * g;
                    fps = fma3(h2, -cc, hpi) * g;
                }
            }
            const float ks = node_par(L.ksp, Y.Ksp, n4);
            if ((flags & F_PISIGMA) && (ks > 1e-6f)) {                    // evalAngleCos
                const float c = dot3(hpi, h);
                const float g = -ks * (c - apar.w) * 2.f;
                fpi = fpi + fma3(hpi, -c, h) * g;
                fb = fb + fma3(h, -c, hpi) * (g * il);
            }
        }
        if (flags & F_ANGLES) {
            const int a13 = (ok && (flags & F_EXCL13)) ? __ldg(Y.a13 + noff + ia) : 0;
            const Cut13 cu(P);
#pragma unroll 1
            for (int d = 1; d < 4; d++) {
                const int p = (q + d) & 3, src = (lane & 28) | p;
                const float3 hp = make_float3(__shfl_sync(0xffffffffu, h.x, src), __shfl_sync(0xffffffffu, h.y, src),
                                              __shfl_sync(0xffffffffu, h.z, src));
                const float lp = __shfl_sync(0xffffffffu, l, src);
                const int jng = __shfl_sync(0xffffffffu, ing, src), jcell = __shfl_sync(0xffffffffu, cell, src);
                if (!v || p >= nbn) continue;
                const float3 hs = h + hp;                                 // evalAngleCosHalf
                // cos and sin of the half angle with their reciprocals (no division)
                const float c2 = dot3(hs, hs) * 0.25f, s2 = fmaxf(1.f - c2 + 1e-14f, 0.f);
                const float rc = rsq(c2), rs = rsq(s2);
                const float fr = il * (-0.25f * apar.z * fmaf(apar.y, sqrt_from(c2, rc), -apar.x * sqrt_from(s2, rs)) * (rc * rs));
                fb = fb + hs * fr + h * (fr * (-2.f * c2));
                if (flags & F_SUB_ANGLE_NB) {
                    const float3 dp = hp * lp - h * l;
                    // x13: the pair sum skipped this central-image pair
                    const bool x13 = ((a13 >> angle_slot(min(q, p), max(q, p))) & 1) && (!(flags & F_PBC) || cell == jcell);
                    float e, ep;
                    float3 fij = dp * pair13<false>(dot3(dp, dp), sREQ[ing], sREQ[jng], x13, cu.Rc2, cu.kq, cu.rc, e, ep);
                    if (flags & F_CLAMP_NB) { const float ff = dot3(fij, fij); if (ff > P.Fmax2NB) fij = fij * sqrtf(P.Fmax2NB / ff); }
                    f13 = f13 + fij;
                }
            }
        }
        // sums over the node's four lanes
        float3 fa = fb;
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            fa.x += __shfl_xor_sync(0xffffffffu, fa.x, o); fa.y += __shfl_xor_sync(0xffffffffu, fa.y, o);
            fa.z += __shfl_xor_sync(0xffffffffu, fa.z, o);
            fpi.x += __shfl_xor_sync(0xffffffffu, fpi.x, o); fpi.y += __shfl_xor_sync(0xffffffffu, fpi.y, o);
            fpi.z += __shfl_xor_sync(0xffffffffu, fpi.z, o);
        }
        if (!ok) return;
        float4* fasm = at<float4>(L.fasm);
        float4* fng = at<float4>(L.fng);
        fng[n4] = make_float4(fb.x + f13.x, fb.y + f13.y, fb.z + f13.z, 0.f);
        fng[4 * L.maxNN + n4] = make_float4(fps.x, fps.y, fps.z, 0.f);
        if (q == 0) fasm[ia] = make_float4(-fa.x, -fa.y, -fa.z, 0.f);
        if (q == 1) fasm[natoms + ia] = make_float4(fpi.x, fpi.y, fpi.z, 0.f);
    }

    // ------------------------------------------------------------------ forces
    template <bool HB>
    __device__ __forceinline__ void pairs(bool pbc, long long* facc) {
        ordered_pairs<HB>(pbc && !(P.Rc2 > 0.f), facc);
        if (nlist > 0) list_pairs<HB>(at<float4>(L.pos), at<float4>(L.REQ), facc);
    }

    // moved: some atom moved more than half the list skin since the lists were
    // built (block-uniform, from the previous step's move)
    __device__ void forces(bool moved) {
        const int flags = P.flags;
        const float4* spos = at<float4>(L.pos);
        const bool pbc = (flags & F_PBC) != 0;
        long long* facc = sums();
        if ((flags & F_NONBONDED) && P.Rc2 > 0.f && L.nimg > 0) {
            if (listok && (!listed || moved)) {
                if (COUNT && tid == 0) atomicAdd(Y.counters + 3, 1ull);
                listok = listed = list_build(spos);
            }
            if (!listok) {
                nlist = 0;
                bbox_from_smem();
                bool any = false;
                for (int k = 0; k < L.nimg; k++) {
                    const int ipbc = image_index(k), nxi = 2 * P.npbc[0] + 1, nyi = 2 * P.npbc[1] + 1;
                    any |= image_within(ipbc % nxi - P.npbc[0], (ipbc / nxi) % nyi - P.npbc[1], ipbc / (nxi * nyi) - P.npbc[2], P.Rc2);
                }
                if (any) {
                    build_candidates(P.Rc2);
                    if (hasH) candidate_rows<true>(spos, at<float4>(L.REQ), facc);
                    else candidate_rows<false>(spos, at<float4>(L.REQ), facc);
                    __syncthreads();                 // the lists share the recoil slots' memory
                }
            }
            if (COUNT && tid == 0 && listok) atomicAdd(Y.counters + 4, (unsigned long long)nlist);
        }
        // Bonded terms and GridFF samples in units of one warp (eight nodes, or
        // eight atoms), dealt to the warps in turn; nothing waits between these
        // units and the pairs.
        float4* fgr = at<float4>(L.fgrid);
        const int nB = (nnode + 7) >> 3, nG = (flags & F_GRID) ? (natoms + 7) >> 3 : 0;
#pragma unroll 1
        for (int u = warp; u < nB; u += NW) {
            const int ia = 8 * u + (lane >> 2);
            bonded_node(min(ia, nnode - 1), ia < nnode);
        }
        double d0 = 0.0;
        if constexpr (CL) {
#pragma unroll 1
            for (int u = cr + cn * warp; u < nG; u += cn * NW) {
                B::template grid_phase<false, true>(32 * u + lane, 1 << 30, fgr, d0);
                __syncwarp();
                const int a = 8 * u + lane;
                if (lane < 8 && a < natoms) fix_add(facc + 3 * a, f3(fgr[a]));
            }
        } else {
#pragma unroll 1
            for (int u = (warp + NW - nB % NW) % NW; u < nG; u += NW)
                B::template grid_phase<false, true>(32 * u + lane, 1 << 30, fgr, d0);
        }
        if (flags & F_NONBONDED) {
            if (hasH) pairs<true>(pbc, facc);
            else pairs<false>(pbc, facc);
        }
        // direct substrate term (getSurfMorse), one thread per atom
        if (flags & F_SURF) {
            __syncthreads();
            const float4* sR = at<float4>(L.REQ);
            for (int a = tid; a < natoms; a += T) {
                const float4 p = spos[a];
                const float4 r = surf_atom(P, make_float3(p.x + lv[9], p.y + lv[10], p.z + lv[11]), sR[a]);
                const float4 g = (!CL && (flags & F_GRID)) ? fgr[a] : make_float4(0.f, 0.f, 0.f, 0.f);
                fgr[a] = make_float4(g.x + r.x, g.y + r.y, g.z + r.z, 0.f);
            }
        }
        if (CL && pairbad) flags_cl()[par] = 1;
    }

    // ---------------------------------------------------------------- assemble
    // assemble + clamp; FP64 partial sums of (vf, vv, ff) and max|f|^2 for this
    // thread; the pair sums are read and cleared for the next step
    __device__ void assemble(double& vf, double& vv, double& ff, float& fmax2, bool& bad) {
        float4* fasm = at<float4>(L.fasm);
        long long* facc = sums();
        const float4* fgr = at<float4>(L.fgrid);
        const float4* flist = at<float4>(L.flist);
        const float4* fng = at<float4>(L.fng);
        const float4* spos = at<float4>(L.pos);
        const float4* svel = B::vels();
        const float Fl2 = P.Flim * P.Flim;
        for (int v = tid; v < nvecs; v += T) {
            const bool pi = v >= natoms;
            const int ia = pi ? v - natoms : v;
            float3 f = make_float3(0.f, 0.f, 0.f);
            if (pi || v < nnode) f = f3(fasm[v]);
            if (!pi) {
                if (P.flags & (CL ? F_SURF : F_GRID | F_SURF)) f = f + f3(fgr[v]);
                if (!CL && nlist > 0) f = f + f3(flist[v]);
                long long s[3] = {0, 0, 0};
                if constexpr (CL) {
                    for (int c = 0; c < cn; c++) {
                        const long long* q = cooperative_groups::this_cluster().map_shared_rank(facc, c) + 3 * v;
                        s[0] += q[0]; s[1] += q[1]; s[2] += q[2];
                    }
                    long long* z = at<long long>(L.facc) + (par ^ 1) * 3 * L.maxNA + 3 * v;
                    z[0] = 0; z[1] = 0; z[2] = 0;
                } else {
                    s[0] = facc[3 * v]; s[1] = facc[3 * v + 1]; s[2] = facc[3 * v + 2];
                    facc[3 * v] = 0; facc[3 * v + 1] = 0; facc[3 * v + 2] = 0;
                }
                f.x += (float)s[0] * (1.f / kFix);
                f.y += (float)s[1] * (1.f / kFix);
                f.z += (float)s[2] * (1.f / kFix);
            }
            const int4 bk = bks(ia);
            const int bks[4] = {bk.x, bk.y, bk.z, bk.w};
            const float4* slots = pi ? fng + 4 * L.maxNN : fng;
            float4 rec[4];                               // all four loads in flight, sums in slot order
#pragma unroll
            for (int k = 0; k < 4; k++) rec[k] = slots[max(bks[k], 0)];
            bool live = true;                            // slots end at the first empty one
#pragma unroll
            for (int k = 0; k < 4; k++) {
                live &= bks[k] >= 0;
                if (live) f = f + f3(rec[k]);
            }
            const float4 p = spos[v];
            if (pi) f = fma3(f3(p), -dot3(f, f3(p)), f);      // Vec3::makeOrthoU
            if ((P.flags & F_BCONS) && !pi) f = bond_constraint_force(Y, isys, v, spos, lv, f);
            if (P.Flim > 0.f) {
                const float fr2 = dot3(f, f);
                if (fr2 > Fl2) f = f * (P.Flim * rsqrtf(fr2));
            }
            if ((P.flags & F_CONSTR) && !pi) f = constraint_force(Y, aoff + v, f3(p), f);
            // a system whose atoms left any sensible range (no force clamp,
            // bad start) is retired like a non-finite one
            if (!pi) bad |= !(fabsf(p.x) + fabsf(p.y) + fabsf(p.z) < 1e5f);
            fasm[v] = make_float4(f.x, f.y, f.z, 0.f);
            const float4 vv4 = svel[v];
            vf += (double)vv4.x * f.x + (double)vv4.y * f.y + (double)vv4.z * f.z;
            vv += (double)vv4.x * vv4.x + (double)vv4.y * vv4.y + (double)vv4.z * vv4.z;
            const double f2 = (double)f.x * f.x + (double)f.y * f.y + (double)f.z * f.z;
            ff += f2;
            fmax2 = fmaxf(fmax2, (float)f2);
            bad |= !isfinite(f.x + f.y + f.z);
        }
        if constexpr (CL) {
            bad |= any_cl(par);
            if (tid == 0) flags_cl()[par ^ 1] = 0;
            par ^= 1;
        } else {
            bad |= pairbad;
        }
    }

    // block reduction of 3 doubles + one float max (+flag); result in all threads
    __device__ void reduce4(double& a, double& b, double& c, float& m, bool& bad) {
        double* red = at<double>(L.red);
        a = wsum(a); b = wsum(b); c = wsum(c);
        m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));      // m >= 0: bits order like values
        const int anybad = __any_sync(0xffffffffu, bad);
        if (lane == 0) {
            red[4 * warp + 0] = a; red[4 * warp + 1] = b; red[4 * warp + 2] = c;
            reinterpret_cast<float*>(red + 4 * warp + 3)[0] = m;
            reinterpret_cast<int*>(red + 4 * warp + 3)[1] = anybad;
        }
        __syncthreads();
        a = 0; b = 0; c = 0; m = 0.f; int nb = 0;
#pragma unroll
        for (int w = 0; w < NW; w++) {
            a += red[4 * w + 0]; b += red[4 * w + 1]; c += red[4 * w + 2];
            m = fmaxf(m, reinterpret_cast<const float*>(red + 4 * w + 3)[0]);
            nb |= reinterpret_cast<const int*>(red + 4 * w + 3)[1];
        }
        bad = nb != 0;
    }

    // -------------------------------------------------------------------- move
    // a moved atom: its copy in the pair arrays, and whether it left the
    // neighbourhood (half the skin) of its position at the lists' build
    __device__ __forceinline__ bool moved_atom(int v, float3 p) {
        soa(0)[v] = p.x; soa(1)[v] = p.y; soa(2)[v] = p.z;
        if (!listed) return false;
        const float* vp = at<float>(L.vp);
        const float dx = p.x - vp[v], dy = p.y - vp[L.maxNA + v], dz = p.z - vp[2 * L.maxNA + v];
        return !(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) <= 0.25f * P.vskin * P.vskin);
    }

    __device__ bool move(double dt, double cv, double cfm) {
        float4* spos = at<float4>(L.pos);
        float4* svel = B::vels();
        const float4* fasm = at<float4>(L.fasm);
        const float dtf = (float)dt;
        const float cvf = (float)cv;
        const float kf = (float)((double)dtf + cfm);
        bool far = false;
        for (int v = tid; v < nvecs; v += T) {
            float3 f = f3(fasm[v]), ve = f3(svel[v]), p = f3(spos[v]);
            const bool bPi = v >= natoms;
            if (bPi) f = fma3(p, -dot3(p, f), f);
            ve = ve * cvf;
            ve = fma3(f, kf, ve);
            if (bPi) ve = fma3(p, -dot3(p, ve), ve);
            p = fma3(ve, dtf, p);
            if (bPi) p = p * rsqrtf(dot3(p, p));
            spos[v] = make_float4(p.x, p.y, p.z, 0.f);
            svel[v] = make_float4(ve.x, ve.y, ve.z, 0.f);
            if (!bPi) far |= moved_atom(v, p);
        }
        return far;
    }

    // Langevin step (MMFFsp3_loc::move_atom_Langevin, MMFFsp3_loc.h:1191-1216):
    // f - gamma v + uniform(-1,1) * sqrt(2 kB T gamma / dt), then v += f dt,
    // p += v dt; pi vectors keep unit length and stay orthogonal to their force
    __device__ bool move_md(int step) {
        float4* spos = at<float4>(L.pos);
        float4* svel = B::vels();
        const float4* fasm = at<float4>(L.fasm);
        const float dt = P.md_dt, g = P.md_gamma, nz = P.md_noise;
        bool far = false;
        for (int v = tid; v < nvecs; v += T) {
            float3 f = f3(fasm[v]), ve = f3(svel[v]), p = f3(spos[v]);
            const bool bPi = v >= natoms;
            if (bPi) f = fma3(p, -dot3(p, f), f);
            f = fma3(ve, -g, f);
            const long long gv = (long long)voff + v;
            f.x = fmaf(langevin_rand(P.md_seed, gv, step, 0), nz, f.x);
            f.y = fmaf(langevin_rand(P.md_seed, gv, step, 1), nz, f.y);
            f.z = fmaf(langevin_rand(P.md_seed, gv, step, 2), nz, f.z);
            ve = fma3(f, dt, ve);
            if (bPi) ve = fma3(p, -dot3(p, ve), ve);
            p = fma3(ve, dt, p);
            if (bPi) p = p * rsqrtf(dot3(p, p));
            spos[v] = make_float4(p.x, p.y, p.z, 0.f);
            svel[v] = make_float4(ve.x, ve.y, ve.z, 0.f);
            if (!bPi) far |= moved_atom(v, p);
        }
        return far;
    }

    // copy of the positions just moved (each thread its own vectors, as in move)
    __device__ void snapshot() {
        const float4* spos = at<float4>(L.pos);
        for (int v = tid; v < nvecs; v += T) Y.minpos[voff + v] = spos[v];
    }

    __device__ void store_state(int status, int steps, float fconv, double dt, double damping, int lastNeg, double total) {
        const float4* spos = at<float4>(L.pos);
        const float4* svel = B::vels();
        const float4* fasm = at<float4>(L.fasm);
        for (int v = tid; v < nvecs; v += T) {
            Y.pos[voff + v] = spos[v];
            if (L.vel >= 0) Y.vel[voff + v] = svel[v];
            Y.force[voff + v] = fasm[v];
        }
        if (tid == 0) {
            Y.fire[isys] = make_double4(dt, damping, (double)lastNeg, total);
            Y.status[isys] = status;
            Y.nsteps[isys] = steps;
            Y.fconv[isys] = fconv;
        }
    }
};

// ---------------------------------------------------------------------------
// Persistent relaxation: claims systems from queue[] via counter.
// resident CTAs per SM the register allocation of the relax kernel targets,
// per thread count (build options; without a target ptxas caps at 128
// registers and spills)
#ifndef MMFF_MINB_T32
#define MMFF_MINB_T32 16
#endif
#ifndef MMFF_MINB_T64
#define MMFF_MINB_T64 8
#endif
#ifndef MMFF_MINB_T128
#define MMFF_MINB_T128 4
#endif
#ifndef MMFF_MINB_T256
#define MMFF_MINB_T256 2
#endif
template <int T> constexpr int relax_min_blocks() {
    return T == 32 ? MMFF_MINB_T32 : T == 64 ? MMFF_MINB_T64 : T == 128 ? MMFF_MINB_T128 : T == 256 ? MMFF_MINB_T256 : 1;
}

// P.vlist (null: none): scratch for the shifted-image pair lists, P.vcap entries per CTA.
// EXPL: the exploring cycle (P.md_mode 2) instead of plain FIRE or the drive.
template <int T, bool COUNT, bool EXPL, bool CL = false>
__global__ void __launch_bounds__(T, relax_min_blocks<T>()) relax_kernel(const __grid_constant__ Params P, const __grid_constant__ Systems Y, const int* __restrict__ queue, int nqueue,
                                                  int* counter, const __grid_constant__ SmemLayout L) {
    extern __shared__ __align__(16) char smem[];
    __shared__ int s_claim;
    RelaxEngine<T, COUNT, CL> E(P, Y, smem, L);
    if constexpr (CL) E.csync();        // the whole cluster runs before anyone writes to a neighbour
    while (true) {
        if constexpr (CL) {
            if (E.cr == 0 && threadIdx.x == 0) {
                const int c = atomicAdd(counter, 1);
                for (int k = 0; k < E.cn; k++) *cooperative_groups::this_cluster().map_shared_rank(&s_claim, k) = c;
            }
        } else if (threadIdx.x == 0) {
            s_claim = atomicAdd(counter, 1);
        }
        E.csync();
        const int q = s_claim;
        if (q >= nqueue) break;
        const int s = queue[q];
        E.load(s);
        const double4 fs = Y.fire[s];
        double dt = fs.x, damping = fs.y;
        int lastNeg = (int)fs.z;
        __syncthreads();
        int status = ST_MAXSTEPS, itr = 0;
        double meas2 = 0.0;         // convergence measure squared
        bool far = false;           // pair lists out of date (block-uniform)
        int ph = 0;                 // exploring cycle: 2 * (steps in the phase) + exploring
        if constexpr (EXPL) { const int4 g = Y.gopt[s]; ph = 2 * g.y + (g.x != 0); }
        for (itr = 0; itr < P.nstep_max; itr++) {
            bool lang = false;      // an exploring step (Langevin instead of FIRE)
            if constexpr (EXPL) {
                const int ev = explore_step(ph, P.n_explore, P.n_relax);
                lang = ev & 1;
                if ((ev & 2) && threadIdx.x == 0) Y.gopt[s].w++;
            }
            E.forces(far);
            E.csync();
            double vf = 0, vv = 0, ff = 0;
            float fmax2 = 0.f;
            bool bad = false;
            E.assemble(vf, vv, ff, fmax2, bad);
            E.reduce4(vf, vv, ff, fmax2, bad);
            if (bad) { status = ST_NAN; break; }
            if (!EXPL && P.md_mode) {   // Langevin drive: fixed number of steps, no FIRE
                far = E.move_md(P.md_step0 + itr);
                meas2 = (double)fmax2;
                far = __syncthreads_or(far) != 0;
                continue;
            }
            // DynamicOpt::FIRE_update_params (FP64, identical in every thread; the
            // sign of cos(v, f) is that of v.f); in the exploring cycle the FIRE
            // scalars evolve in exploring steps too (MolWorld_sp3.h:2401-2424)
            const double renorm_vf = length_ratio(vv, ff);
            double cv, cf;
            if (vf < 0.0) { cv = P.cv_kill; cf = 0.0; } else { cv = 1.0 - damping; cf = damping; }
            cf = renorm_vf * cf;
            if (vf < 0.0) {
                dt = fmax(dt * P.fdec, P.dt_min);
                lastNeg = 0;
                damping = P.damp_max;
            } else {
                if (lastNeg > P.minLastNeg) { dt = fmin(dt * P.finc, P.dt_max); damping = damping * P.falpha; }
                lastNeg++;
            }
            if (EXPL && lang) far = E.move_md(P.md_step0 + itr);
            else far = E.move(dt, cv, P.fire_variant == 1 ? cf : renorm_vf * cf);
            const double m = (P.conv_mode == 0) ? ff : (double)fmax2;
            meas2 = m;
            if constexpr (EXPL) {
                if (!lang && m < P.Fconv2) {
                    // a minimum (MolWorld_sp3.h:2465-2473): keep it, start exploring
                    E.snapshot();
                    if (threadIdx.x == 0) Y.gopt[s].z++;
                    ph = 1;
                }
            } else {
                if (m < P.Fconv2) { status = ST_CONVERGED; itr++; break; }
            }
            far = __syncthreads_or(far) != 0;   // the end-of-step barrier
        }
        // converged at step itr-1 (reference returns the loop index at break)
        const int steps = (status == ST_CONVERGED) ? itr - 1 : itr;
        __syncthreads();
        if (CL && E.cr != 0) { E.csync(); continue; }      // every CTA has the same state: the first writes it
        // (a system retired as not finite had no move in its last step)
        E.store_state(status, steps, (float)sqrt(meas2), dt, damping, lastNeg, fs.w + (double)itr);
        if (EXPL && threadIdx.x == 0) { Y.gopt[s].x = ph & 1; Y.gopt[s].y = ph >> 1; }
        if (COUNT) {
            // force evaluations done for this system: itr loop iterations
            if (threadIdx.x == 0) {
                atomicAdd(Y.counters + 1, (unsigned long long)itr * (unsigned long long)E.natoms);
                atomicAdd(Y.counters + 2, (unsigned long long)itr);
            }
        }
        E.csync();
    }
    if (COUNT) atomicAdd(Y.counters, E.npair);
}

// address of the kernel instantiation for T threads
template <bool COUNT, bool EXPL> static void* relax_of(int T) {
    switch (T) {
        case 32: return (void*)relax_kernel<32, COUNT, EXPL>;
        case 64: return (void*)relax_kernel<64, COUNT, EXPL>;
        case 128: return (void*)relax_kernel<128, COUNT, EXPL>;
        case 256: return (void*)relax_kernel<256, COUNT, EXPL>;
        case 512: return (void*)relax_kernel<512, COUNT, EXPL>;
        default: return nullptr;
    }
}
// ... by a cluster of CTAs per system
void* relax_cluster_fn(int T) {
    switch (T) {
        case 128: return (void*)relax_kernel<128, false, false, true>;
        case 256: return (void*)relax_kernel<256, false, false, true>;
        case 512: return (void*)relax_kernel<512, false, false, true>;
        default: return nullptr;
    }
}
void* relax_fn(int T, bool count) { return count ? relax_of<true, false>(T) : relax_of<false, false>(T); }
void* relax_explore_fn(int T) { return relax_of<false, true>(T); }

}  // namespace mmff
