// mmff_relax.cu -- persistent relaxation kernels for sm_100a, one CTA per system.
//
// The system's whole state (positions, velocities, topology, force-field
// parameters, recoil slots) is staged in shared memory, and every FIRE step
// runs inside the CTA with three block barriers:
//   forces   units of one warp, claimed in turn: bonded terms (a node per lane),
//            pair tiles, runs of the pair lists, GridFF samples (4 lanes per atom)
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
// A relaxation amplifies the last bit of a force: two or three molecules of a few
// hundred part after some hundred steps, and the largest differences reach the
// size of a bond.  So every FP32 sum here has a fixed order that depends on the
// system alone, not on the block size, the cluster or which warp takes a unit:
// partial sums over a tile or a run of list entries go to 64-bit integer totals,
// everything else is summed by one lane.  The packed instructions below take two
// independent sums side by side, never two terms of one sum.
#include "mmff_pairs.cuh"

#include <cooperative_groups.h>

namespace mmff {

// ---- packed FP32 pairs (sm_100: one instruction, two IEEE operations)
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) { f32x2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { f32x2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) { f32x2 d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ float lo2(f32x2 v) { float a, b; unpack2(v, a, b); return a; }
__device__ __forceinline__ float hi2(f32x2 v) { float a, b; unpack2(v, a, b); return b; }
__device__ __forceinline__ f32x2 neg2(f32x2 v) { return v ^ 0x8000000080000000ull; }

// two atoms side by side.  x, y, z of an own atom are the negatives, so that
// d = p_j - p_i is one addition; its Q is the negative too (see force2)
struct Atom2 { f32x2 x, y, z, R, E, Q, H; };
struct PairC { f32x2 nkq, m12, m1; float Rc2; };

__device__ __forceinline__ Atom2 atom2(float4 p0, float4 R0, float4 p1, float4 R1) {
    Atom2 a;
    a.x = pack2(p0.x, p1.x); a.y = pack2(p0.y, p1.y); a.z = pack2(p0.z, p1.z);
    a.R = pack2(R0.x, R1.x); a.E = pack2(R0.y, R1.y); a.Q = pack2(R0.z, R1.z); a.H = pack2(R0.w, R1.w);
    return a;
}
__device__ __forceinline__ Atom2 own2(float4 p0, float4 R0, float4 p1, float4 R1) {
    Atom2 a = atom2(p0, R0, p1, R1);
    a.x = neg2(a.x); a.y = neg2(a.y); a.z = neg2(a.z); a.Q = neg2(a.Q);
    return a;
}

// Two pairs: d = p_j - p_i and the scalar F of pair_force (mmff_device.cuh), operation
// for operation in both halves (signs moved between factors do not round).
// ex0, ex1: pair excluded.
template <bool HB>
__device__ __forceinline__ f32x2 force2(const Atom2& j, const Atom2& i, const PairC& c, bool ex0, bool ex1, f32x2& dx,
                                        f32x2& dy, f32x2& dz, bool& ok0, bool& ok1) {
    dx = add2(j.x, i.x); dy = add2(j.y, i.y); dz = add2(j.z, i.z);
    const f32x2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
    float a, b;
    unpack2(r2, a, b);
    ok0 = !ex0 && a < c.Rc2;
    ok1 = !ex1 && b < c.Rc2;
    a = ok0 ? a : 1e30f;
    b = ok1 ? b : 1e30f;
    const f32x2 ir = pack2(rsq(a), rsq(b));
    const f32x2 ir2 = mul2(ir, ir);
    const f32x2 R0 = add2(i.R, j.R);
    const f32x2 nQ = mul2(i.Q, j.Q);
    const f32x2 u2 = mul2(mul2(R0, R0), ir2);
    const f32x2 u6 = mul2(mul2(u2, u2), u2);
    const f32x2 vdW = mul2(u6, mul2(i.E, j.E));
    f32x2 X;
    if (HB) {
        float h0, h1;
        unpack2(mul2(i.H, j.H), h0, h1);
        X = fma2(add2(u6, c.m1), vdW, mul2(mul2(u6, vdW), pack2(fminf(h0, 0.f), fminf(h1, 0.f))));
    } else {
        X = mul2(add2(u6, c.m1), vdW);
    }
    const f32x2 F = fma2(mul2(c.m12, ir2), X, mul2(mul2(nQ, ir), ir2));
    return fma2(mul2(nQ, c.nkq), ir, F);
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
// share of the tiles, list runs, image rows and GridFF samples.  Fixed-point sums
// are added over all CTAs in assemble, through distributed shared memory; what one
// lane summed (an atom's grid force, its image rows) is read from the CTA that has
// it.  So all CTAs get the same bits, and with the same code on the same bits they
// take every decision alike: the cluster barrier after the forces is the only one
// of a step.  Two sets of sums alternate, so that the next step's writes never meet
// a neighbour that still reads.  A non-finite pair force, which one CTA alone sees,
// is exchanged before it decides anything.
template <int T, bool COUNT, bool CL = false>
struct RelaxEngine : PairEngine<T, 1, false, COUNT, true> {
    using B = PairEngine<T, 1, false, COUNT, true>;
    using B::P; using B::Y; using B::L; using B::tid; using B::lane; using B::warp;
    using B::isys; using B::natoms; using B::nnode; using B::nvecs; using B::aoff; using B::noff; using B::voff;
    using B::lv; using B::hasH; using B::hasX; using B::xrow; using B::nbw; using B::pairbad; using B::kFix; using B::kFixMax;
    using B::ngs; using B::ngc; using B::bks; using B::image_within; using B::build_candidates; using B::fix_add;
    using B::image_excluded; using B::bbox_from_smem; using B::npair; using B::tile_mask; using B::bbmin; using B::bbmax;
    template <class X> __device__ __forceinline__ X* at(int off) { return B::template at<X>(off); }
    static constexpr int NW = T / 32;
    // shifted-image pair lists of the current system (block-uniform)
    enum { LIST_NONE, LIST_QUIET, LIST_BUILT };     // QUIET: no image within cutoff + skin of the positions vp
    bool listok = false;               // usable (a scratch slot, no overflow so far)
    int lstate = LIST_NONE;
    int nlist = 0;                     // entries
    bool use_list = false;             // this step evaluates them
    int cr = 0, cn = 1, par = 0;       // CL: rank in the cluster, its size; which set of sums (and unit counter) this step uses

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
    __device__ __forceinline__ float4* gridf() { return at<float4>(L.fgrid) + (CL ? par * L.maxNA : 0); }
    __device__ __forceinline__ float4* listf() { return at<float4>(L.flist) + (CL ? par * L.maxNA : 0); }
    // [0, 1] a non-finite pair force (CL, per set of sums), [2, 3] units claimed (per step parity)
    __device__ __forceinline__ int* shared_ints() const {
        __shared__ int f[4];
        return f;
    }
    // some CTA of the cluster set flag k
    __device__ __forceinline__ bool any_cl(int k) const {
        int a = 0;
        if constexpr (CL)
            for (int c = 0; c < cn; c++) a |= cooperative_groups::this_cluster().map_shared_rank(shared_ints(), c)[k];
        return a != 0;
    }

    // pair forces beside the fixed-point sums: the small systems' whole pair sums, else
    // without a cutoff the image rows
    __device__ __forceinline__ bool image_row_path() const { return (P.flags & F_PBC) && !(P.Rc2 > 0.f) && !L.small; }
    __device__ __forceinline__ bool has_listf() const { return (P.flags & F_NONBONDED) && (L.small || image_row_path()); }

    __device__ void load(int s) {
        B::load(s);
        listok = P.vlist != nullptr && natoms <= 4096 && P.Rc2 > 0.f && L.nimg > 0 && L.nimg <= kListMaxImages &&
                 (P.flags & F_NONBONDED);
        lstate = LIST_NONE;
        nlist = 0;
        use_list = false;
        par = 0;
        __syncthreads();
        if (L.shf >= 0 && tid < L.nimg) {
            const float3 sh = image_of(image_index(tid));
            at<float4>(L.shf)[tid] = make_float4(sh.x, sh.y, sh.z, 0.f);
        }
        long long* facc = at<long long>(L.facc);
        for (int a = tid; a < 3 * natoms; a += T) facc[a] = 0;
        if constexpr (CL)
            for (int a = tid; a < 3 * natoms; a += T) facc[3 * L.maxNA + a] = 0;
        if (tid < 4) shared_ints()[tid] = 0;
    }
    __device__ __forceinline__ PairC pair_consts() const {
        PairC C;
        C.Rc2 = P.Rc2 > 0.f ? P.Rc2 : 3.0e38f;
        C.nkq = pack2(-P.kq_rc2, -P.kq_rc2); C.m12 = pack2(-12.f, -12.f); C.m1 = pack2(-1.f, -1.f);
        return C;
    }

    // ---- central image, two 32 x 32 tiles at a time ---------------------------
    // Tiles of PairEngine (off_tile, diag_tile), sums in the same order: lane l owns
    // atom i of block bi0 and one of block bi1, the atoms j of block bj0 (and bj1)
    // rotate past it, the reactions with them.  KIND 0: both tiles have block bj0, so
    // that a j is loaded once for both; 1: two unrelated tiles; 2: two diagonal ones.
    // A block < 0: no second tile.
    // Bound: the FP32 pipe (29 packed operations) and issue (about 60) a rotation step
    // of 64 unordered pairs.
    template <bool HB, int KIND>
    __device__ void tile2(int bi0, int bi1, int bj0, int bj1, long long* facc) {
        const float4* spos = at<float4>(L.pos);
        const float4* sREQ = at<float4>(L.REQ);
        const PairC C = pair_consts();
        const int last = natoms - 1;
        const int i0 = 32 * bi0 + lane, i1 = 32 * bi1 + lane;
        const bool v0 = i0 < natoms, v1 = bi1 >= 0 && i1 < natoms;
        const int a0 = v0 ? i0 : 0, a1 = v1 ? i1 : 0;
        const Atom2 I = own2(spos[a0], sREQ[a0], spos[a1], sREQ[a1]);
        // excluded j by rotation step
        uint32_t m0 = v0 ? __ldg(xrow + i0 * nbw + bj0) : ~0u, m1 = v1 ? __ldg(xrow + i1 * nbw + (KIND == 0 ? bj0 : bj1)) : ~0u;
        m0 = __funnelshift_r(m0, m0, lane);
        m1 = __funnelshift_r(m1, m1, lane);
        const int b0 = 32 * bj0, b1 = KIND == 0 ? b0 : 32 * max(bj1, 0);
        f32x2 fx = 0, fy = 0, fz = 0, rx = 0, ry = 0, rz = 0;
        const int nxt = (lane + 1) & 31;
        constexpr int s0 = KIND == 2 ? 1 : 0, s1 = KIND == 2 ? 17 : 32;
        if (KIND == 2) { m0 >>= 1; m1 >>= 1; }
#pragma unroll 2
        for (int s = s0; s < s1; s++) {
            const int jl = (lane + s) & 31;
            const int j0 = min(b0 + jl, last);
            const float4 p0 = spos[j0], R0 = sREQ[j0];
            Atom2 J;
            if (KIND == 0) {
                J = atom2(p0, R0, p0, R0);
            } else {
                const int j1 = min(b1 + jl, last);
                J = atom2(p0, R0, spos[j1], sREQ[j1]);
            }
            const bool half = KIND == 2 && s == 16 && lane >= 16;
            f32x2 dx, dy, dz;
            bool ok0, ok1;
            const f32x2 F = force2<HB>(J, I, C, (m0 & 1u) || half, (m1 & 1u) || half, dx, dy, dz, ok0, ok1);
            m0 >>= 1; m1 >>= 1;
            if (COUNT) npair += (ok0 ? 2 : 0) + (ok1 ? 2 : 0);
            fx = fma2(dx, F, fx); fy = fma2(dy, F, fy); fz = fma2(dz, F, fz);
            const f32x2 nF = neg2(F);
            if (KIND == 2) {
                const int src = (lane - s) & 31;     // the lane whose partner this lane's atoms were
                const f32x2 gx = mul2(dx, nF), gy = mul2(dy, nF), gz = mul2(dz, nF);
                fx = add2(fx, __shfl_sync(0xffffffffu, gx, src));
                fy = add2(fy, __shfl_sync(0xffffffffu, gy, src));
                fz = add2(fz, __shfl_sync(0xffffffffu, gz, src));
            } else {
                rx = __shfl_sync(0xffffffffu, fma2(dx, nF, rx), nxt);
                ry = __shfl_sync(0xffffffffu, fma2(dy, nF, ry), nxt);
                rz = __shfl_sync(0xffffffffu, fma2(dz, nF, rz), nxt);
            }
        }
        if (v0) fix_add(facc + 3 * i0, make_float3(lo2(fx), lo2(fy), lo2(fz)));
        if (v1) fix_add(facc + 3 * i1, make_float3(hi2(fx), hi2(fy), hi2(fz)));
        if (KIND != 2) {
            const int j0 = b0 + lane, j1 = b1 + lane;
            if (j0 < natoms) fix_add(facc + 3 * j0, make_float3(lo2(rx), lo2(ry), lo2(rz)));
            if (bi1 >= 0 && j1 < natoms) fix_add(facc + 3 * j1, make_float3(hi2(rx), hi2(ry), hi2(rz)));
        }
    }
    // units of tiles: doubles (2m, 2m + 1 | bj), the tiles (bj - 1, bj) of odd bj in
    // pairs, the diagonal ones in pairs
    __device__ __forceinline__ int double_tiles() const { return ((nbw - 1) / 2) * (nbw / 2); }
    __device__ __forceinline__ int single_units() const { return (nbw / 2 + 1) >> 1; }
    __device__ __forceinline__ int diag_units() const { return (nbw + 1) >> 1; }
    template <bool HB>
    __device__ void tile_unit(int u, long long* facc) {
        const int nd = double_tiles(), ns = single_units();
        if (u < nd) {
            int bj = 2;
            while (u >= bj / 2) { u -= bj / 2; bj++; }
            tile2<HB, 0>(2 * u, 2 * u + 1, bj, bj, facc);
        } else if (u < nd + ns) {
            const int b = 4 * (u - nd);
            const bool two = b + 3 < nbw;
            tile2<HB, 1>(b, two ? b + 2 : -1, b + 1, two ? b + 3 : -1, facc);
        } else {
            const int d = 2 * (u - nd - ns), d1 = d + 1 < nbw ? d + 1 : -1;
            tile2<HB, 2>(d, d1, d, d1, facc);
        }
    }

    // ---- shifted images -------------------------------------------------------
    // shifted image k (0 .. nimg-1, without the central one) -> image index with it, and its shift
    __device__ __forceinline__ int image_index(int k) const { return k < L.nimg / 2 ? k : k + 1; }
    __device__ __forceinline__ float3 image_of(int ipbc) const {
        const int nxi = 2 * P.npbc[0] + 1, nyi = 2 * P.npbc[1] + 1;
        return image_shift(lv, ipbc % nxi - P.npbc[0], (ipbc / nxi) % nyi - P.npbc[1], ipbc / (nxi * nyi) - P.npbc[2]);
    }
    // some shifted image within sqrt(R2) of the box of the atoms
    __device__ __forceinline__ bool any_image(float R2) const {
        bool any = false;
        const int nxi = 2 * P.npbc[0] + 1, nyi = 2 * P.npbc[1] + 1;
        for (int k = 0; k < L.nimg; k++) {
            const int ipbc = image_index(k);
            any |= image_within(ipbc % nxi - P.npbc[0], (ipbc / nxi) % nyi - P.npbc[1], ipbc / (nxi * nyi) - P.npbc[2], R2);
        }
        return any;
    }

    // Without a cutoff: atoms i of unit u (64 of them, two per lane) against all atoms of
    // every shifted image, images and atoms j in order; each atom's sum in one accumulator.
    template <bool HB>
    __device__ void image_row_unit(int u, float4* out) {
        const float4* spos = at<float4>(L.pos);
        const float4* sREQ = at<float4>(L.REQ);
        const PairC C = pair_consts();
        const int i0 = 64 * u + lane, i1 = i0 + 32;
        const bool v0 = i0 < natoms, v1 = i1 < natoms;
        const int a0 = v0 ? i0 : 0, a1 = v1 ? i1 : 0;
        const float4 p0 = spos[a0], p1 = spos[a1];
        Atom2 I = own2(p0, sREQ[a0], p1, sREQ[a1]);
        const int4 g0 = ngs(a0), c0 = ngc(a0), g1 = ngs(a1), c1 = ngc(a1);
        const int nim = (2 * P.npbc[0] + 1) * (2 * P.npbc[1] + 1) * (2 * P.npbc[2] + 1), central = nim / 2;
        f32x2 fx = 0, fy = 0, fz = 0;
        for (int im = 0; im < nim; im++) {
            if (im == central) continue;
            const float3 s = image_of(im);
            I.x = pack2(s.x - p0.x, s.x - p1.x); I.y = pack2(s.y - p0.y, s.y - p1.y); I.z = pack2(s.z - p0.z, s.z - p1.z);
            auto cell = [&](int c, int g) { return c == im ? g : -1; };
            const int e0 = cell(c0.x, g0.x), e1 = cell(c0.y, g0.y), e2 = cell(c0.z, g0.z), e3 = cell(c0.w, g0.w);
            const int h0 = cell(c1.x, g1.x), h1 = cell(c1.y, g1.y), h2 = cell(c1.z, g1.z), h3 = cell(c1.w, g1.w);
            const bool bonds = __any_sync(0xffffffffu, max(max(max(e0, e1), max(e2, e3)), max(max(h0, h1), max(h2, h3))) >= 0);
            auto pass = [&](auto excl) {
#pragma unroll 2
                for (int j = 0; j < natoms; j++) {
                    const float4 p = spos[j], R = sREQ[j];
                    const Atom2 J = atom2(p, R, p, R);
                    f32x2 dx, dy, dz;
                    bool ok0, ok1, x0, x1;
                    excl(j, x0, x1);
                    const f32x2 F = force2<HB>(J, I, C, x0, x1, dx, dy, dz, ok0, ok1);
                    if (COUNT) npair += (ok0 && v0 ? 1 : 0) + (ok1 && v1 ? 1 : 0);
                    fx = fma2(dx, F, fx); fy = fma2(dy, F, fy); fz = fma2(dz, F, fz);
                }
            };
            if (!bonds) pass([&](int j, bool& x0, bool& x1) { x0 = j == i0; x1 = j == i1; });
            else pass([&](int j, bool& x0, bool& x1) {
                x0 = j == i0 || j == e0 || j == e1 || j == e2 || j == e3;
                x1 = j == i1 || j == h0 || j == h1 || j == h2 || j == h3;
            });
        }
        if (v0) out[i0] = make_float4(lo2(fx), lo2(fy), lo2(fz), 0.f);
        if (v1) out[i1] = make_float4(hi2(fx), hi2(fy), hi2(fz), 0.f);
    }

    // Shifted-image pair lists (Verlet lists with a skin, P.vskin, 1 A by
    // default).  Of the pairs the candidate tiles of the shifted images
    // evaluate, only a few percent lie inside the cutoff: for a large molecule
    // the candidates of an image span its whole cross-section.  With lists,
    // the ordered pairs (i, j + shift of image k) over every shifted image k
    // closer than Rc + skin are collected once and evaluated every step (both
    // orders of a pair are listed, so no reaction is needed) until some atom
    // has moved more than skin/2 since the build (move() checks); then they are
    // rebuilt.  The entries are numbered by image, then atom i, then atom j, and cut
    // into L.runs runs of equal length; within a run the consecutive entries of an atom
    // i have one FP32 sum.  Entry e of run v lies at word e L.runs + v of the CTA's
    // slot of global scratch (a warp's 32 runs read whole lines), and the first entry's
    // number of every row (image, i) behind the entries.
    __device__ __forceinline__ uint32_t* vslot() const { return P.vlist + (size_t)blockIdx.x * P.vstride; }
    __device__ __forceinline__ uint32_t run_start(uint32_t v) const { return (uint32_t)nlist * v / (uint32_t)L.runs; }

    // pass over the listed pairs of row r by one warp: f(pair listed here, entry) per 32 candidates
    template <class F>
    __device__ __forceinline__ void row_pass(int r, const float4* spos, float Rv2, F&& f) {
        const int* ccnt = at<int>(L.ccnt);
        const unsigned short* clist = at<unsigned short>(L.clist);
        int k = 0;
        while (r >= ccnt[L.nimg - 1 - k]) { r -= ccnt[L.nimg - 1 - k]; k++; }
        const int i = clist[(L.nimg - 1 - k) * L.maxNA + r], ipbc = image_index(k);
        const float4 pi = spos[i], s = at<float4>(L.shf)[k];
        const float qx = pi.x - s.x, qy = pi.y - s.y, qz = pi.z - s.z;
        const unsigned short* Jl = clist + k * L.maxNA;
        const int nJ = ccnt[k];
        for (int j0 = 0; j0 < nJ; j0 += 32) {
            const int j = Jl[min(j0 + lane, nJ - 1)];
            const float4 pj = spos[j];
            const float dx = pj.x - qx, dy = pj.y - qy, dz = pj.z - qz;
            f(j0 + lane < nJ && fmaf(dx, dx, fmaf(dy, dy, dz * dz)) < Rv2 && !image_excluded(i, j, ipbc),
              (uint32_t)i | ((uint32_t)j << 12) | ((uint32_t)k << 24));
        }
    }

    // rebuild this system's lists from the current positions; false
    // (block-uniform) when they do not fit in the slot.  All threads; barriers.
    __device__ bool list_build(const float4* spos, float Rv2) {
        store_vp(spos);
        build_candidates(Rv2);
        const int* ccnt = at<int>(L.ccnt);
        uint32_t* ent = vslot();
        uint32_t* rows = ent + P.vcap + L.runs;
        int R = 0;
        for (int k = 0; k < L.nimg; k++) R += ccnt[k];
        for (int r = warp; r < R; r += NW) {                 // entries of every row
            int c = 0;
            row_pass(r, spos, Rv2, [&](bool in, uint32_t) { c += __popc(__ballot_sync(0xffffffffu, in)); });
            if (lane == 0) rows[r] = c;
        }
        __syncthreads();
        int* tmp = at<int>(L.red);                           // exclusive sums
        const int r0 = (int)((long long)R * tid / T), r1 = (int)((long long)R * (tid + 1) / T);
        int c = 0;
        for (int r = r0; r < r1; r++) c += rows[r];
        int incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) tmp[warp] = incl;
        __syncthreads();
        int base = 0, total = 0;
        for (int w = 0; w < NW; w++) {
            if (w < warp) base += tmp[w];
            total += tmp[w];
        }
        if (total > P.vcap) return false;
        base += incl - c;
        for (int r = r0; r < r1; r++) { const int n = rows[r]; rows[r] = base; base += n; }
        nlist = total;
        __syncthreads();
        for (int r = warp; r < R; r += NW) {                 // write (CL: the runs of this CTA)
            const uint32_t q0 = rows[r], q1 = r + 1 < R ? rows[r + 1] : (uint32_t)total;
            if (q0 == q1) continue;
            uint32_t at0 = q0;
            row_pass(r, spos, Rv2, [&](bool in, uint32_t w) {
                const uint32_t bal = __ballot_sync(0xffffffffu, in);
                if (in) {
                    const uint32_t q = at0 + __popc(bal & ((1u << lane) - 1u));
                    const uint32_t v = ((q + 1) * (uint32_t)L.runs - 1) / (uint32_t)total;      // the last run that starts at or before q
                    if (!CL || (int)(v >> 5) % cn == cr) ent[(q - run_start(v)) * L.runs + v] = w;
                }
                at0 += __popc(bal);
            });
        }
        __syncthreads();
        return true;
    }
    __device__ __forceinline__ void store_vp(const float4* spos) {
        float* vp = at<float>(L.vp);
        for (int a = tid; a < natoms; a += T) {
            const float4 p = spos[a];
            vp[a] = p.x; vp[L.maxNA + a] = p.y; vp[2 * L.maxNA + a] = p.z;
        }
    }

    // runs 32 g .. 32 g + 31 of the listed pairs, one per lane
    template <bool HB>
    __device__ void list_unit(int g, long long* facc) {
        const float4* spos = at<float4>(L.pos);
        const float4* sREQ = at<float4>(L.REQ);
        const float4* shf = at<float4>(L.shf);
        const int v = 32 * g + lane;
        const int n = (int)(run_start(v + 1) - run_start(v));
        if (n <= 0) return;
        const uint32_t* ent = vslot() + v;
        int ci = -1;
        float3 fi = make_float3(0.f, 0.f, 0.f);
        float4 pi = make_float4(0.f, 0.f, 0.f, 0.f), Ri = pi;
        uint32_t wn = ent[0], wn2 = n > 1 ? ent[L.runs] : 0;
        for (int e = 0; e < n; e++) {
            const uint32_t w = wn;
            wn = wn2;
            if (e + 2 < n) wn2 = ent[(e + 2) * L.runs];
            const int i = (int)(w & 0xFFFu), j = (int)((w >> 12) & 0xFFFu);
            if (i != ci) {
                if (ci >= 0) fix_add(facc + 3 * ci, fi);
                ci = i; fi = make_float3(0.f, 0.f, 0.f);
                pi = spos[i]; Ri = sREQ[i];
            }
            const float4 s = shf[w >> 24], pj = spos[j];
            const float dx = pj.x + s.x - pi.x, dy = pj.y + s.y - pi.y, dz = pj.z + s.z - pi.z;
            bool ok;
            float en;
            const float F = pair_force<false, HB>(dx, dy, dz, Ri, sREQ[j], false, P.Rc2, P.kq_rc2, 0.f, true, ok, en);
            if (!ok) continue;
            if (COUNT) npair++;
            fi.x = fmaf(dx, F, fi.x); fi.y = fmaf(dy, F, fi.y); fi.z = fmaf(dz, F, fi.z);
        }
        fix_add(facc + 3 * ci, fi);
    }

    // ---- small systems (up to 64 atoms): one warp has every pair sum ----------
    // Lane l owns atoms l and l + 32; every atom's sum is one FP32 accumulator over the
    // images in order.  Up to 32 atoms: atoms j in order in every image.  Above: in the
    // central image each pair once, lane l meeting the atoms of lane l + s at rotation
    // step s, the reactions coming back by shuffle.  Two sums per packed instruction.
    __device__ __forceinline__ void small_excl(int a, int ipbc, bool pbc, uint32_t& lo, uint32_t& hi) {
        lo = hi = 0;
        if (a >= natoms) { lo = hi = ~0u; return; }
        const int4 g = ngs(a), c = ngc(a);
        auto set = [&](int j) { if (j >= 0) { if (j < 32) lo |= 1u << j; else hi |= 1u << (j - 32); } };
        set(a);
        if (!pbc || c.x == ipbc) set(g.x);
        if (!pbc || c.y == ipbc) set(g.y);
        if (!pbc || c.z == ipbc) set(g.z);
        if (!pbc || c.w == ipbc) set(g.w);
    }
    __device__ __forceinline__ void small_rows(int a, uint32_t& lo, uint32_t& hi) const {
        if (a >= natoms) { lo = hi = ~0u; return; }
        lo = __ldg(xrow + a * nbw);
        hi = nbw > 1 ? __ldg(xrow + a * nbw + 1) : ~0u;
    }
    // central image of 33 .. 64 atoms; m: excluded atoms of the own two
    template <bool HB>
    __device__ __forceinline__ void small_central(const Atom2& I, const PairC& C, uint32_t m0lo, uint32_t m0hi, uint32_t m1lo,
                                                  uint32_t m1hi, f32x2& fx, f32x2& fy, f32x2& fz) {
        const float4* spos = at<float4>(L.pos);
        const float4* sREQ = at<float4>(L.REQ);
        const int last = natoms - 1;
        const uint32_t inv_hi = natoms >= 64 ? 0u : ~((1u << (natoms - 32)) - 1u);      // slots beyond the system
        m0hi |= inv_hi; m1hi |= inv_hi;
        bool ok0, ok1;
        f32x2 dx, dy, dz;
        {   // s = 0: (A, B) of this lane
            const int b = min(lane + 32, last);
            const float4 p = spos[b], R = sREQ[b];
            const f32x2 F2 = force2<HB>(atom2(p, R, p, R), I, C, (m0hi >> lane) & 1u, true, dx, dy, dz, ok0, ok1);
            const float F = lo2(F2);
            if (COUNT && ok0) npair += 2;
            fx = pack2(fmaf(lo2(dx), F, lo2(fx)), fmaf(-lo2(dx), F, hi2(fx)));
            fy = pack2(fmaf(lo2(dy), F, lo2(fy)), fmaf(-lo2(dy), F, hi2(fy)));
            fz = pack2(fmaf(lo2(dz), F, lo2(fz)), fmaf(-lo2(dz), F, hi2(fz)));
        }
        m0lo = __funnelshift_r(m0lo, m0lo, lane); m0hi = __funnelshift_r(m0hi, m0hi, lane);
        m1lo = __funnelshift_r(m1lo, m1lo, lane); m1hi = __funnelshift_r(m1hi, m1hi, lane);
#pragma unroll 1
        for (int s = 1; s <= 16; s++) {
            const int p = (lane + s) & 31, src = (lane - s) & 31;
            const bool half = s == 16 && lane >= 16;
            m0lo >>= 1; m0hi >>= 1; m1lo >>= 1; m1hi >>= 1;
            const int jb = min(p + 32, last);
            const float4 pA = spos[p], RA = sREQ[p], pB = spos[jb], RB = sREQ[jb];
            float3 r;
            {   // (A, A') and (B, A'); s = 16: the second is (A', B) of lane p, done there
                const f32x2 F = force2<HB>(atom2(pA, RA, pA, RA), I, C, (m0lo & 1u) || half, (m1lo & 1u) || s == 16, dx, dy, dz, ok0, ok1);
                if (COUNT) npair += (ok0 ? 2 : 0) + (ok1 ? 2 : 0);
                fx = fma2(dx, F, fx); fy = fma2(dy, F, fy); fz = fma2(dz, F, fz);
                r.x = fmaf(-hi2(dx), hi2(F), -lo2(dx) * lo2(F));
                r.y = fmaf(-hi2(dy), hi2(F), -lo2(dy) * lo2(F));
                r.z = fmaf(-hi2(dz), hi2(F), -lo2(dz) * lo2(F));
            }
            fx = pack2(lo2(fx) + __shfl_sync(0xffffffffu, r.x, src), hi2(fx));
            fy = pack2(lo2(fy) + __shfl_sync(0xffffffffu, r.y, src), hi2(fy));
            fz = pack2(lo2(fz) + __shfl_sync(0xffffffffu, r.z, src), hi2(fz));
            {   // (A, B') and (B, B')
                const f32x2 F = force2<HB>(atom2(pB, RB, pB, RB), I, C, m0hi & 1u, (m1hi & 1u) || half, dx, dy, dz, ok0, ok1);
                if (COUNT) npair += (ok0 ? 2 : 0) + (ok1 ? 2 : 0);
                fx = fma2(dx, F, fx); fy = fma2(dy, F, fy); fz = fma2(dz, F, fz);
                r.x = fmaf(-lo2(dx), lo2(F), -hi2(dx) * hi2(F));
                r.y = fmaf(-lo2(dy), lo2(F), -hi2(dy) * hi2(F));
                r.z = fmaf(-lo2(dz), lo2(F), -hi2(dz) * hi2(F));
            }
            fx = pack2(lo2(fx), hi2(fx) + __shfl_sync(0xffffffffu, r.x, src));
            fy = pack2(lo2(fy), hi2(fy) + __shfl_sync(0xffffffffu, r.y, src));
            fz = pack2(lo2(fz), hi2(fz) + __shfl_sync(0xffffffffu, r.z, src));
        }
    }

    template <bool HB>
    __device__ void small_pairs(float4* out) {
        const float4* spos = at<float4>(L.pos);
        const float4* sREQ = at<float4>(L.REQ);
        const PairC C = pair_consts();
        const bool pbc = (P.flags & F_PBC) != 0, cut = P.Rc2 > 0.f, two = natoms > 32;
        const int npx = pbc ? P.npbc[0] : 0, npy = pbc ? P.npbc[1] : 0, npz = pbc ? P.npbc[2] : 0;
        const int a0 = lane, a1 = lane + 32, last = natoms - 1;
        float mn[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, mx[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        if (cut && (npx | npy | npz)) {              // the atoms' box
            for (int i = lane; i < natoms; i += 32) {
                const float4 p = spos[i];
                mn[0] = fminf(mn[0], p.x); mn[1] = fminf(mn[1], p.y); mn[2] = fminf(mn[2], p.z);
                mx[0] = fmaxf(mx[0], p.x); mx[1] = fmaxf(mx[1], p.y); mx[2] = fmaxf(mx[2], p.z);
            }
#pragma unroll
            for (int k = 0; k < 3; k++) { mn[k] = wmin(mn[k]); mx[k] = wmax(mx[k]); }
        }
        const float4 q0 = spos[min(a0, last)], q1 = spos[min(a1, last)];
        Atom2 I = own2(q0, sREQ[min(a0, last)], q1, sREQ[min(a1, last)]);
        f32x2 fx = 0, fy = 0, fz = 0;
        int im = 0;
#pragma unroll 1
        for (int iz = -npz; iz <= npz; iz++)
#pragma unroll 1
            for (int iy = -npy; iy <= npy; iy++)
#pragma unroll 1
                for (int ix = -npx; ix <= npx; ix++, im++) {
                    const float3 s = image_shift(lv, ix, iy, iz);
                    const bool central = (ix | iy | iz) == 0;
                    if (cut && !central) {
                        const float gx = fmaxf(0.f, fabsf(s.x) - (mx[0] - mn[0]));
                        const float gy = fmaxf(0.f, fabsf(s.y) - (mx[1] - mn[1]));
                        const float gz = fmaxf(0.f, fabsf(s.z) - (mx[2] - mn[2]));
                        if (gx * gx + gy * gy + gz * gz >= P.Rc2) continue;   // image out of reach (uniform)
                    }
                    uint32_t m0lo, m0hi, m1lo, m1hi;
                    if (central) { small_rows(a0, m0lo, m0hi); small_rows(a1, m1lo, m1hi); }
                    else { small_excl(a0, im, pbc, m0lo, m0hi); small_excl(a1, im, pbc, m1lo, m1hi); }
                    if (two) {
                        if (central) {
                            I.x = neg2(pack2(q0.x, q1.x)); I.y = neg2(pack2(q0.y, q1.y)); I.z = neg2(pack2(q0.z, q1.z));
                            small_central<HB>(I, C, m0lo, m0hi, m1lo, m1hi, fx, fy, fz);
                            continue;
                        }
                        I.x = pack2(s.x - q0.x, s.x - q1.x); I.y = pack2(s.y - q0.y, s.y - q1.y); I.z = pack2(s.z - q0.z, s.z - q1.z);
#pragma unroll 1
                        for (int j = 0; j < natoms; j++) {
                            const float4 p = spos[j], R = sREQ[j];
                            f32x2 dx, dy, dz;
                            bool ok0, ok1;
                            const f32x2 F = force2<HB>(atom2(p, R, p, R), I, C, m0lo & 1u, m1lo & 1u, dx, dy, dz, ok0, ok1);
                            if (COUNT) npair += (ok0 ? 1 : 0) + (ok1 ? 1 : 0);
                            m0lo = (m0lo >> 1) | (m0hi << 31); m0hi >>= 1;
                            m1lo = (m1lo >> 1) | (m1hi << 31); m1hi >>= 1;
                            fx = fma2(dx, F, fx); fy = fma2(dy, F, fy); fz = fma2(dz, F, fz);
                        }
                    } else {
                        // one atom per lane: two atoms j side by side, one sum
                        Atom2 K = I;
                        K.x = pack2(s.x - q0.x, s.x - q0.x); K.y = pack2(s.y - q0.y, s.y - q0.y); K.z = pack2(s.z - q0.z, s.z - q0.z);
                        K.R = pack2(lo2(I.R), lo2(I.R)); K.E = pack2(lo2(I.E), lo2(I.E)); K.Q = pack2(lo2(I.Q), lo2(I.Q)); K.H = pack2(lo2(I.H), lo2(I.H));
                        float3 f = make_float3(lo2(fx), lo2(fy), lo2(fz));
#pragma unroll 1
                        for (int j = 0; j < natoms; j += 2) {
                            const int j1 = min(j + 1, last);
                            f32x2 dx, dy, dz;
                            bool ok0, ok1;
                            const f32x2 F = force2<HB>(atom2(spos[j], sREQ[j], spos[j1], sREQ[j1]), K, C, (m0lo >> j) & 1u, (m0lo >> j1) & 1u,
                                                       dx, dy, dz, ok0, ok1);
                            if (COUNT) npair += (ok0 ? 1 : 0) + (ok1 && j1 > j ? 1 : 0);
                            f.x = fmaf(lo2(dx), lo2(F), f.x); f.y = fmaf(lo2(dy), lo2(F), f.y); f.z = fmaf(lo2(dz), lo2(F), f.z);
                            if (j1 > j) { f.x = fmaf(hi2(dx), hi2(F), f.x); f.y = fmaf(hi2(dy), hi2(F), f.y); f.z = fmaf(hi2(dz), hi2(F), f.z); }
                        }
                        fx = pack2(f.x, 0.f); fy = pack2(f.y, 0.f); fz = pack2(f.z, 0.f);
                    }
                }
        if (a0 < natoms) out[a0] = make_float4(lo2(fx), lo2(fy), lo2(fz), 0.f);
        if (a1 < natoms) out[a1] = make_float4(hi2(fx), hi2(fy), hi2(fz), 0.f);
    }

    // ------------------------------------------------------------------ forces
    // bonded terms of nodes 32 u .. 32 u + 31, one per lane
    __device__ void bonded_unit(int u) {
        const int ia = 32 * u + lane;
        if (ia >= nnode) return;
        float4* fasm = at<float4>(L.fasm);
        float4* fng = at<float4>(L.fng);
        BondedOut o;
        eval_atom<false>(ia, natoms, nnode, P.flags, P.Fmax2NB, at<float4>(L.pos), at<float4>(L.REQ), ngs(ia), ngc(ia),
                         B::npar(L.apar, Y.apars, ia), B::npar(L.bL, Y.bLs, ia), B::npar(L.bK, Y.bKs, ia),
                         B::npar(L.ksp, Y.Ksp, ia), B::npar(L.kpp, Y.Kpp, ia), lv, P.npbc[0], P.npbc[1], P.npbc[2],
                         __ldg(Y.a13 + noff + ia), Cut13(P), o);
        fasm[ia] = make_float4(o.fa.x, o.fa.y, o.fa.z, 0.f);
        fasm[natoms + ia] = make_float4(o.fpi.x, o.fpi.y, o.fpi.z, 0.f);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            fng[ia * 4 + k] = make_float4(o.fbs[k].x, o.fbs[k].y, o.fbs[k].z, 0.f);
            fng[4 * L.maxNN + ia * 4 + k] = make_float4(o.fps[k].x, o.fps[k].y, o.fps[k].z, 0.f);
        }
    }

    // GridFF samples of atoms 8 g .. 8 g + 7, four lanes each (x-slices); the four
    // slices are added in pairs, in small systems one after another
    __device__ void grid_unit(int g, float4* fgr) {
        const float4* spos = at<float4>(L.pos);
        const int i = 8 * g + (lane >> 2), a = lane & 3;
        const bool ok = i < natoms;
        const int ic = ok ? i : natoms - 1;
        const float4 p = spos[ic];
        const float3 uu = make_float3((p.x + lv[9]) * P.ginv[0], (p.y + lv[10]) * P.ginv[1], (p.z + lv[11]) * P.ginv[2]);
        float3 e;                            // d/dy, d/dz and value of the slice
        float4 bx, dx;
        if (Y.gkey != nullptr)
            e = grid_slice_cached(P.grid, P.gn[0], P.gn[1], P.gn[2], uu, B::plq(ic), a, ok, at<unsigned>(L.key) + ic,
                                  Y.gkey + aoff + ic, Y.gcs + (size_t)(aoff + ic) * 16, bx, dx);
        else
            e = grid_slice<(T >= MMFF_UNROLL_MIN_T) ? 4 : 1>(P.grid, P.gn[0], P.gn[1], P.gn[2], uu, B::plq(ic), a, bx, dx);
        float4 r;
        if (L.small) {
            r = make_float4(0.f, 0.f, 0.f, 0.f);
            const int l0 = lane & 28;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float ex = __shfl_sync(0xffffffffu, e.x, l0 | k), ey = __shfl_sync(0xffffffffu, e.y, l0 | k);
                const float ez = __shfl_sync(0xffffffffu, e.z, l0 | k);
                r.x = fmaf(comp(dx, k), ez, r.x); r.y = fmaf(comp(bx, k), ex, r.y); r.z = fmaf(comp(bx, k), ey, r.z);
            }
        } else {
            r = make_float4(comp(dx, a) * e.z, comp(bx, a) * e.x, comp(bx, a) * e.y, 0.f);
#pragma unroll
            for (int o = 2; o > 0; o >>= 1) {
                r.x += __shfl_xor_sync(0xffffffffu, r.x, o);
                r.y += __shfl_xor_sync(0xffffffffu, r.y, o);
                r.z += __shfl_xor_sync(0xffffffffu, r.z, o);
            }
        }
        if (ok && a == 0) fgr[i] = make_float4(r.x * P.gmi[0], r.y * P.gmi[1], r.z * P.gmi[2], 0.f);
    }

    // all units of this step, claimed by the warps in turn, the long ones first:
    // image rows, bonded terms, pair sums of a small system, tiles, list runs, grid
    template <bool HB>
    __device__ void units(long long* facc) {
        const bool nb = (P.flags & F_NONBONDED) != 0;
        auto mine = [&](int n) { return CL ? (n - cr + cn - 1) / cn : n; };       // units cr, cr + cn, ... of n
        const int nI = mine(nb && image_row_path() ? (natoms + 63) >> 6 : 0);
        const int nS = nb && L.small ? 1 : 0;
        const int nB = (nnode + 31) >> 5;
        const int nT = mine(nb && !L.small ? double_tiles() + single_units() + diag_units() : 0);
        const int nL = mine(use_list ? L.runs >> 5 : 0);
        const int nG = mine((P.flags & F_GRID) ? (natoms + 7) >> 3 : 0);
        const int e0 = nI, e1 = e0 + nS, e2 = e1 + nB, e3 = e2 + nT, e4 = e3 + nL, e5 = e4 + nG;
        int* claim = shared_ints() + 2 + par;
        auto global_unit = [&](int m) { return CL ? cr + cn * m : m; };
        while (true) {
            int u = 0;
            if (lane == 0) u = atomicAdd(claim, 1);
            u = __shfl_sync(0xffffffffu, u, 0);
            if (u >= e5) break;
            if (u < e0) image_row_unit<HB>(global_unit(u), listf());
            else if (u < e1) small_pairs<HB>(listf());
            else if (u < e2) bonded_unit(u - e1);
            else if (u < e3) tile_unit<HB>(global_unit(u - e2), facc);
            else if (u < e4) list_unit<HB>(global_unit(u - e3), facc);
            else grid_unit(global_unit(u - e4), gridf());
            __syncwarp();
        }
    }

    // moved: some atom moved more than half the list skin since the positions vp
    // (block-uniform, from the previous step's move)
    __device__ void forces(bool moved) {
        const int flags = P.flags;
        const float4* spos = at<float4>(L.pos);
        long long* facc = sums();
        use_list = false;
        if ((flags & F_NONBONDED) && P.Rc2 > 0.f && L.nimg > 0) {
            use_list = listok && lstate == LIST_BUILT && !moved;
            if (!use_list && !(listok && lstate == LIST_QUIET && !moved)) {
                bbox_from_smem();
                if (any_image(P.Rc2)) {
                    const float Rv = sqrtf(P.Rc2) + P.vskin, Rv2 = Rv * Rv;
                    if (listok) {
                        if (COUNT && tid == 0) atomicAdd(Y.counters + 3, 1ull);
                        use_list = listok = list_build(spos, Rv2);
                        lstate = LIST_BUILT;
                    }
                    if (!listok) {
                        __syncthreads();
                        build_candidates(P.Rc2);
                        if (hasH) candidate_units<true>(spos, facc);
                        else candidate_units<false>(spos, facc);
                        __syncthreads();                 // the lists share the recoil slots' memory
                    }
                } else if (listok && lstate != LIST_BUILT) {
                    // nothing in reach: no need to look again until an atom has moved
                    const float Rv = sqrtf(P.Rc2) + P.vskin;
                    lstate = any_image(Rv * Rv) ? LIST_NONE : LIST_QUIET;
                    if (lstate == LIST_QUIET) store_vp(spos);
                }
            }
            if (COUNT && tid == 0 && use_list) atomicAdd(Y.counters + 4, (unsigned long long)nlist);
        }
        if (hasH) units<true>(facc);
        else units<false>(facc);
        // direct substrate term (getSurfMorse), one thread per atom (never in a cluster)
        if (flags & F_SURF) {
            __syncthreads();
            float4* fgr = gridf();
            const float4* sR = at<float4>(L.REQ);
            for (int a = tid; a < natoms; a += T) {
                const float4 p = spos[a];
                const float4 r = surf_atom(P, make_float3(p.x + lv[9], p.y + lv[10], p.z + lv[11]), sR[a]);
                const float4 g = (flags & F_GRID) ? fgr[a] : make_float4(0.f, 0.f, 0.f, 0.f);
                fgr[a] = make_float4(g.x + r.x, g.y + r.y, g.z + r.z, 0.f);
            }
        }
        if (CL && pairbad) shared_ints()[par] = 1;
    }
    template <bool HB>
    __device__ void candidate_units(const float4* spos, long long* facc) {
        const float4* sREQ = at<float4>(L.REQ);
        float ec = 0.f;
        const int n = B::image_tile_count();
        for (int u = cr * NW + warp; u < n; u += cn * NW) B::template image_tile_unit<HB>(u, spos, sREQ, facc, ec);
        B::template image_rows<HB>(cr * T + tid, cn * T, spos, sREQ, true, facc, ec);
    }

    // ---------------------------------------------------------------- assemble
    // assemble + clamp; FP64 partial sums of (vf, vv, ff) and max|f|^2 for this
    // thread; the pair sums are read and cleared for the next step
    __device__ void assemble(double& vf, double& vv, double& ff, float& fmax2, bool& bad) {
        float4* fasm = at<float4>(L.fasm);
        long long* facc = sums();
        float4* fgr = gridf();
        float4* flist = listf();
        const bool with_list = has_listf(), with_grid = (P.flags & (F_GRID | F_SURF)) != 0;
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
                long long s[3] = {0, 0, 0};
                float3 b = make_float3(0.f, 0.f, 0.f), g = b;
                if constexpr (CL) {
                    for (int c = 0; c < cn; c++) {
                        const long long* q = cooperative_groups::this_cluster().map_shared_rank(facc, c) + 3 * v;
                        s[0] += q[0]; s[1] += q[1]; s[2] += q[2];
                    }
                    long long* z = at<long long>(L.facc) + (par ^ 1) * 3 * L.maxNA + 3 * v;
                    z[0] = 0; z[1] = 0; z[2] = 0;
                    // (the owners of the atom's image row and grid sample)
                    if (with_list) b = f3(cooperative_groups::this_cluster().map_shared_rank(flist, (v >> 6) % cn)[v]);
                    if (with_grid) g = f3(cooperative_groups::this_cluster().map_shared_rank(fgr, (v >> 3) % cn)[v]);
                } else {
                    s[0] = facc[3 * v]; s[1] = facc[3 * v + 1]; s[2] = facc[3 * v + 2];
                    facc[3 * v] = 0; facc[3 * v + 1] = 0; facc[3 * v + 2] = 0;
                    if (with_list) b = f3(flist[v]);
                    if (with_grid) g = f3(fgr[v]);
                }
                f.x = f.x + ((float)s[0] * (1.f / kFix) + b.x) + g.x;
                f.y = f.y + ((float)s[1] * (1.f / kFix) + b.y) + g.y;
                f.z = f.z + ((float)s[2] * (1.f / kFix) + b.z) + g.z;
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
        if (CL) bad |= any_cl(par);
        else bad |= pairbad;
        if (tid == 0) { shared_ints()[par ^ 1] = 0; shared_ints()[2 + (par ^ 1)] = 0; }
        par ^= 1;
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
    // whether a moved atom left the neighbourhood (half the skin) of its position vp
    __device__ __forceinline__ bool moved_atom(int v, float3 p) {
        if (lstate == LIST_NONE) return false;
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
