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
// without a host round trip.  G > 1: a CTA of G such systems, T threads each, that
// begin every step together, so that the SM's warps run the same code at a time.
//
// A relaxation amplifies the last bit of a force: two or three molecules of a few
// hundred part after some hundred steps, and the largest differences reach the
// size of a bond.  So every FP32 sum here has a fixed order that depends on the
// system alone, not on the block size, the cluster or which warp takes a unit:
// partial sums over a tile or a run of list entries go to 64-bit integer totals,
// everything else is summed by one lane.  The packed instructions below take two
// independent sums side by side, never two terms of one sum.
//
// Bound: latency and issue with 16 warps per SM (128 registers, shared memory): about
// half of the issue slots are used, the FP32 pipe a third.  Time per system-step with the
// chip full (us), the kernels whose sums these are / here: 28 atoms 0.0087 / 0.0076, 60:
// 0.0323 / 0.0193, 100: 0.0610 / 0.0410, 200: 0.148 / 0.106, 330: 0.368 / 0.260; without
// a cutoff 127 atoms 0.286 / 0.191, 330 atoms 1.76 / 1.20.  Per step of few systems: 16 x
// 24 atoms without a cutoff 18.2 / 11.0, 37 x 350 atoms 53.7 / 27.6.
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
template <int T, bool COUNT, bool CL = false, int G = 1>
struct RelaxEngine : PairEngine<T, 1, false, COUNT, true, G> {
    using B = PairEngine<T, 1, false, COUNT, true, G>;
    using B::sync; using B::sync_or; using B::group;
    using B::P; using B::Y; using B::L; using B::tid; using B::lane; using B::warp;
    using B::isys; using B::natoms; using B::nnode; using B::nvecs; using B::aoff; using B::noff; using B::voff;
    using B::lv; using B::hasH; using B::hasX; using B::xrow; using B::nbw; using B::pairbad; using B::kFix; using B::kFixMax;
    using B::ngs; using B::ngc; using B::bks; using B::image_within; using B::build_candidates; using B::fix_add;
    using B::image_excluded; using B::bbox_from_smem; using B::npair; using B::tile_mask; using B::bbmin; using B::bbmax;
    template <class X> __device__ __forceinline__ X* at(int off) { return B::template at<X>(off); }
    static constexpr int NW = T / 32;
    static constexpr int kGridChunk = T == 32 ? 8 : 2;         // grid units (8 atoms) per claim
    static constexpr int kRowUnroll = T >= MMFF_UNROLL_MIN_T ? 2 : 1;
    static constexpr int kTileUnroll = CL ? 4 : T >= MMFF_UNROLL_MIN_T ? 2 : 1;
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
        else sync();
    }
    // this step's force sums
    __device__ __forceinline__ long long* sums() { return at<long long>(L.facc) + (CL ? par * 3 * L.maxNA : 0); }
    __device__ __forceinline__ float4* gridf() { return at<float4>(L.fgrid) + (CL ? par * L.maxNA : 0); }
    __device__ __forceinline__ float4* listf() {
        if (!CL && B::kMayCompact && L.flist < 0) return Y.force + voff;
        return at<float4>(L.flist) + (CL ? par * L.maxNA : 0);
    }
    // [0, 1] a non-finite pair force (CL, per set of sums), [2, 3] units claimed (per step parity)
    __device__ __forceinline__ int* shared_ints() const {
        __shared__ int f[4 * G];
        return f + 4 * group();
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
    __device__ __forceinline__ bool image_row_path() const {
        return (P.flags & F_PBC) && !(P.Rc2 > 0.f) && !L.small && (P.npbc[0] | P.npbc[1] | P.npbc[2]);
    }
    __device__ __forceinline__ bool has_listf() const { return (P.flags & F_NONBONDED) && (L.small || image_row_path()); }

    __device__ void load(int s) {
        B::load(s);
        listok = P.vlist != nullptr && natoms <= 4096 && P.Rc2 > 0.f && L.nimg > 0 && L.nimg <= kListMaxImages &&
                 (P.flags & F_NONBONDED);
        lstate = LIST_NONE;
        nlist = 0;
        use_list = false;
        par = 0;
        sync();
        if (L.shf >= 0 && tid < L.nimg) {
            const float3 sh = image_of(image_index(tid));
            at<float4>(L.shf)[tid] = make_float4(sh.x, sh.y, sh.z, 0.f);
        }
        put_all();
        long long* facc = at<long long>(L.facc);
        for (int a = tid; a < 3 * natoms; a += T) facc[a] = 0;
        if constexpr (CL)
            for (int a = tid; a < 3 * natoms; a += T) facc[3 * L.maxNA + a] = 0;
        if (tid < 4) shared_ints()[tid] = tid < 2 ? 0 : NW;
    }
    __device__ __forceinline__ PairC pair_consts() const {
        PairC C;
        C.Rc2 = P.Rc2 > 0.f ? P.Rc2 : 3.0e38f;
        C.nkq = pack2(-P.kq_rc2, -P.kq_rc2); C.m12 = pack2(-12.f, -12.f); C.m1 = pack2(-1.f, -1.f);
        return C;
    }

    // ---- pair arrays --------------------------------------------------------
    // Positions and parameters of the atoms as the packed loops load them.  Blocks of 32
    // atoms in pairs (L.pj): word 4 (a mod 32) + (block mod 2) + 2 c of array q holds
    // quantity 2 q + c of (x, y, z, R0, sqrt E0, Q, H), so that one 16-byte load gives two
    // quantities of atom j and of the atom 32 further.  Atom after atom (L.soa): seven
    // arrays.  Slots beyond the system have no charge and no LJ, and are excluded.
    __device__ __forceinline__ float* pj(int a) { return at<float>(L.pj) + (a >> 6) * 512 + 4 * (a & 31) + ((a >> 5) & 1); }
    __device__ __forceinline__ float* soa(int k) { return at<float>(L.soa) + k * 32 * L.nwords; }
    __device__ __forceinline__ void put_pos(int a, float3 p) {
        if (L.pj >= 0) { float* q = pj(a); q[0] = p.x; q[2] = p.y; q[128] = p.z; }
        if (L.soa >= 0 && a < 32 * L.nwords) { soa(0)[a] = p.x; soa(1)[a] = p.y; soa(2)[a] = p.z; }
    }
    __device__ void put_all() {
        const float4* spos = at<float4>(L.pos);
        const float4* sREQ = at<float4>(L.REQ);
        for (int a = tid; a < 64 * ((L.nwords + 1) >> 1); a += T) {
            const bool v = a < natoms;
            const float4 r = v ? sREQ[a] : make_float4(0.f, 0.f, 0.f, 0.f);
            if (L.pj >= 0) { float* q = pj(a); q[130] = r.x; q[256] = r.y; q[258] = r.z; q[384] = r.w; }
            if (L.soa >= 0 && a < 32 * L.nwords) { soa(3)[a] = r.x; soa(4)[a] = r.y; soa(5)[a] = r.z; soa(6)[a] = r.w; }
            put_pos(a, v ? f3(spos[a]) : make_float3(0.f, 0.f, 0.f));
        }
    }
    // slot l of block pair m, both halves
    template <bool HB>
    __device__ __forceinline__ Atom2 load2(int m, int l) {
        const ulonglong2* q = at<ulonglong2>(L.pj) + 128 * m + l;
        const ulonglong2 a = q[0], b = q[32], c = q[64];
        Atom2 r;
        r.x = a.x; r.y = a.y; r.z = b.x; r.R = b.y; r.E = c.x; r.Q = c.y;
        r.H = HB ? q[96].x : 0;
        return r;
    }
    static __device__ __forceinline__ f32x2 dup_lo(f32x2 v) { return pack2(lo2(v), lo2(v)); }
    static __device__ __forceinline__ f32x2 dup_hi(f32x2 v) { return pack2(hi2(v), hi2(v)); }
    template <bool HI>
    static __device__ __forceinline__ Atom2 dup(const Atom2& v) {
        auto d = [](f32x2 x) { return HI ? dup_hi(x) : dup_lo(x); };
        return {d(v.x), d(v.y), d(v.z), d(v.R), d(v.E), d(v.Q), d(v.H)};
    }
    static __device__ __forceinline__ Atom2 as_own(Atom2 a) {
        a.x = neg2(a.x); a.y = neg2(a.y); a.z = neg2(a.z); a.Q = neg2(a.Q);
        return a;
    }
    // 64-bit fixed point of two FP32 sums
    __device__ __forceinline__ void fix_add2(long long* a, f32x2 x, f32x2 y, f32x2 z) {
        pairbad |= !isfinite(lo2(x) + lo2(y) + lo2(z)) | !isfinite(hi2(x) + hi2(y) + hi2(z));
        auto fix = [](float v) { return __float2ll_rn(fminf(fmaxf(v, -kFixMax), kFixMax) * kFix); };
        B::add64(a + 0, fix(lo2(x)) + fix(hi2(x)));
        B::add64(a + 1, fix(lo2(y)) + fix(hi2(y)));
        B::add64(a + 2, fix(lo2(z)) + fix(hi2(z)));
    }

    // ---- central image, two 32 x 32 tiles at a time ---------------------------
    // Tiles of PairEngine (off_tile, diag_tile), sums in the same order: lane l owns
    // atom i of block bi, the atoms j of another block rotate past it, the reactions
    // (as sums of d F; negated at the end) with them.  KIND 0: block bi against both
    // blocks of pair m; 1: blocks bi and bi2 against the lone last block; 2: two
    // tiles (lower, upper block) of the pairs m and m2; 3: the diagonal tiles of pair m.
    // m2, bi2 < 0: no second tile.
    // Bound: the FP32 pipe (29 packed operations, 58 clocks a rotation step of 64
    // unordered pairs), then issue.
    template <bool HB, int KIND>
    __device__ void tile2(int bi, int bi2, int m, int m2, long long* facc) {
        const PairC C = pair_consts();
        Atom2 I;
        uint32_t x0, x1;                             // excluded j by slot
        auto row = [&](int i, int bj) { return i < natoms ? __ldg(xrow + i * nbw + bj) : ~0u; };
        if (KIND == 0) {
            const Atom2 o = load2<HB>(bi >> 1, lane);
            I = (bi & 1) ? dup<true>(o) : dup<false>(o);
            x0 = row(32 * bi + lane, 2 * m); x1 = row(32 * bi + lane, 2 * m + 1);
        } else if (KIND == 1) {
            I = load2<HB>(bi >> 1, lane);            // bi even, bi2 = bi + 1
            x0 = row(32 * bi + lane, 2 * m); x1 = bi2 >= 0 ? row(32 * bi2 + lane, 2 * m) : ~0u;
        } else if (KIND == 2) {
            const Atom2 o = load2<HB>(m, lane), p = load2<HB>(max(m2, 0), lane);
            auto c = [](f32x2 a, f32x2 b) { return pack2(lo2(a), lo2(b)); };
            I = {c(o.x, p.x), c(o.y, p.y), c(o.z, p.z), c(o.R, p.R), c(o.E, p.E), c(o.Q, p.Q), c(o.H, p.H)};
            x0 = row(64 * m + lane, 2 * m + 1); x1 = m2 >= 0 ? row(64 * m2 + lane, 2 * m2 + 1) : ~0u;
        } else {
            I = load2<HB>(m, lane);
            x0 = row(64 * m + lane, 2 * m); x1 = 2 * m + 1 < nbw ? row(64 * m + 32 + lane, 2 * m + 1) : ~0u;
        }
        I = as_own(I);
        constexpr int s0 = KIND == 3 ? 1 : 0, s1 = KIND == 3 ? 17 : 32;
        x0 = __funnelshift_r(x0, x0, lane + s0);     // by rotation step, from s0
        x1 = __funnelshift_r(x1, x1, lane + s0);
        f32x2 fx = 0, fy = 0, fz = 0, rx = 0, ry = 0, rz = 0;
        const int nxt = (lane + 1) & 31;
        // d and F of a rotation step; the next step's are on their way while this one's are added
        auto eval = [&](int s, f32x2& dx, f32x2& dy, f32x2& dz) {
            const int jl = (lane + s) & 31;
            Atom2 J;
            if (KIND == 0 || KIND == 3) {
                J = load2<HB>(m, jl);
            } else if (KIND == 1) {
                J = dup<false>(load2<HB>(m, jl));
            } else {
                const Atom2 o = load2<HB>(m, jl), p = load2<HB>(max(m2, 0), jl);
                auto c = [](f32x2 a, f32x2 b) { return pack2(hi2(a), hi2(b)); };
                J = {c(o.x, p.x), c(o.y, p.y), c(o.z, p.z), c(o.R, p.R), c(o.E, p.E), c(o.Q, p.Q), c(o.H, p.H)};
            }
            const bool half = KIND == 3 && (s > 16 || (s == 16 && lane >= 16)), past = KIND != 3 && s >= 32;
            bool ok0, ok1;
            const f32x2 F = force2<HB>(J, I, C, (x0 & 1u) || half, (x1 & 1u) || half, dx, dy, dz, ok0, ok1);
            x0 >>= 1; x1 >>= 1;
            if (COUNT && !past) npair += (ok0 ? 2 : 0) + (ok1 ? 2 : 0);
            return F;
        };
        f32x2 dx, dy, dz, F = eval(s0, dx, dy, dz);
#pragma unroll kTileUnroll
        for (int s = s0; s < s1; s++) {
            f32x2 ex, ey, ez;
            const f32x2 Fn = eval(s + 1, ex, ey, ez);
            fx = fma2(dx, F, fx); fy = fma2(dy, F, fy); fz = fma2(dz, F, fz);
            if (KIND == 3) {
                const int src = (lane - s) & 31;     // the lane whose partner this lane's atoms were
                const f32x2 nF = neg2(F);
                fx = add2(fx, __shfl_sync(0xffffffffu, mul2(dx, nF), src));
                fy = add2(fy, __shfl_sync(0xffffffffu, mul2(dy, nF), src));
                fz = add2(fz, __shfl_sync(0xffffffffu, mul2(dz, nF), src));
            } else {
                rx = __shfl_sync(0xffffffffu, fma2(dx, F, rx), nxt);
                ry = __shfl_sync(0xffffffffu, fma2(dy, F, ry), nxt);
                rz = __shfl_sync(0xffffffffu, fma2(dz, F, rz), nxt);
            }
            F = Fn; dx = ex; dy = ey; dz = ez;
        }
        rx = neg2(rx); ry = neg2(ry); rz = neg2(rz);
        auto add1 = [&](int a, f32x2 x, f32x2 y, f32x2 z, bool hi) {
            if (a < natoms) fix_add(facc + 3 * a, hi ? make_float3(hi2(x), hi2(y), hi2(z)) : make_float3(lo2(x), lo2(y), lo2(z)));
        };
        if (KIND == 0) {
            fix_add2(facc + 3 * (32 * bi + lane), fx, fy, fz);
            add1(64 * m + lane, rx, ry, rz, false);
            add1(64 * m + 32 + lane, rx, ry, rz, true);
        } else if (KIND == 1) {
            add1(32 * bi + lane, fx, fy, fz, false);
            if (bi2 >= 0) add1(32 * bi2 + lane, fx, fy, fz, true);
            if (64 * m + lane < natoms) fix_add2(facc + 3 * (64 * m + lane), rx, ry, rz);
        } else if (KIND == 2) {
            add1(64 * m + lane, fx, fy, fz, false);
            add1(64 * m + 32 + lane, rx, ry, rz, false);
            if (m2 >= 0) {
                add1(64 * m2 + lane, fx, fy, fz, true);
                add1(64 * m2 + 32 + lane, rx, ry, rz, true);
            }
        } else {
            add1(64 * m + lane, fx, fy, fz, false);
            add1(64 * m + 32 + lane, fx, fy, fz, true);
        }
    }
    // units of tiles.  nbw blocks are nbw / 2 pairs and, if odd, a lone last block:
    // every block below a pair against it; below the lone block, two blocks at a
    // time; the tile within a pair, two pairs at a time; diagonals by pairs.
    __device__ __forceinline__ int tile_units() const {
        const int H = nbw >> 1;
        return H * (H - 1) + ((nbw & 1) ? H : 0) + ((H + 1) >> 1) + ((nbw + 1) >> 1);
    }
    template <bool HB>
    __device__ void tile_unit(int u, long long* facc) {
        const int H = nbw >> 1, n0 = H * (H - 1), n1 = (nbw & 1) ? H : 0, n2 = (H + 1) >> 1;
        if (u < n0) {
            int m = 1;
            while (u >= 2 * m) { u -= 2 * m; m++; }
            tile2<HB, 0>(u, -1, m, -1, facc);
        } else if (u < n0 + n1) {
            const int b = 2 * (u - n0);
            tile2<HB, 1>(b, b + 1, H, -1, facc);
        } else if (u < n0 + n1 + n2) {
            const int m = 2 * (u - n0 - n1);
            tile2<HB, 2>(2 * m, -1, m, m + 1 < H ? m + 1 : -1, facc);
        } else {
            tile2<HB, 3>(0, -1, u - n0 - n1 - n2, -1, facc);
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

    // Two pairs (i; j, j + 1), added one after the other to atom i's sum.  K: atom i in both
    // halves, dx.. from it; two: j + 1 is an atom of the system
    // (ARRAYS: from the arrays atom after atom, which the largest systems do not have)
    template <bool HB, bool ARRAYS = true>
    __device__ __forceinline__ void row_step(int j, const Atom2& K, const PairC& C, bool x0, bool x1, bool two, float3& f) {
        Atom2 J;
        if (!ARRAYS) {
            const int j1 = two ? j + 1 : j;
            J = atom2(at<float4>(L.pos)[j], at<float4>(L.REQ)[j], at<float4>(L.pos)[j1], at<float4>(L.REQ)[j1]);
        } else {
            auto ld = [&](int k) { return *reinterpret_cast<const f32x2*>(soa(k) + j); };
            J.x = ld(0); J.y = ld(1); J.z = ld(2); J.R = ld(3); J.E = ld(4); J.Q = ld(5); J.H = HB ? ld(6) : 0;
        }
        f32x2 dx, dy, dz;
        bool ok0, ok1;
        const f32x2 F = force2<HB>(J, K, C, x0, x1, dx, dy, dz, ok0, ok1);
        if (COUNT) npair += (ok0 ? 1 : 0) + (ok1 && two ? 1 : 0);
        f.x = fmaf(lo2(dx), lo2(F), f.x); f.y = fmaf(lo2(dy), lo2(F), f.y); f.z = fmaf(lo2(dz), lo2(F), f.z);
        if (two) { f.x = fmaf(hi2(dx), hi2(F), f.x); f.y = fmaf(hi2(dy), hi2(F), f.y); f.z = fmaf(hi2(dz), hi2(F), f.z); }
    }
    static __device__ __forceinline__ Atom2 own_dup(float4 p, float4 R) { return own2(p, R, p, R); }
    static __device__ __forceinline__ void shift_own(Atom2& K, float4 p, float3 s) {
        K.x = pack2(s.x - p.x, s.x - p.x); K.y = pack2(s.y - p.y, s.y - p.y); K.z = pack2(s.z - p.z, s.z - p.z);
    }

    // Without a cutoff: atoms 32 u .. 32 u + 31, one per lane, against all atoms of
    // every shifted image, images and atoms j in order; each atom's sum in one accumulator.
    template <bool HB>
    __device__ void image_row_unit(int u, float4* out) {
        const PairC C = pair_consts();
        const int i = 32 * u + lane, a = min(i, natoms - 1);
        const float4 p = at<float4>(L.pos)[a];
        Atom2 K = own_dup(p, at<float4>(L.REQ)[a]);
        const int4 g = ngs(a), c = ngc(a);
        const int nim = (2 * P.npbc[0] + 1) * (2 * P.npbc[1] + 1) * (2 * P.npbc[2] + 1), central = nim / 2;
        float3 f = make_float3(0.f, 0.f, 0.f);
        for (int im = 0; im < nim; im++) {
            if (im == central) continue;
            shift_own(K, p, image_of(im));
            const int e0 = c.x == im ? g.x : -1, e1 = c.y == im ? g.y : -1, e2 = c.z == im ? g.z : -1, e3 = c.w == im ? g.w : -1;
            const bool arrays = !B::kMayCompact || L.soa >= 0;
            if (arrays && !__any_sync(0xffffffffu, max(max(e0, e1), max(e2, e3)) >= 0)) {
#pragma unroll kRowUnroll
                for (int j = 0; j < natoms; j += 2) row_step<HB>(j, K, C, j == a, j + 1 == a, j + 1 < natoms, f);
            } else {
#pragma unroll 1
                for (int j = 0; j < natoms; j += 2) {
                    auto ex = [&](int q) { return q == a || q == e0 || q == e1 || q == e2 || q == e3; };
                    if (arrays) row_step<HB>(j, K, C, ex(j), ex(j + 1), j + 1 < natoms, f);
                    else row_step<HB, false>(j, K, C, ex(j), ex(j + 1), j + 1 < natoms, f);
                }
            }
        }
        if (i < natoms) out[i] = make_float4(f.x, f.y, f.z, 0.f);
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
    __device__ __forceinline__ uint32_t* vslot() const { return P.vlist + ((size_t)blockIdx.x * G + group()) * P.vstride; }
    __device__ __forceinline__ uint32_t run_start(uint32_t v) const { return (uint32_t)nlist * v / (uint32_t)L.runs; }

    // Rows (image k, candidate i of its mirror), k-major, in groups of 32 of one image, a
    // row per lane: f(row, i, k) starts a row and returns what to do with its listed pairs'
    // atoms j (in order) and at its end.
    template <class F>
    __device__ __forceinline__ void for_rows(const float4* spos, float Rv2, F&& f) {
        const int* ccnt = at<int>(L.ccnt);
        const unsigned short* clist = at<unsigned short>(L.clist);
        int k = 0, base = 0, g = warp;
        while (true) {
            int n = 0;
            for (; k < L.nimg; k++) {
                n = ccnt[L.nimg - 1 - k];
                if (32 * g < n) break;
                g -= (n + 31) >> 5;
                base += n;
            }
            if (k >= L.nimg) break;
            const int c = 32 * g + lane, ipbc = image_index(k), nJ = ccnt[k];
            const bool v = c < n;
            const int i = clist[(L.nimg - 1 - k) * L.maxNA + min(c, n - 1)];
            const float4 pi = spos[i], sh = at<float4>(L.shf)[k];
            const float qx = pi.x - sh.x, qy = pi.y - sh.y, qz = pi.z - sh.z;
            const unsigned short* Jl = clist + k * L.maxNA;
            auto pairs = f(base + c, i, k, v);
            for (int j0 = 0; j0 < nJ; j0 += 4) {             // four distances at a time
                int j[4];
                float d2[4];
#pragma unroll
                for (int q = 0; q < 4; q++) j[q] = Jl[min(j0 + q, nJ - 1)];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float4 pj = spos[j[q]];
                    const float dx = pj.x - qx, dy = pj.y - qy, dz = pj.z - qz;
                    d2[q] = j0 + q < nJ && v ? fmaf(dx, dx, fmaf(dy, dy, dz * dz)) : FLT_MAX;
                }
                if (fminf(fminf(d2[0], d2[1]), fminf(d2[2], d2[3])) < Rv2) {
#pragma unroll
                    for (int q = 0; q < 4; q++) if (d2[q] < Rv2 && !image_excluded(i, j[q], ipbc)) pairs.add(j[q]);
                }
            }
            pairs.end();
            g += NW;
        }
    }
    struct RowCount {
        uint32_t* out; int n; bool v;
        __device__ __forceinline__ void add(int) { n++; }
        __device__ __forceinline__ void end() { if (v) *out = n; }
    };
    struct RowWrite {
        RelaxEngine& E;
        uint32_t* ent;
        uint32_t w, q, v, qs, qe;                // entry without its j; number; its run, that run's first entry and the next one's
        __device__ __forceinline__ void add(int j) {
            while (q >= qe) { v++; qs = qe; qe = E.run_start(v + 1); }
            if (!CL || (int)(v >> 5) % E.cn == E.cr) ent[(q - qs) * E.L.runs + v] = w | ((uint32_t)j << 12);
            q++;
        }
        __device__ __forceinline__ void end() {}
    };

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
        for_rows(spos, Rv2, [&](int r, int, int, bool v) { return RowCount{rows + r, 0, v}; });       // entries of every row
        sync();
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
        sync();
        int base = 0, total = 0;
        for (int w = 0; w < NW; w++) {
            if (w < warp) base += tmp[w];
            total += tmp[w];
        }
        if (total > P.vcap) return false;
        base += incl - c;
        for (int r = r0; r < r1; r++) { const int n = rows[r]; rows[r] = base; base += n; }
        nlist = total;
        sync();
        for_rows(spos, Rv2, [&](int r, int i, int k, bool v) {                                        // (CL: the runs of this CTA)
            RowWrite w{*this, ent, (uint32_t)i | ((uint32_t)k << 24), v ? rows[r] : 0u, 0, 0, 0};
            w.v = total ? ((w.q + 1) * (uint32_t)L.runs - 1) / (uint32_t)total : 0;                   // the last run that starts at or before q
            w.qs = run_start(w.v); w.qe = run_start(w.v + 1);
            return w;
        });
        sync();
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
        // entry e + 3 comes from memory, the atoms and shift of entry e + 1 from shared
        // memory while entry e is evaluated
        uint32_t w = ent[0], w1 = n > 1 ? ent[L.runs] : w, w2 = n > 2 ? ent[2 * L.runs] : w;
        auto jof = [](uint32_t x) { return (int)((x >> 12) & 0xFFFu); };
        float4 pj = spos[jof(w)], Rj = sREQ[jof(w)], sh = shf[w >> 24];
        int ci = (int)(w & 0xFFFu);
        float3 fi = make_float3(0.f, 0.f, 0.f);
        float4 pi = spos[ci], Ri = sREQ[ci];
        for (int e = 0; e < n; e++) {
            const float4 pn = spos[jof(w1)], Rn = sREQ[jof(w1)], sn = shf[w1 >> 24];
            uint32_t w3 = w2;
            if (e + 3 < n) w3 = ent[(e + 3) * L.runs];
            const int i = (int)(w & 0xFFFu);
            if (i != ci) {
                fix_add(facc + 3 * ci, fi);
                ci = i; fi = make_float3(0.f, 0.f, 0.f);
                pi = spos[i]; Ri = sREQ[i];
            }
            const float dx = pj.x + sh.x - pi.x, dy = pj.y + sh.y - pi.y, dz = pj.z + sh.z - pi.z;
            bool ok;
            float en;
            const float F = pair_force<false, HB>(dx, dy, dz, Ri, Rj, false, P.Rc2, P.kq_rc2, 0.f, true, ok, en);
            if (ok) {
                if (COUNT) npair++;
                fi.x = fmaf(dx, F, fi.x); fi.y = fmaf(dy, F, fi.y); fi.z = fmaf(dz, F, fi.z);
            }
            w = w1; w1 = w2; w2 = w3;
            pj = pn; Rj = Rn; sh = sn;
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
    // central image of 33 .. 64 atoms; m: excluded atoms of the own two (A, B)
    template <bool HB>
    __device__ __forceinline__ void small_central(const PairC& C, uint32_t m0lo, uint32_t m0hi, uint32_t m1lo, uint32_t m1hi,
                                                  float3& f0, float3& f1) {
        const uint32_t inv_hi = natoms >= 64 ? 0u : ~((1u << (natoms - 32)) - 1u);      // slots beyond the system
        m0hi |= inv_hi; m1hi |= inv_hi;
        const Atom2 own = as_own(load2<HB>(0, lane)), A = dup<false>(own), Bo = dup<true>(own);
        bool ok0, ok1;
        f32x2 dx, dy, dz;
        {   // s = 0: (A, B) of this lane
            const float F = hi2(force2<HB>(load2<HB>(0, lane), A, C, true, (m0hi >> lane) & 1u, dx, dy, dz, ok0, ok1));
            if (COUNT && ok1) npair += 2;
            f0.x = fmaf(hi2(dx), F, f0.x); f0.y = fmaf(hi2(dy), F, f0.y); f0.z = fmaf(hi2(dz), F, f0.z);
            f1.x = fmaf(-hi2(dx), F, f1.x); f1.y = fmaf(-hi2(dy), F, f1.y); f1.z = fmaf(-hi2(dz), F, f1.z);
        }
        m0lo = __funnelshift_r(m0lo, m0lo, lane); m0hi = __funnelshift_r(m0hi, m0hi, lane);
        m1lo = __funnelshift_r(m1lo, m1lo, lane); m1hi = __funnelshift_r(m1hi, m1hi, lane);
#pragma unroll 1
        for (int s = 1; s <= 16; s++) {
            const int src = (lane - s) & 31;
            const bool half = s == 16 && lane >= 16;
            m0lo >>= 1; m0hi >>= 1; m1lo >>= 1; m1hi >>= 1;
            const Atom2 J = load2<HB>(0, (lane + s) & 31);                 // A', B' of lane l + s
            f32x2 ex, ey, ez;
            const f32x2 Fa = force2<HB>(J, A, C, (m0lo & 1u) || half, m0hi & 1u, dx, dy, dz, ok0, ok1);
            if (COUNT) npair += (ok0 ? 2 : 0) + (ok1 ? 2 : 0);
            // s = 16: (B, A') is (A', B) of lane l + s, done there
            const f32x2 Fb = force2<HB>(J, Bo, C, (m1lo & 1u) || s == 16, (m1hi & 1u) || half, ex, ey, ez, ok0, ok1);
            if (COUNT) npair += (ok0 ? 2 : 0) + (ok1 ? 2 : 0);
            auto axis = [&](f32x2 d, f32x2 e, float& a, float& b) {
                const float d0 = lo2(d), d1 = hi2(d), e0 = lo2(e), e1 = hi2(e), A0 = lo2(Fa), A1 = hi2(Fa), B0 = lo2(Fb), B1 = hi2(Fb);
                a = fmaf(d0, A0, a);                                       // (A, A'), the reaction of (A', A) and (A', B), (A, B')
                b = fmaf(e0, B0, b);                                       // (B, A'), (B, B'), the reaction of (B', B) and (B', A)
                a -= __shfl_sync(0xffffffffu, fmaf(e0, B0, d0 * A0), src);
                a = fmaf(d1, A1, a);
                b = fmaf(e1, B1, b);
                b -= __shfl_sync(0xffffffffu, fmaf(d1, A1, e1 * B1), src);
            };
            axis(dx, ex, f0.x, f1.x);
            axis(dy, ey, f0.y, f1.y);
            axis(dz, ez, f0.z, f1.z);
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
        Atom2 K = own_dup(q0, sREQ[min(a0, last)]);
        float3 f0 = make_float3(0.f, 0.f, 0.f), f1 = f0;
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
                    if (!two) {
                        shift_own(K, q0, s);
#pragma unroll 1
                        for (int j = 0; j < natoms; j += 2) {
                            row_step<HB>(j, K, C, m0lo & 1u, m0lo & 2u, j + 1 < natoms, f0);
                            m0lo >>= 2;
                        }
                    } else if (central) {
                        small_central<HB>(C, m0lo, m0hi, m1lo, m1hi, f0, f1);
                    } else {
                        Atom2 I = own2(q0, sREQ[a0], q1, sREQ[min(a1, last)]);
                        I.x = pack2(s.x - q0.x, s.x - q1.x); I.y = pack2(s.y - q0.y, s.y - q1.y); I.z = pack2(s.z - q0.z, s.z - q1.z);
                        f32x2 fx = pack2(f0.x, f1.x), fy = pack2(f0.y, f1.y), fz = pack2(f0.z, f1.z);
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
                        f0 = make_float3(lo2(fx), lo2(fy), lo2(fz)); f1 = make_float3(hi2(fx), hi2(fy), hi2(fz));
                    }
                }
        if (a0 < natoms) out[a0] = make_float4(f0.x, f0.y, f0.z, 0.f);
        if (a1 < natoms) out[a1] = make_float4(f1.x, f1.y, f1.z, 0.f);
    }

    // Few systems of up to 32 atoms: the scalar forces F of all pairs by every warp, into
    // L.fbuf [image][j][i]; after a barrier the same sums as small_pairs, an axis per warp
    // (one FP32 accumulator per atom and axis, images and atoms j in order).  A system's
    // step waits for its longest warp: 16 x 24 atoms without a cutoff, where one warp with
    // every pair took 24 of 28 thousand clocks.
    __device__ __forceinline__ bool split_sums() const { return L.fbuf >= 0; }
    // images of the pair sum, and whether image im is in reach of the cutoff (small_pairs)
    __device__ __forceinline__ int split_images() const {
        return (P.flags & F_PBC) ? (2 * P.npbc[0] + 1) * (2 * P.npbc[1] + 1) * (2 * P.npbc[2] + 1) : 1;
    }
    __device__ __forceinline__ float3 split_shift(int im) const { return (P.flags & F_PBC) ? image_of(im) : make_float3(0.f, 0.f, 0.f); }
    // F of atoms j = 8 q .. 8 q + 7 of one image for atom i = lane; unit u = (image, q)
    template <bool HB>
    __device__ void split_forces(int u) {
        const int nq = (natoms + 7) >> 3, im = u / nq, q = u - im * nq, a = min(lane, natoms - 1);
        const bool pbc = (P.flags & F_PBC) != 0;
        const PairC C = pair_consts();
        const float4 p = at<float4>(L.pos)[a];
        Atom2 K = own_dup(p, at<float4>(L.REQ)[a]);
        shift_own(K, p, split_shift(im));
        uint32_t m, hi;
        if (im == split_images() / 2) small_rows(lane, m, hi);
        else small_excl(lane, im, pbc, m, hi);
        m >>= 8 * q;
        float* out = at<float>(L.fbuf) + (im * L.maxNA + 8 * q) * 32 + lane;
#pragma unroll 2
        for (int j = 8 * q; j < min(natoms, 8 * q + 8); j += 2) {
            Atom2 J;
            auto ld = [&](int k) { return *reinterpret_cast<const f32x2*>(soa(k) + j); };
            J.x = ld(0); J.y = ld(1); J.z = ld(2); J.R = ld(3); J.E = ld(4); J.Q = ld(5); J.H = HB ? ld(6) : 0;
            f32x2 dx, dy, dz;
            bool ok0, ok1;
            const f32x2 F = force2<HB>(J, K, C, m & 1u, m & 2u, dx, dy, dz, ok0, ok1);
            if (COUNT) npair += (ok0 ? 1 : 0) + (ok1 && j + 1 < natoms ? 1 : 0);
            m >>= 2;
            out[0] = lo2(F);
            if (j + 1 < natoms) out[32] = hi2(F);
            out += 64;
        }
    }
    // axis c of every atom's sum
    __device__ void split_sum(int c, float4* out) {
        const float* X = soa(c);
        const int a = min(lane, natoms - 1), nim = split_images();
        const float pc = X[a];
        const bool cut = P.Rc2 > 0.f;
        float mn[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, mx[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        if (cut && nim > 1) {
#pragma unroll
            for (int k = 0; k < 3; k++) { const float v = soa(k)[a]; mn[k] = wmin(v); mx[k] = wmax(v); }
        }
        float f = 0.f;
        for (int im = 0; im < nim; im++) {
            const float3 s = split_shift(im);
            if (cut && im != nim / 2) {
                const float gx = fmaxf(0.f, fabsf(s.x) - (mx[0] - mn[0]));
                const float gy = fmaxf(0.f, fabsf(s.y) - (mx[1] - mn[1]));
                const float gz = fmaxf(0.f, fabsf(s.z) - (mx[2] - mn[2]));
                if (gx * gx + gy * gy + gz * gz >= P.Rc2) continue;
            }
            const float sc = c == 0 ? s.x : c == 1 ? s.y : s.z, o = sc - pc;
            const float* F = at<float>(L.fbuf) + im * L.maxNA * 32 + lane;
            int j = 0;
            for (; j + 8 <= natoms; j += 8) {            // loads ahead of the chain
                float x[8], g[8];
#pragma unroll
                for (int q = 0; q < 8; q++) { x[q] = X[j + q]; g[q] = F[32 * (j + q)]; }
#pragma unroll
                for (int q = 0; q < 8; q++) f = fmaf(x[q] + o, g[q], f);
            }
            for (; j < natoms; j++) f = fmaf(X[j] + o, F[32 * j], f);
        }
        if (lane < natoms) reinterpret_cast<float*>(out + lane)[c] = f;
    }

    // ------------------------------------------------------------------ forces
    // recoil slot of neighbour k of node n (host numbering 4 n + k): lanes on consecutive words
    __device__ __forceinline__ int slot(int i) const { return (i & 3) * L.maxNN + (i >> 2); }
    // word 4 ia + k of a per-node (or per-atom) array of four
    template <class X>
    __device__ __forceinline__ X node_word(int off, const void* g, int i) {
        return B::compact() ? __ldg(reinterpret_cast<const X*>(g) + i) : at<X>(off)[i];
    }

    // eval_atom in straight-line code, whose independent terms overlap: for few systems,
    // where a step waits for its longest warp (24 atoms: 9.7 -> 6.9 thousand clocks)
    __device__ void bonded_straight(int ia) {
        float4* fasm = at<float4>(L.fasm);
        float4* sig = at<float4>(L.fng) + ia;
        BondedOut o;
        eval_atom<false>(ia, natoms, nnode, P.flags, P.Fmax2NB, at<float4>(L.pos), at<float4>(L.REQ), ngs(ia), ngc(ia),
                         B::npar(L.apar, Y.apars, ia), B::npar(L.bL, Y.bLs, ia), B::npar(L.bK, Y.bKs, ia),
                         B::npar(L.ksp, Y.Ksp, ia), B::npar(L.kpp, Y.Kpp, ia), lv, P.npbc[0], P.npbc[1], P.npbc[2],
                         __ldg(Y.a13 + noff + ia), Cut13(P), o);
        fasm[ia] = make_float4(o.fa.x, o.fa.y, o.fa.z, 0.f);
        fasm[natoms + ia] = make_float4(o.fpi.x, o.fpi.y, o.fpi.z, 0.f);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            sig[k * L.maxNN] = make_float4(o.fbs[k].x, o.fbs[k].y, o.fbs[k].z, 0.f);
            sig[(4 + k) * L.maxNN] = make_float4(o.fps[k].x, o.fps[k].y, o.fps[k].z, 0.f);
        }
    }

    // Bonded terms of nodes 32 u .. 32 u + 31, one per lane: MMFFsp3_loc::eval_atom
    // (MMFFsp3_loc.h:250-575), the terms of eval_atom in mmff_device.cuh, operation for
    // operation, as loops over neighbours and angles instead of some 1000 straight-line
    // instructions (of which the small blocks, eight per SM in different phases, mostly
    // waited for the instruction cache).  The bond vectors wait in the node's own recoil
    // slots: (h, 1/l) in the pi slot until the pi forces go there, l beside the sigma force.
    __device__ void bonded_unit(int u) {
        const int ia = 32 * u + lane;
        if (ia >= nnode) return;
        if (CL || (T >= 128 && split_sums())) { bonded_straight(ia); return; }
        const float4* spos = at<float4>(L.pos);
        const float4* sREQ = at<float4>(L.REQ);
        float4* fasm = at<float4>(L.fasm);
        float4* sig = at<float4>(L.fng) + ia;                  // slot k: [k * maxNN]
        float4* pis = sig + 4 * L.maxNN;
        const int flags = P.flags, step = L.maxNN;
        const float4 apar = B::npar(L.apar, Y.apars, ia);
        const float3 pa = f3(spos[ia]), hpi = f3(spos[natoms + ia]);
        const int central = ((2 * P.npbc[1] + 1) * P.npbc[2] + P.npbc[1]) * (2 * P.npbc[0] + 1) + P.npbc[0];
        float3 fa = make_float3(0.f, 0.f, 0.f), fpi = fa;
        int nb = 0;
#pragma unroll 1
        for (; nb < 4; nb++) {
            const int n4 = 4 * ia + nb, ing = node_word<int>(L.ng, Y.neighs + aoff, n4);
            if (ing < 0) break;
            float3 h = f3(spos[ing]) - pa, fb = make_float3(0.f, 0.f, 0.f);
            if (flags & F_PBC) {
                // most bonds stay in the central cell: no shift, and none of the divisions that name the cell
                const int c = node_word<int>(L.ngC, Y.neighCell + aoff, n4);
                if (c != central) {
                    const float3 cell = image_cell(c, P.npbc[0], P.npbc[1], P.npbc[2]);
                    h.x += lv[0] * cell.x + lv[3] * cell.y + lv[6] * cell.z;
                    h.y += lv[1] * cell.x + lv[4] * cell.y + lv[7] * cell.z;
                    h.z += lv[2] * cell.x + lv[5] * cell.y + lv[8] * cell.z;
                }
            }
            const float l2 = dot3(h, h);
            const float il = rsqrtf(l2);
            const float l = l2 * il;
            h = h * il;
            if ((flags & F_BONDS) && ia < ing) {
                const float dl = l - node_word<float>(L.bL, Y.bLs + noff, n4);
                const float fr = dl * node_word<float>(L.bK, Y.bKs + noff, n4);
                float3 f1 = h * fr;
                if (flags & F_SUB_BOND_NB) {
                    const float4 Ri = sREQ[ia], Rj = sREQ[ing];
                    float e;
                    const float3 dp = h * l;
                    const float F = ljqh<false>(l * l, Ri.x + Rj.x, Ri.y * Rj.y, Ri.z * Rj.z, fminf(Ri.w * Rj.w, 0.f), e);
                    float3 fij = dp * F;
                    if (flags & F_CLAMP_NB) { const float f2 = dot3(fij, fij); if (f2 > P.Fmax2NB) fij = fij * sqrtf(P.Fmax2NB / f2); }
                    f1 = f1 - fij;
                }
                fb = fb - f1; fa = fa + f1;
            }
            const float ks = node_word<float>(L.ksp, Y.Ksp + noff, n4);
            if ((flags & F_PISIGMA) && (ks > 1e-6f)) {         // evalAngleCos
                const float c = dot3(hpi, h);
                const float3 b = fma3(h, -c, hpi);
                const float fang = -ks * (c - apar.w) * 2.f;
                const float3 f2 = b * (fang * il);
                fa = fa - f2;
                fb = fb + f2;
            }
            sig[nb * step] = make_float4(fb.x, fb.y, fb.z, l);
            pis[nb * step] = make_float4(h.x, h.y, h.z, il);
        }
        if (flags & F_ANGLES) {
            const int a13 = __ldg(Y.a13 + noff + ia);
            const Cut13 cu(P);
#pragma unroll 1
            for (int i = 0; i + 1 < nb; i++) {
                const float4 H1 = pis[i * step], S1 = sig[i * step];
                float3 fi = f3(S1);
                const int ing = node_word<int>(L.ng, Y.neighs + aoff, 4 * ia + i), ic = node_word<int>(L.ngC, Y.neighCell + aoff, 4 * ia + i);
#pragma unroll 1
                for (int j = i + 1; j < nb; j++) {             // evalAngleCosHalf
                    const float4 H2 = pis[j * step], S2 = sig[j * step];
                    const float3 h1 = f3(H1), h2 = f3(H2), h = h1 + h2;
                    float c2 = dot3(h, h) * 0.25f;
                    const float s2 = 1.f - c2 + 1e-14f;
                    const float c = sqrtf(c2);
                    const float sn = sqrtf(fmaxf(s2, 0.f));
                    const float csy = fmaf(apar.y, c, -apar.x * sn);
                    float fr = -apar.z * csy;
                    c2 *= -2.f;
                    fr = __fdividef(fr, 4.f * c * sn);
                    const float fr1 = fr * H1.w, fr2 = fr * H2.w;
                    float3 f1 = make_float3(h.x * fr1 + h1.x * (fr1 * c2), h.y * fr1 + h1.y * (fr1 * c2), h.z * fr1 + h1.z * (fr1 * c2));
                    float3 f2 = make_float3(h.x * fr2 + h2.x * (fr2 * c2), h.y * fr2 + h2.y * (fr2 * c2), h.z * fr2 + h2.z * (fr2 * c2));
                    fa = fa - (f1 + f2);
                    if (flags & F_SUB_ANGLE_NB) {
                        const int jng = node_word<int>(L.ng, Y.neighs + aoff, 4 * ia + j), jc = node_word<int>(L.ngC, Y.neighCell + aoff, 4 * ia + j);
                        const float3 dp = h2 * S2.w - h1 * S1.w;
                        // x13: the pair sum skipped this central-image pair
                        const bool x13 = (flags & F_EXCL13) && ((a13 >> angle_slot(i, j)) & 1) && (!(flags & F_PBC) || ic == jc);
                        float e, ep;
                        const float F = pair13<false>(dot3(dp, dp), sREQ[ing], sREQ[jng], x13, cu.Rc2, cu.kq, cu.rc, e, ep);
                        float3 fij = dp * F;
                        if (flags & F_CLAMP_NB) { const float ff = dot3(fij, fij); if (ff > P.Fmax2NB) fij = fij * sqrtf(P.Fmax2NB / ff); }
                        f1 = f1 + fij;
                        f2 = f2 - fij;
                    }
                    fi = fi + f1;
                    sig[j * step] = make_float4(S2.x + f2.x, S2.y + f2.y, S2.z + f2.z, S2.w);
                }
                sig[i * step] = make_float4(fi.x, fi.y, fi.z, S1.w);
            }
        }
#pragma unroll 1
        for (int k = 0; k < nb; k++) {                         // forces on the pi vectors
            const int n4 = 4 * ia + k, ing = node_word<int>(L.ng, Y.neighs + aoff, n4);
            const float3 h = f3(pis[k * step]);
            float3 fp = make_float3(0.f, 0.f, 0.f);
            const float kk = node_word<float>(L.kpp, Y.Kpp + noff, n4), ks = node_word<float>(L.ksp, Y.Ksp + noff, n4);
            if ((flags & F_PIPI) && ia < ing && ing < nnode && kk > 1e-6f) {        // evalPiAling
                const float3 h2 = f3(spos[natoms + ing]);
                const float c = dot3(hpi, h2);
                const float3 a = fma3(hpi, -c, h2), b = fma3(h2, -c, hpi);
                const float fang = c < 0.f ? -kk : kk;
                fpi = fpi + a * fang;
                fp = b * fang;
            }
            if ((flags & F_PISIGMA) && (ks > 1e-6f)) {
                const float c = dot3(hpi, h);
                const float3 a = fma3(hpi, -c, h);
                const float fang = -ks * (c - apar.w) * 2.f;
                fpi = fpi + a * fang;
            }
            pis[k * step] = make_float4(fp.x, fp.y, fp.z, 0.f);
        }
#pragma unroll 1
        for (int k = nb; k < 4; k++) sig[k * step] = pis[k * step] = make_float4(0.f, 0.f, 0.f, 0.f);
        fasm[ia] = make_float4(fa.x, fa.y, fa.z, 0.f);
        fasm[natoms + ia] = make_float4(fpi.x, fpi.y, fpi.z, 0.f);
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

    // A warp's first unit.  The first units are the longest, and warp w of a block issues
    // from scheduler w mod 4: the systems of a block start with different ones.
    __device__ __forceinline__ int first_unit() const {
        if (G == 1 || NW == 1) return warp;
        const int g = group(), s = NW == 2 ? (g ^ (g >> 1)) & 1 : g;
        return (warp + NW - s % NW) % NW;
    }

    // all units of this step, claimed by the warps in turn, the long ones first:
    // image rows, bonded terms, pair sums of a small system, tiles, list runs, grid
    template <bool HB>
    __device__ void units(long long* facc) {
        const bool nb = (P.flags & F_NONBONDED) != 0;
        auto mine = [&](int n) { return CL ? (n - cr + cn - 1) / cn : n; };       // units cr, cr + cn, ... of n
        const int nI = mine(nb && image_row_path() ? (natoms + 31) >> 5 : 0);
        const int nS = nb && L.small ? (split_sums() ? split_images() * ((natoms + 7) >> 3) : 1) : 0;
        const int nB = (nnode + 31) >> 5;
        const int nT = mine(nb && !L.small ? tile_units() : 0);
        const int nL = mine(use_list ? L.runs >> 5 : 0);
        const int nG = mine((P.flags & F_GRID) ? (natoms + 7) >> 3 : 0);
        const int nGc = (nG + kGridChunk - 1) / kGridChunk;
        int* claim = shared_ints() + 2 + par;            // starts at NW: every warp has its first unit
        auto next = [&]() {
            int u = 0;
            if (lane == 0) u = atomicAdd(claim, 1);
            __syncwarp();
            return __shfl_sync(0xffffffffu, u, 0);
        };
        auto global_unit = [&](int m) { return CL ? cr + cn * m : m; };
        // one loop per kind: claims only grow, and a kind's code stays in the instruction cache
        int u = first_unit(), e = nI, base = 0;
        for (; u < e; u = next()) image_row_unit<HB>(global_unit(u), listf());
        if (split_sums()) {                              // (the bonded terms are the longest then)
            for (base = e, e += nB; u < e; u = next()) bonded_unit(u - base);
            for (base = e, e += nS; u < e; u = next()) split_forces<HB>(u - base);
        } else {
            for (base = e, e += nS; u < e; u = next()) small_pairs<HB>(listf());
            for (base = e, e += nB; u < e; u = next()) bonded_unit(u - base);
        }
        for (base = e, e += nT; u < e; u = next()) tile_unit<HB>(global_unit(u - base), facc);
        for (base = e, e += nL; u < e; u = next()) list_unit<HB>(global_unit(u - base), facc);
        for (base = e, e += nGc; u < e; u = next())
#pragma unroll 1
            for (int g = kGridChunk * (u - base), g1 = min(nG, g + kGridChunk); g < g1; g++) grid_unit(global_unit(g), gridf());
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
                        sync();
                        build_candidates(P.Rc2);
                        if (hasH) candidate_units<true>(spos, facc);
                        else candidate_units<false>(spos, facc);
                        sync();                 // the lists share the recoil slots' memory
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
        if (split_sums() && (flags & F_NONBONDED)) {
            sync();
            for (int c = warp; c < 3; c += NW) split_sum(c, listf());
        }
        // direct substrate term (getSurfMorse), one thread per atom (never in a cluster)
        if (flags & F_SURF) {
            sync();
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
#pragma unroll 4
                    for (int c = 0; c < cn; c++) {
                        const long long* q = cooperative_groups::this_cluster().map_shared_rank(facc, c) + 3 * v;
                        s[0] += q[0]; s[1] += q[1]; s[2] += q[2];
                    }
                    long long* z = at<long long>(L.facc) + (par ^ 1) * 3 * L.maxNA + 3 * v;
                    z[0] = 0; z[1] = 0; z[2] = 0;
                    // (the owners of the atom's image row and grid sample)
                    if (with_list) b = f3(cooperative_groups::this_cluster().map_shared_rank(flist, (v >> 5) % cn)[v]);
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
            for (int k = 0; k < 4; k++) rec[k] = slots[slot(max(bks[k], 0))];
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
        if (tid == 0) { shared_ints()[par ^ 1] = 0; shared_ints()[2 + (par ^ 1)] = NW; }
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
        sync();
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
    // a moved atom: its copy in the pair arrays, and whether it left the neighbourhood
    // (half the skin) of its position vp
    __device__ __forceinline__ bool moved_atom(int v, float3 p) {
        put_pos(v, p);
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
template <int T, bool COUNT, bool EXPL, bool CL = false, int G = 1>
__global__ void __launch_bounds__(T * G, G == 1 ? relax_min_blocks<T>() : 512 / (T * G)) relax_kernel(const __grid_constant__ Params P, const __grid_constant__ Systems Y, const int* __restrict__ queue, int nqueue,
                                                  int* counter, const __grid_constant__ SmemLayout L) {
    extern __shared__ __align__(16) char smem[];
    using Eng = RelaxEngine<T, COUNT, CL, G>;
    __shared__ int claims[G];
    int& s_claim = claims[Eng::group()];
    Eng E(P, Y, smem + Eng::group() * L.total, L);
    if constexpr (CL) E.csync();        // the whole cluster runs before anyone writes to a neighbour
    while (true) {
        if constexpr (CL) {
            if (E.cr == 0 && E.tid == 0) {
                const int c = atomicAdd(counter, 1);
                for (int k = 0; k < E.cn; k++) *cooperative_groups::this_cluster().map_shared_rank(&s_claim, k) = c;
            }
        } else if (E.tid == 0) {
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
        E.sync();
        int status = ST_MAXSTEPS, itr = 0;
        double meas2 = 0.0;         // convergence measure squared
        bool far = false;           // pair lists out of date (block-uniform)
        int ph = 0;                 // exploring cycle: 2 * (steps in the phase) + exploring
        if constexpr (EXPL) { const int4 g = Y.gopt[s]; ph = 2 * g.y + (g.x != 0); }
        for (itr = 0; itr < P.nstep_max; itr++) {
            if constexpr (G > 1) __syncthreads_or(1);        // the block's systems step together
            bool lang = false;      // an exploring step (Langevin instead of FIRE)
            if constexpr (EXPL) {
                const int ev = explore_step(ph, P.n_explore, P.n_relax);
                lang = ev & 1;
                if ((ev & 2) && E.tid == 0) Y.gopt[s].w++;
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
                far = E.sync_or(far);
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
                    if (E.tid == 0) Y.gopt[s].z++;
                    ph = 1;
                }
            } else {
                if (m < P.Fconv2) { status = ST_CONVERGED; itr++; break; }
            }
            far = E.sync_or(far);   // the end-of-step barrier
        }
        // converged at step itr-1 (reference returns the loop index at break)
        const int steps = (status == ST_CONVERGED) ? itr - 1 : itr;
        E.sync();
        if (CL && E.cr != 0) { E.csync(); continue; }      // every CTA has the same state: the first writes it
        // (a system retired as not finite had no move in its last step)
        E.store_state(status, steps, (float)sqrt(meas2), dt, damping, lastNeg, fs.w + (double)itr);
        if (EXPL && E.tid == 0) { Y.gopt[s].x = ph & 1; Y.gopt[s].y = ph >> 1; }
        if (COUNT) {
            // force evaluations done for this system: itr loop iterations
            if (E.tid == 0) {
                atomicAdd(Y.counters + 1, (unsigned long long)itr * (unsigned long long)E.natoms);
                atomicAdd(Y.counters + 2, (unsigned long long)itr);
            }
        }
        E.csync();
    }
    if constexpr (G > 1) while (__syncthreads_or(0)) {}      // until its last one is done
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
// ... several systems per block
int relax_group(int T) { return T == 32 ? 16 : T == 64 ? 8 : T == 128 ? 4 : 1; }
void* relax_group_fn(int T) {
    switch (T) {
        case 32: return (void*)relax_kernel<32, false, false, false, 16>;
        case 64: return (void*)relax_kernel<64, false, false, false, 8>;
        case 128: return (void*)relax_kernel<128, false, false, false, 4>;
        default: return nullptr;
    }
}
void* relax_fn(int T, bool count) { return count ? relax_of<true, false>(T) : relax_of<false, false>(T); }
void* relax_explore_fn(int T) { return relax_of<false, true>(T); }

}  // namespace mmff
