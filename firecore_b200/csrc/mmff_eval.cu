// mmff_eval.cu -- one force (and energy) evaluation of every system, one CTA
// per system (systems of more than 64 atoms, batches of no more systems than
// SMs, or any size with forced launch shapes), and the grid sampler.
//
//   phase 1  bonded terms (thread per node), non-bonded pairs (32 x 32 tiles,
//            each unordered pair once) and the B-spline GridFF sample (4 lanes
//            per atom, one x-slice of the 4x4x4 stencil each)
//   phase 2  recoil assembly (MMFFsp3_loc::assemble_atom)
#include "mmff_pairs.cuh"

namespace mmff {

// ---------------------------------------------------------------------------
// The per-system engine.  T threads, S threads per atom in the pair sum.
template <int T, int S, bool ENERGY>
struct Engine : PairEngine<T, S, ENERGY> {
    using B = PairEngine<T, S, ENERGY>;
    using B::P; using B::Y; using B::L; using B::tid; using B::lane; using B::warp;
    using B::natoms; using B::nnode; using B::nvecs;
    using B::lv; using B::hasH; using B::pairbad; using B::kFix;
    using B::ngs; using B::ngc; using B::bks; using B::image_active; using B::build_candidates;
    template <class X> __device__ __forceinline__ X* at(int off) { return B::template at<X>(off); }
    double e13 = 0.0;           // ENERGY: pair energies of the skipped 1-3 pairs (energy split)

    __device__ Engine(const Params& p, const Systems& y, char* smem, const SmemLayout& l) : B(p, y, smem, l) {}

    // Threads given to the bonded terms when the GridFF runs beside them on
    // the remaining warps; T = no split.  Cost model in units of one grid
    // round (4 lanes x 16 float4 gathers per atom): one bonded pass (one node
    // per thread) costs ~10 rounds.  Split when the longer of the two
    // concurrent parts beats running them one after the other.
    __device__ __forceinline__ int bonded_grid_split() const {
        if (!(P.flags & F_GRID)) return T;
        const int Tb = ((nnode + 31) / 32) * 32;
        if (Tb >= T || Tb == 0) return T;
        const int Tg = T - Tb;
        const int now = 10 * ((nnode + T - 1) / T) + (4 * natoms + T - 1) / T;
        const int par = max(10, (4 * natoms + Tg - 1) / Tg);
        return par < now ? Tb : T;
    }

    // pair forces of every atom as plain FP32 sums, a thread per atom over the images and
    // atoms j in order: for systems with a force beyond the fixed-point sums' range (atoms
    // on top of one another), whose clamped terms would lose its size and direction
    __device__ void plain_pairs(float4* fnb, bool pbc, int central) {
        const float4* spos = at<float4>(L.pos);
        const float4* sREQ = at<float4>(L.REQ);
        const int npx = pbc ? P.npbc[0] : 0, npy = pbc ? P.npbc[1] : 0, npz = pbc ? P.npbc[2] : 0;
        const float Rc2 = P.Rc2 > 0.f ? P.Rc2 : 3.0e38f;
        for (int i = tid; i < natoms; i += T) {
            const float4 pi = spos[i], Ri = sREQ[i];
            float3 f = make_float3(0.f, 0.f, 0.f);
            int ipbc = 0;
            for (int iz = -npz; iz <= npz; iz++) for (int iy = -npy; iy <= npy; iy++) for (int ix = -npx; ix <= npx; ix++, ipbc++) {
                if (ipbc != central && !image_active(ix, iy, iz)) continue;
                const float3 s = image_shift(lv, ix, iy, iz);
                for (int j = 0; j < natoms; j++) {
                    const bool ex = ipbc == central ? (__ldg(B::xrow + i * B::nbw + (j >> 5)) >> (j & 31)) & 1u
                                                    : B::image_excluded(i, j, ipbc);
                    const float4 pj = spos[j];
                    const float dx = pj.x + s.x - pi.x, dy = pj.y + s.y - pi.y, dz = pj.z + s.z - pi.z;
                    bool ok;
                    float e;
                    const float F = hasH ? pair_force<false, true>(dx, dy, dz, Ri, sREQ[j], ex, Rc2, P.kq_rc2, 0.f, true, ok, e)
                                         : pair_force<false, false>(dx, dy, dz, Ri, sREQ[j], ex, Rc2, P.kq_rc2, 0.f, true, ok, e);
                    f.x = fmaf(dx, F, f.x); f.y = fmaf(dy, F, f.y); f.z = fmaf(dz, F, f.z);
                }
            }
            fnb[i] = make_float4(f.x, f.y, f.z, 0.f);
        }
    }
    // Some term may have been clamped (2^20 eV/A): then the outermost of the atoms on top of
    // one another has a total of that size, as nothing pushes it back; or some was not finite.
    static constexpr float kPlainAbove = 65536.f;

    // ------------------------------------------------------------------ phase 1
    // returns this thread's energy contributions (only meaningful if ENERGY)
    __device__ void forces(double& Eb, double& Enb, double& Eg) {
        const int flags = P.flags;
        const float4* spos = at<float4>(L.pos);
        float4* fnb = at<float4>(L.fnb);
        float4* fgr = at<float4>(L.fgrid);
        const float4* sREQ = at<float4>(L.REQ);
        // Bonded terms and the GridFF stencil are independent: when the nodes
        // fill only part of the block, the other warps sample the grid at the
        // same time (block-uniform choice, see bonded_grid_split)
        const int Tb = bonded_grid_split();
        const bool split = Tb < T;
        if (split && tid >= Tb) B::template grid_phase<ENERGY>(tid - Tb, T - Tb, fgr, Eg);
        B::template bonded_phase<ENERGY>(Tb, Eb, e13);
        // --- non-bonded pairs: S lanes per atom i, j strided by S
        if (flags & F_NONBONDED) {
            const bool pbc = (flags & F_PBC) != 0;
            const int npx = pbc ? P.npbc[0] : 0, npy = pbc ? P.npbc[1] : 0, npz = pbc ? P.npbc[2] : 0;
            const int nxi = 2 * npx + 1, nyi = 2 * npy + 1;
            // cutoff + PBC: candidate lists per shifted image, built only when the
            // bounding-box test keeps some shifted image (block-uniform)
            bool any_shift = false;
            for (int iz = -npz; iz <= npz; iz++)
                for (int iy = -npy; iy <= npy; iy++)
                    for (int ix = -npx; ix <= npx; ix++)
                        if ((ix | iy | iz) != 0) any_shift |= image_active(ix, iy, iz);
            const bool lists = L.nimg > 0 && any_shift;
            if (lists) build_candidates(P.Rc2);
            const int central = (npz * nyi + npy) * nxi + npx;
            // central image and (with candidate lists) the shifted images:
            // every unordered pair once or ordered rows, into fixed-point sums
            long long* facc = at<long long>(L.facc);
            for (int a = tid; a < 3 * natoms; a += T) facc[a] = 0;
            __syncthreads();
            {
                float ec = 0.f;
                if (hasH) {
                    if (lists) B::template pair_tiles<true, true>(spos, sREQ, pbc, central, facc, ec);
                    else B::template pair_tiles<true, false>(spos, sREQ, pbc, central, facc, ec);
                } else {
                    if (lists) B::template pair_tiles<false, true>(spos, sREQ, pbc, central, facc, ec);
                    else B::template pair_tiles<false, false>(spos, sREQ, pbc, central, facc, ec);
                }
                if (ENERGY) Enb += (double)ec;
            }
            __syncthreads();
            bool beyond = pairbad;
            for (int a = tid; a < natoms; a += T) {
                const float3 f = make_float3((float)facc[3 * a] * (1.f / kFix), (float)facc[3 * a + 1] * (1.f / kFix),
                                             (float)facc[3 * a + 2] * (1.f / kFix));
                fnb[a] = make_float4(f.x, f.y, f.z, 0.f);
                beyond |= fmaxf(fabsf(f.x), fmaxf(fabsf(f.y), fabsf(f.z))) > kPlainAbove;
            }
            beyond = __syncthreads_or(beyond) != 0;
            if (beyond) plain_pairs(fnb, pbc, central);
            // without candidate lists: the other images of the bounding-box test,
            // ordered pairs (i, j + shift), S lanes per atom
            if (!lists && any_shift) {
                __syncthreads();
                const int nunits = natoms * S;
                for (int u0 = 0; u0 < nunits; u0 += T) {
                    const int u = u0 + tid;
                    const int i = u / S, sub = u % S;
                    float fx = 0.f, fy = 0.f, fz = 0.f;
                    double e = 0.0;
                    if (i < natoms) {
                        const float4 pi = spos[i];
                        const float4 Ri = sREQ[i];
                        const int4 ng = ngs(i), ngC = ngc(i);
                        for (int iz = -npz; iz <= npz; iz++)
                            for (int iy = -npy; iy <= npy; iy++)
                                for (int ix = -npx; ix <= npx; ix++) {
                                    const int ipbc = ((iz + npz) * nyi + (iy + npy)) * nxi + (ix + npx);
                                    if (ipbc == central || !image_active(ix, iy, iz)) continue;
                                    float ei = 0.f;
                                    B::pair_image_row(spos, sREQ, i, sub, pi, Ri, ng, ngC, pbc, ipbc, ix, iy, iz, nullptr, 0, fx, fy, fz, ei);
                                    if (ENERGY) e += (double)ei;
                                }
                    }
#pragma unroll
                    for (int o = S / 2; o > 0; o >>= 1) {
                        fx += __shfl_xor_sync(0xffffffffu, fx, o);
                        fy += __shfl_xor_sync(0xffffffffu, fy, o);
                        fz += __shfl_xor_sync(0xffffffffu, fz, o);
                    }
                    if (i < natoms && sub == 0 && !beyond) {
                        const float4 a = fnb[i];
                        fnb[i] = make_float4(a.x + fx, a.y + fy, a.z + fz, 0.f);
                    }
                    if (ENERGY) Enb += 0.5 * e;
                }
            }
        } else {
            for (int a = tid; a < natoms; a += T) fnb[a] = make_float4(0, 0, 0, 0);
        }
        // --- GridFF B-spline (unless it ran beside the bonded terms)
        if (!split) B::template grid_phase<ENERGY>(tid, T, fgr, Eg);
        // --- direct substrate term (getSurfMorse), one thread per atom
        if (flags & F_SURF) {
            __syncthreads();
            const float4* sR = at<float4>(L.REQ);
            for (int a = tid; a < natoms; a += T) {
                const float4 p = spos[a];
                const float4 r = surf_atom(P, make_float3(p.x + lv[9], p.y + lv[10], p.z + lv[11]), sR[a]);
                const float4 g = fgr[a];
                fgr[a] = make_float4(g.x + r.x, g.y + r.y, g.z + r.z, 0.f);
                if (ENERGY) Eg += (double)r.w;
            }
        }
    }

    // ------------------------------------------------------------------ phase 2
    // assembled forces; this thread's max |f|^2
    __device__ void assemble(float& fmax2) {
        float4* fasm = at<float4>(L.fasm);
        const float4* fnb = at<float4>(L.fnb);
        const float4* fgr = at<float4>(L.fgrid);
        const float4* fng = at<float4>(L.fng);
        const float4* spos = at<float4>(L.pos);
        for (int v = tid; v < nvecs; v += T) {
            const bool pi = v >= natoms;
            const int ia = pi ? v - natoms : v;
            float3 f = f3(fasm[v]);
            if (!pi) {
                const float4 b = fnb[v], c = fgr[v];
                f = make_float3(f.x + b.x + c.x, f.y + b.y + c.y, f.z + b.z + c.z);
            }
            const int4 bk = bks(ia);
            const int bks[4] = {bk.x, bk.y, bk.z, bk.w};
            const float4* slots = pi ? fng + 4 * L.maxNN : fng;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (bks[k] < 0) break;
                f = f + f3(slots[bks[k]]);
            }
            if (pi) {
                const float3 u = f3(spos[v]);
                f = fma3(u, -dot3(f, u), f);      // Vec3::makeOrthoU
            }
            fasm[v] = make_float4(f.x, f.y, f.z, 0.f);
            fmax2 = fmaxf(fmax2, dot3(f, f));
        }
    }

    // block reduction of 3 doubles + one float max (+flag); result in all threads
    __device__ void reduce4(double& a, double& b, double& c, float& m, bool& bad) {
        double* red = at<double>(L.red);
        a = wsum(a); b = wsum(b); c = wsum(c); m = wmax(m);
        const int anybad = __any_sync(0xffffffffu, bad);
        if (lane == 0) {
            red[4 * warp + 0] = a; red[4 * warp + 1] = b; red[4 * warp + 2] = c;
            reinterpret_cast<float*>(red + 4 * warp + 3)[0] = m;
            reinterpret_cast<int*>(red + 4 * warp + 3)[1] = anybad;
        }
        __syncthreads();
        a = 0; b = 0; c = 0; m = 0.f; int nb = 0;
        for (int w = 0; w < L.nwarps; w++) {
            a += red[4 * w + 0]; b += red[4 * w + 1]; c += red[4 * w + 2];
            m = fmaxf(m, reinterpret_cast<const float*>(red + 4 * w + 3)[0]);
            nb |= reinterpret_cast<const int*>(red + 4 * w + 3)[1];
        }
        bad = nb != 0;
    }
};

// One force (and energy) evaluation per system; blockIdx.x indexes queue[].
template <int T, int S, bool ENERGY>
__global__ void __launch_bounds__(T) eval_kernel(Params P, Systems Y, const int* __restrict__ queue, int nqueue,
                                                 const __grid_constant__ SmemLayout L) {
    extern __shared__ __align__(16) char smem[];
    Engine<T, S, ENERGY> E(P, Y, smem, L);
    const int q = blockIdx.x;
    if (q >= nqueue) return;
    const int s = queue[q];
    E.load(s);
    __syncthreads();
    E.bbox_from_smem();
    double Eb = 0, Enb = 0, Eg = 0;
    E.forces(Eb, Enb, Eg);
    __syncthreads();
    // (the host passes Flim <= 0 here: eval reports unclamped forces)
    float fmax2 = 0.f;
    E.assemble(fmax2);
    float* wm = E.template at<float>(L.red);          // largest force of the system, by warps
    fmax2 = wmax(fmax2);
    if (E.lane == 0) wm[E.warp] = fmax2;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < T / 32; w++) fmax2 = fmaxf(fmax2, wm[w]);
        Y.fconv[s] = sqrtf(fmax2);
    }
    const float4* fasm = E.template at<float4>(L.fasm);
    for (int v = threadIdx.x; v < E.nvecs; v += T) Y.force[E.voff + v] = fasm[v];
    if (ENERGY) {
        // the reference's split: the skipped 1-3 pair energies belong to the
        // pair sum and their subtraction to the bonded part; the total is
        // summed without them
        double eb = Eb, enb = Enb, eg = Eg, x13 = E.e13, z0 = 0.0, z1 = 0.0;
        float dummy = 0.f;
        bool b2 = false;
        __syncthreads();
        E.reduce4(eb, enb, eg, dummy, b2);
        __syncthreads();
        E.reduce4(x13, z0, z1, dummy, b2);
        if (threadIdx.x == 0) Y.energy[s] = make_double4(eb - x13, enb + x13, eg, eb + enb + eg);
    }
}

// B-spline sample of n points (grid parity tests): fe = (Fx, Fy, Fz, E)
__global__ void grid_sample_kernel(Params P, int n, const float4* __restrict__ pos, const float4* __restrict__ PLQ,
                                   float4* __restrict__ fe) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = u >> 2, a = u & 3;
    float4 r = make_float4(0, 0, 0, 0);
    if (i < n) {
        const float4 p = pos[i];
        const float3 uu = make_float3(p.x * P.ginv[0], p.y * P.ginv[1], p.z * P.ginv[2]);
        float4 bx, dx;
        const float3 e = grid_slice(P.grid, P.gn[0], P.gn[1], P.gn[2], uu, PLQ[i], a, bx, dx);
        r = slice_force(e, bx, dx, a);
    }
#pragma unroll
    for (int o = 2; o > 0; o >>= 1) {
        r.x += __shfl_xor_sync(0xffffffffu, r.x, o);
        r.y += __shfl_xor_sync(0xffffffffu, r.y, o);
        r.z += __shfl_xor_sync(0xffffffffu, r.z, o);
        r.w += __shfl_xor_sync(0xffffffffu, r.w, o);
    }
    if (i < n && a == 0) fe[i] = make_float4(r.x * P.gmi[0], r.y * P.gmi[1], r.z * P.gmi[2], r.w);
}


// address of the kernel instantiation for (T, S)
#define MMFF_TS_SWITCH(T, S, ...)                                                            \
    switch (T * 16 + S) {                                                                     \
        case 64 * 16 + 1: { constexpr int T_ = 64, S_ = 1; __VA_ARGS__; }                            \
        case 64 * 16 + 2: { constexpr int T_ = 64, S_ = 2; __VA_ARGS__; }                            \
        case 64 * 16 + 4: { constexpr int T_ = 64, S_ = 4; __VA_ARGS__; }                            \
        case 64 * 16 + 8: { constexpr int T_ = 64, S_ = 8; __VA_ARGS__; }                            \
        case 128 * 16 + 1: { constexpr int T_ = 128, S_ = 1; __VA_ARGS__; }                          \
        case 128 * 16 + 2: { constexpr int T_ = 128, S_ = 2; __VA_ARGS__; }                          \
        case 128 * 16 + 4: { constexpr int T_ = 128, S_ = 4; __VA_ARGS__; }                          \
        case 128 * 16 + 8: { constexpr int T_ = 128, S_ = 8; __VA_ARGS__; }                          \
        case 256 * 16 + 1: { constexpr int T_ = 256, S_ = 1; __VA_ARGS__; }                          \
        case 256 * 16 + 2: { constexpr int T_ = 256, S_ = 2; __VA_ARGS__; }                          \
        case 256 * 16 + 4: { constexpr int T_ = 256, S_ = 4; __VA_ARGS__; }                          \
        case 256 * 16 + 8: { constexpr int T_ = 256, S_ = 8; __VA_ARGS__; }                          \
        case 512 * 16 + 1: { constexpr int T_ = 512, S_ = 1; __VA_ARGS__; }                          \
        case 512 * 16 + 2: { constexpr int T_ = 512, S_ = 2; __VA_ARGS__; }                          \
        case 512 * 16 + 4: { constexpr int T_ = 512, S_ = 4; __VA_ARGS__; }                          \
        case 512 * 16 + 8: { constexpr int T_ = 512, S_ = 8; __VA_ARGS__; }                          \
        default: return nullptr;                                                              \
    }

void* eval_fn(int T, int S, bool energy) {
    if (energy) { MMFF_TS_SWITCH(T, S, return (void*)eval_kernel<T_, S_, true>) }
    MMFF_TS_SWITCH(T, S, return (void*)eval_kernel<T_, S_, false>)
}

}  // namespace mmff
