// mmff_grid.cu -- one-time GridFF construction on the GPU (FP64).
//
//  1. node potentials of a rigid substrate, GridFF::evalBsplineRef semantics
//     with bUseEwald=false (cpp/common/molecular/GridFF.h:847-891):
//       Pauli   sum  sqrt(E0_j) * exp(-2 a (r - R0_j))      (evalGridFFPoint_Mors :582)
//       London  sum -2 sqrt(E0_j) * exp(-a (r - R0_j))
//       Coulomb sum  k_e Q_j / r                             (evalGridFFPoint_Coul :614)
//     Morse over the nPBC_mors images, Coulomb over the nPBC_coul images.  The
//     Coulomb images far from the grid box enter through a tensor-product
//     Chebyshev interpolation of their potential, which is analytic there
//     (see FarPlan in mmff_world.cu); the near ones are summed per node.
//  2. exact cubic B-spline interpolation coefficients: periodic tridiagonal
//     solves along x and y, and a solve with zero coefficients outside the
//     grid along z -- the fixed point the reference's damped-MD least-squares
//     fit (Bspline::fit3D_omp, cpp/common/math/Bspline_fit_3D.h:411-495, bPBC)
//     iterates towards.
//  3. packing to float4 (P, L, Q, 0), z fastest (GridFF::pack_Bspline_d,
//     GridFF.h:1203-1216).
#include <cuda_runtime.h>
#include <stdint.h>

#include "mmff_device.cuh"

namespace mmff {

#define MMFF_COULOMB_D 14.3996448915

// (x, y, z, k_e Q) of a substrate atom
__device__ __forceinline__ double4 charge_scaled(double4 s) { return make_double4(s.x, s.y, s.z, MMFF_COULOMB_D * s.w); }

// Node potentials: Morse sums and the near Coulomb images directly, the far
// ones as sum_c Lz[iz][c] far[ix][iy][c].  One thread takes kGridNX nodes that
// differ in x only, so that the y and z parts of every squared distance and
// the loads of atom and image are shared (FP64 arithmetic is the limit: 8 + 5 /
// kGridNX operations per node, atom and image instead of 18 with a thread per node
// and the library's rsqrt).
__global__ void __launch_bounds__(128) grid_potential_kernel(int nx, int ny, int nz, double3 pos0, double3 step, int nsub,
                                      const double4* __restrict__ sposq,   // (x, y, z, Q)
                                      const double2* __restrict__ sRE,     // (R0, sqrt(E0))
                                      const double3* __restrict__ shm, int nm,
                                      const double3* __restrict__ shc, int nc, double alpha, int pz,
                                      const double* __restrict__ far, const double* __restrict__ Lz,
                                      double* __restrict__ V) {
    const int ngx = (nx + kGridNX - 1) / kGridNX;
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    __shared__ double4 sa[128];
    __shared__ double2 sr[128];
    const bool valid = i < (long)ngx * ny * nz;
    int iz = 0, iy = 0, ix = 0;
    if (valid) { iz = (int)(i % nz); iy = (int)((i / nz) % ny); ix = kGridNX * (int)(i / ((long)nz * ny)); }
    const double px = pos0.x + step.x * ix, py = pos0.y + step.y * iy, pz0 = pos0.z + step.z * iz;
    double vp[kGridNX], vl[kGridNX], vc[kGridNX];
#pragma unroll
    for (int m = 0; m < kGridNX; m++) { vp[m] = 0; vl[m] = 0; vc[m] = 0; }
    for (int t0 = 0; t0 < nsub; t0 += 128) {
        __syncthreads();
        if (t0 + (int)threadIdx.x < nsub) { sa[threadIdx.x] = charge_scaled(sposq[t0 + threadIdx.x]); sr[threadIdx.x] = sRE[t0 + threadIdx.x]; }
        __syncthreads();
        const int nt = min(128, nsub - t0);
        if (!valid) continue;
        for (int a = 0; a < nt; a++) {
            const double4 s = sa[a];
            const double2 r = sr[a];
            const double dx0 = px - s.x, dy0 = py - s.y, dz0 = pz0 - s.z;
            for (int k = 0; k < nm; k++) {
                const double3 sh = shm[k];
                const double dx = dx0 + sh.x, dy = dy0 + sh.y, dz = dz0 + sh.z;
                const double yz = dy * dy + (dz * dz + 1e-32);
#pragma unroll
                for (int m = 0; m < kGridNX; m++) {
                    const double x = dx + m * step.x, r2 = fma(x, x, yz);
                    const double rr = r2 * inv_sqrt64(r2);
                    const double e = exp(-alpha * (rr - r.x));
                    const double eM = e * r.y;
                    vp[m] += eM * e;
                    vl[m] += eM * -2.0;
                }
            }
        }
        // Coulomb: the atoms of one image after another, so that the partial sums
        // stay near the neutral cell's.  (The images of one charge first add up to
        // 10^2 eV, whose last place, 10^-11 eV over the sum, is as large as the last
        // FP32 place of the coefficients some Angstrom above the slab.)
        for (int k = 0; k < nc; k++) {
            const double3 sh = shc[k];
            const double bx = px + sh.x, by = py + sh.y, bz = pz0 + sh.z;
            for (int a = 0; a < nt; a++) {
                const double4 s = sa[a];
                const double dx = bx - s.x, dy = by - s.y, dz = bz - s.z;
                const double yz = dy * dy + (dz * dz + 1e-32);
#pragma unroll
                for (int m = 0; m < kGridNX; m++) {
                    const double x = dx + m * step.x;
                    vc[m] = fma(s.w, inv_sqrt64(fma(x, x, yz)), vc[m]);
                }
            }
        }
    }
    if (!valid) return;
#pragma unroll
    for (int m = 0; m < kGridNX; m++) {
        if (ix + m >= nx) break;
        const long col = (long)(ix + m) * ny + iy;
        double f = 0.0;
        for (int c = 0; c < pz; c++) f = fma(Lz[iz * pz + c], far[col * pz + c], f);
        double* v = V + 3 * (col * nz + iz);
        v[0] = vp[m]; v[1] = vl[m]; v[2] = vc[m] + f;
    }
}

// Coulomb potential of images k0 .. of the far set at the p^3 Chebyshev nodes
// (x slowest): blockIdx.y takes its share of the images, partial[blockIdx.y][node]
__global__ void __launch_bounds__(128) far_potential_kernel(int p, const double* __restrict__ xn,   // node coordinates [3][p]
                                     int nsub, const double4* __restrict__ sposq, const double3* __restrict__ shc,
                                     int nc, double* __restrict__ partial) {
    __shared__ double4 sa[128];
    const int node = blockIdx.x * blockDim.x + threadIdx.x, n3 = p * p * p;
    const bool valid = node < n3;
    const int c = valid ? node : 0;
    const double px = xn[c / (p * p)], py = xn[p + (c / p) % p], pz = xn[2 * p + c % p];
    const int k0 = (int)((long)nc * blockIdx.y / gridDim.y), k1 = (int)((long)nc * (blockIdx.y + 1) / gridDim.y);
    double v = 0.0;
    for (int t0 = 0; t0 < nsub; t0 += 128) {
        __syncthreads();
        if (t0 + (int)threadIdx.x < nsub) sa[threadIdx.x] = charge_scaled(sposq[t0 + threadIdx.x]);
        __syncthreads();
        const int nt = min(128, nsub - t0);
        for (int k = k0; k < k1; k++) {          // (order: see grid_potential_kernel)
            const double3 sh = shc[k];
            const double bx = px + sh.x, by = py + sh.y, bz = pz + sh.z;
            for (int a = 0; a < nt; a++) {
                const double4 s = sa[a];
                const double dx = bx - s.x, dy = by - s.y, dz = bz - s.z;
                v = fma(s.w, inv_sqrt64(fma(dx, dx, fma(dy, dy, dz * dz))), v);
            }
        }
    }
    if (valid) partial[(long)blockIdx.y * n3 + node] = v;
}

// G[a][b][c] = sum over the shares, in order
__global__ void far_sum_kernel(int n3, int nparts, const double* __restrict__ partial, double* __restrict__ G) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n3) return;
    double v = 0.0;
    for (int s = 0; s < nparts; s++) v += partial[(long)s * n3 + i];
    G[i] = v;
}

// contraction of the second index: out[o][n][q] = sum_a M[n][a] in[o][a][q]
__global__ void far_contract_kernel(int no, int n, int p, int nq, const double* __restrict__ M, const double* __restrict__ in,
                                    double* __restrict__ out) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long)no * n * nq) return;
    const int q = (int)(i % nq), k = (int)((i / nq) % n);
    const long o = i / ((long)nq * n);
    double v = 0.0;
    for (int a = 0; a < p; a++) v = fma(M[k * p + a], in[(o * p + a) * nq + q], v);
    out[i] = v;
}

// ---- spline fit: (c[i-1] + 4c[i] + c[i+1]) / 6 = v[i] along one axis.  The
// elimination coefficients depend on the axis length only; the host computes
// them once (cp, inv = 1 / pivot; periodic: z = T^-1 u of the Sherman-Morrison
// correction and 1 / (1 + v.z)), so the lines need no division.  A thread takes
// one channel of one line; consecutive threads take consecutive words.

// z axis: zero outside [0, n).  Lines are contiguous (3 n words): a block
// stages zl of them in shared memory (rows one word longer: no bank
// conflicts), or, zl = 0, works on lines too long for that in place.
__global__ void __launch_bounds__(128) solve_open_kernel(double* __restrict__ C, long nlines, int n, int zl,
                                  const double* __restrict__ cp, const double* __restrict__ inv) {
    extern __shared__ double sl[];
    const int w = 3 * n, ws = w + 1, per = zl > 0 ? zl : 40;
    const long l0 = (long)blockIdx.x * per;
    const int nl = (int)min((long)per, nlines - l0), line = threadIdx.x / 3, ch = threadIdx.x % 3;
    if (zl > 0) {
        for (int i = threadIdx.x; i < nl * w; i += blockDim.x) sl[(i / w) * ws + i % w] = C[l0 * w + i];
        __syncthreads();
    }
    const double a = 1.0 / 6.0;
    if (line < nl) {
        double* y = zl > 0 ? sl + line * ws + ch : C + (l0 + line) * w + ch;
        double u = y[0] * inv[0];
        y[0] = u;
        for (int i = 1; i < n; i++) { u = (y[3 * i] - a * u) * inv[i]; y[3 * i] = u; }
        for (int i = n - 2; i >= 0; i--) { u = y[3 * i] - cp[i] * u; y[3 * i] = u; }
    }
    if (zl > 0) {
        __syncthreads();
        for (int i = threadIdx.x; i < nl * w; i += blockDim.x) C[l0 * w + i] = sl[(i / w) * ws + i % w];
    }
}

// x and y axes: periodic (Sherman-Morrison on the cyclic tridiagonal system).
// Lines l = (outer, inner word): word address outer * outer_stride + inner + i * elem.
__global__ void __launch_bounds__(128) solve_periodic_kernel(double* __restrict__ C, long nlines, int n, long ninner, long outer_stride,
                                      long elem, const double* __restrict__ cp, const double* __restrict__ inv,
                                      const double* __restrict__ z, double rzden, double ag) {
    const long l = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= nlines) return;
    double* y = C + (l / ninner) * outer_stride + l % ninner;
    const double a = 1.0 / 6.0;
    double u = y[0] * inv[0];
    y[0] = u;
#pragma unroll 8
    for (int i = 1; i < n; i++) { u = (y[i * elem] - a * u) * inv[i]; y[i * elem] = u; }
    const double ulast = u;
#pragma unroll 8
    for (int i = n - 2; i >= 0; i--) { u = y[i * elem] - cp[i] * u; y[i * elem] = u; }
    const double fact = (u + ag * ulast) * rzden;
#pragma unroll 8
    for (int i = 0; i < n; i++) y[i * elem] -= fact * z[i];
}

__global__ void pack_grid_kernel(long ntot, const double* __restrict__ C, float4* __restrict__ G) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < ntot) G[i] = make_float4((float)C[3 * i], (float)C[3 * i + 1], (float)C[3 * i + 2], 0.f);
}

}  // namespace mmff
