// ns_kernels.cu -- device kernels of the explicit RHS and SSP-RK3 stage.
//
// Per RK stage (TimeScheme::step, src/time_scheme.cpp:33-66):
//   k_fill_prim      boundary fill + halo exchange of U on the face halos, then
//                    W = prim(U) on every cell (time_scheme.cpp:133-135)
//   k_op_faces       WENO-5 face fluxes along every axis, one thread per face
//                    (Weno5::x/y/z_sweep, Weno5cw::*_sweep), for operator calls;
//                    k_face_flux<d> in FP32
//   k_update         flux differences + centered viscous terms + RK combination
//                    (Weno5::compute_residual, CenteredDiffusion::compute_residual,
//                    TimeScheme::substep), for operator calls and steps without
//                    convection
// (an FP64 time step with convection: ns_stage64.cu and ns_viscous64.cu)
// Per step: k_step_begin (dt reduction over W, then U = cons(W), U0 = U).
#include <cuda_runtime.h>

#include <algorithm>

#include <cfloat>
#include <cmath>

#include "ns_common.cuh"
#include "ns_eos.cuh"
#include "ns_face.cuh"
#include "ns_face64.cuh"
#include "ns_kernels.h"
#include "ns_tcgen05.cuh"
#include "ns_viscous.cuh"

namespace nsb {

// ---------------------------------------------------------------------------
// step begin: dt from W at the step start (TimeScheme::set_dt), then
// U = cons(W) on every cell (time_scheme.cpp:124) and U0 = U (:126), also on
// every cell.
// FROM_U: the state is U after the previous step; W = prim(U) first
// (time_scheme.cpp:69).  Grid: (ceil(NZp/32), ceil(NY/4), NX).

template <bool FROM_U, bool PHYS>
__global__ void __launch_bounds__(128) k_step_begin(double* __restrict__ W, double* __restrict__ U,
                                                    double* __restrict__ U0, Box b, Consts c,
                                                    unsigned long long* __restrict__ slot, int ih0) {
    int kh = blockIdx.x * 32 + threadIdx.x;
    int jh = blockIdx.y * 4 + threadIdx.y;
    int ih = blockIdx.z + ih0;
    double best = INFINITY;
    if (kh < b.nz + 2 * NG && jh < b.NY) {
        long long o = b.at(ih, jh, kh);
        double w[5], u[5];
        if (FROM_U) {
#pragma unroll
            for (int q = 0; q < 5; q++) u[q] = U[q * b.fstride + o];
            prim_from_cons(u, c.gm1, w);
#pragma unroll
            for (int q = 0; q < 5; q++) W[q * b.fstride + o] = w[q];
        } else {
#pragma unroll
            for (int q = 0; q < 5; q++) w[q] = W[q * b.fstride + o];
        }
        bool interior = ih >= NG && ih < b.nx + NG && jh >= NG && jh < b.ny + NG && kh >= NG &&
                        kh < b.nz + NG;
        if (interior) {
            double dt = PHYS ? local_dt_physical(w, c) : local_dt(w, c);
            if (dt < best) best = dt;  // NaN never lowers the minimum (time_scheme.cpp:117)
        }
        cons_from_prim(w, c.inv_gm1, u);
#pragma unroll
        for (int q = 0; q < 5; q++) {
            U[q * b.fstride + o] = u[q];
            U0[q * b.fstride + o] = u[q];  // all cells: the stages that start from U0 keep its edges
        }
    }
    block_min_to(best, slot);
}

// W = prim(U) on every cell (end of TimeScheme::step, time_scheme.cpp:69)
__global__ void __launch_bounds__(128) k_prim_all(double* __restrict__ W, const double* __restrict__ U,
                                                  Box b, Consts c, int ih0) {
    int kh = blockIdx.x * 32 + threadIdx.x;
    int jh = blockIdx.y * 4 + threadIdx.y;
    int ih = blockIdx.z + ih0;
    if (kh >= b.nz + 2 * NG || jh >= b.NY) return;
    long long o = b.at(ih, jh, kh);
    double u[5], w[5];
#pragma unroll
    for (int q = 0; q < 5; q++) u[q] = U[q * b.fstride + o];
    prim_from_cons(u, c.gm1, w);
#pragma unroll
    for (int q = 0; q < 5; q++) W[q * b.fstride + o] = w[q];
}

// U = cons(W) on every cell
__global__ void __launch_bounds__(128) k_cons_all(const double* __restrict__ W, double* __restrict__ U,
                                                  Box b, Consts c) {
    int kh = blockIdx.x * 32 + threadIdx.x;
    int jh = blockIdx.y * 4 + threadIdx.y;
    int ih = blockIdx.z;
    if (kh >= b.nz + 2 * NG || jh >= b.NY) return;
    long long o = b.at(ih, jh, kh);
    double u[5], w[5];
#pragma unroll
    for (int q = 0; q < 5; q++) w[q] = W[q * b.fstride + o];
    cons_from_prim(w, c.inv_gm1, u);
#pragma unroll
    for (int q = 0; q < 5; q++) U[q * b.fstride + o] = u[q];
}

// CFL minimum over the interior of W (TimeScheme::get_local_max_dt, time_scheme.cpp:98-125)
template <bool PHYS>
__global__ void __launch_bounds__(128) k_min_dt(const double* __restrict__ W, Box b, Consts c,
                                                unsigned long long* __restrict__ slot) {
    int k = blockIdx.x * 32 + threadIdx.x;
    int j = blockIdx.y * 4 + threadIdx.y;
    int i = blockIdx.z;
    double best = INFINITY;
    if (k < b.nz && j < b.ny) {
        long long o = b.at(i + NG, j + NG, k + NG);
        double w[5];
#pragma unroll
        for (int q = 0; q < 5; q++) w[q] = W[q * b.fstride + o];
        double dt = PHYS ? local_dt_physical(w, c) : local_dt(w, c);
        if (dt < best) best = dt;
    }
    block_min_to(best, slot);
}

// ---------------------------------------------------------------------------
// stage prologue: Neumann copy / periodic wrap of U on the face halos
// (boundary_neumann.cpp:22-132, communicator.cpp:6-143: face regions only),
// then W = prim(U) on every cell (eq_of_state.cpp:61-87).

__global__ void __launch_bounds__(128) k_fill_prim(double* __restrict__ W, double* __restrict__ U,
                                                   Box b, Consts c) {
    int kh = blockIdx.x * 32 + threadIdx.x;
    int jh = blockIdx.y * 4 + threadIdx.y;
    int ih = blockIdx.z;
    if (kh >= b.nz + 2 * NG || jh >= b.NY) return;
    int i = ih - NG, j = jh - NG, k = kh - NG;
    bool ox = i < 0 || i >= b.nx, oy = j < 0 || j >= b.ny, oz = k < 0 || k >= b.nz;
    // a slab's exchanged x ghost plane holds a neighbour's cells: its y and z ghost
    // rows fold within the plane like those of an interior plane
    if (ox && x_exchanged(i >= b.nx, b.nx, c)) ox = false;
    long long o = b.at(ih, jh, kh);
    double u[5], w[5];
    if ((int)ox + (int)oy + (int)oz == 1) {
        int si = ox ? fold(i, b.nx, c.periodic[0]) : i;
        int sj = oy ? fold(j, b.ny, c.periodic[1]) : j;
        int sk = oz ? fold(k, b.nz, c.periodic[2]) : k;
        long long s = b.at(si + NG, sj + NG, sk + NG);
#pragma unroll
        for (int q = 0; q < 5; q++) {
            u[q] = U[q * b.fstride + s];
            U[q * b.fstride + o] = u[q];
        }
    } else {
#pragma unroll
        for (int q = 0; q < 5; q++) u[q] = U[q * b.fstride + o];
    }
    prim_from_cons(u, c.gm1, w);
#pragma unroll
    for (int q = 0; q < 5; q++) W[q * b.fstride + o] = w[q];
}

// An FP64 stage's W from its input U: W = prim(U) of the cell that each cell folds
// onto, ghost cells beyond edges and corners too (the mixed derivatives of the
// viscous terms read them); U's own ghost cells are left as they are, except that a
// slab's exchanged x ghost planes are neighbours' cells.  On every cell of the planes
// from ih0 on, or (SHELL) on the ghost cells alone.  Grid: cells as k_fill_prim's, or
// (ceil(cells / 128), 3 parts of the shell: x ghost planes, y ghost rows, z ghost cells).
template <bool PHYS, bool SHELL>
__global__ void __launch_bounds__(128) k_fill_w(double* __restrict__ W, const double* __restrict__ U, Box b, Consts c,
                                                int ih0) {
    const int NZ = b.nz + 2 * NG;
    int i, j, k;
    if constexpr (SHELL) {
        const long long t = (long long)blockIdx.x * 128 + threadIdx.x;
        const int part = blockIdx.y;
        const int n0 = part == 0 ? 2 * NG : b.nx, n1 = part == 0 ? b.NY : (part == 1 ? 2 * NG : b.ny),
                  n2 = part == 2 ? 2 * NG : NZ;
        if (t >= (long long)n0 * n1 * n2) return;
        const int a0 = (int)(t / ((long long)n1 * n2)), a1 = (int)(t / n2 % n1), a2 = (int)(t % n2);
        auto ghost = [](int a, int n) { return a < NG ? a - NG : a - NG + n; };
        i = part == 0 ? ghost(a0, b.nx) : a0;
        j = part == 0 ? a1 - NG : (part == 1 ? ghost(a1, b.ny) : a1);
        k = part == 2 ? ghost(a2, b.nz) : a2 - NG;
    } else {
        k = blockIdx.x * 32 + threadIdx.x - NG;
        j = blockIdx.y * 4 + threadIdx.y - NG;
        i = blockIdx.z + ih0 - NG;
        if (k >= b.nz + NG || j >= b.ny + NG) return;
    }
    const long long s = b.at(fold_x(i, b.nx, c) + NG, fold(j, b.ny, c.periodic[1]) + NG, fold(k, b.nz, c.periodic[2]) + NG);
    double u[5], w[5];
#pragma unroll
    for (int q = 0; q < 5; q++) u[q] = U[q * b.fstride + s];
    prim_from_cons(u, c.gm1, w);
    store_w<PHYS>(W, b.fstride, b.at(i + NG, j + NG, k + NG), w, c.gamma);
}

// The face halos of U that a step leaves behind (the regions
// apply_boundary_conditions + communicate fill): the third stage's input Us at the cell
// each folds onto.  Grid: (ceil(3 * max face area / 128), 6 regions: x-, x+, y-, y+, z-, z+).
__global__ void __launch_bounds__(128) k_fill_uhalo(double* __restrict__ U, const double* __restrict__ Us, Box b,
                                                    Consts c) {
    const int ax = blockIdx.y >> 1, hi = blockIdx.y & 1;
    const long long t = (long long)blockIdx.x * 128 + threadIdx.x;
    // on a slab the y and z ghost rows of exchanged x ghost planes are filled too
    const int ilo = x_exchanged(0, b.nx, c) ? -NG : 0, ihi = b.nx + (x_exchanged(1, b.nx, c) ? NG : 0);
    const int nxe = ihi - ilo;
    int i, j, k, layer;
    if (ax == 0) {
        if (t >= 3LL * b.ny * b.nz) return;
        k = (int)(t % b.nz); j = (int)((t / b.nz) % b.ny); layer = (int)(t / ((long long)b.nz * b.ny));
        i = hi ? b.nx + layer : layer - NG;
    } else if (ax == 1) {
        if (t >= 3LL * nxe * b.nz) return;
        k = (int)(t % b.nz); i = ilo + (int)((t / b.nz) % nxe); layer = (int)(t / ((long long)b.nz * nxe));
        j = hi ? b.ny + layer : layer - NG;
    } else {
        if (t >= 3LL * nxe * b.ny) return;
        layer = (int)(t % 3); j = (int)((t / 3) % b.ny); i = ilo + (int)(t / (3LL * b.ny));
        k = hi ? b.nz + layer : layer - NG;
    }
    const long long o = b.at(i + NG, j + NG, k + NG);
    const int sj = ax == 1 ? fold(j, b.ny, c.periodic[1]) : j;
    const int sk = ax == 2 ? fold(k, b.nz, c.periodic[2]) : k;
    const long long src = b.at(fold_x(i, b.nx, c) + NG, sj + NG, sk + NG);
#pragma unroll
    for (int q = 0; q < 5; q++) U[q * b.fstride + o] = Us[q * b.fstride + src];
}

// ---------------------------------------------------------------------------
// WENO-5 face fluxes (device functions in ns_face.cuh)

// Minimum resident blocks per SM requested from the register allocator for the
// FP32 face kernels (128 threads each), chosen by a sweep on B200 at 256^3 (1, 5, 6
// characteristic-wise): the cap trades a few spilled registers for 20 resident warps
// instead of 8.
template <bool CHAR>
struct FaceMinBlocks {
    static constexpr int value = CHAR ? 5 : 1;
};

// Every face of an FP64 operator call from the caller's W and U, one thread per face,
// the axes one after the other in one launch (blocks n0, n1, n2 of the axes).  The
// grids of these calls are small and their launches latency: three axes with a launch
// each and two more for the last planes of y and z took 61 us of a 48x60x52 residual.
struct OpFaces {
    double* F[3];
    FaceBox fb[3];
    unsigned blocks[3];
};
template <int DIR, bool CHAR, bool BORGES, bool PHYS>
__device__ __forceinline__ void op_face(const double* __restrict__ W, const double* __restrict__ U, const Box& b,
                                        const Consts& c, const OpFaces& o, unsigned block) {
    const FaceBox& fb = o.fb[DIR];
    const long long e = (long long)block * 128 + threadIdx.x;
    if (e >= (long long)fb.n0 * fb.n1 * fb.n2) return;
    const int kk = (int)(e % fb.n2), bb = (int)(e / fb.n2 % fb.n1), aa = (int)(e / fb.n2 / fb.n1);
    long long step;
    const long long o0 = face_origin<DIR>(b, aa, bb, kk, step);
    double f[5];
    face_flux64_wu<DIR, CHAR, BORGES, PHYS>(W, U, b, c, o0, step, f);
#pragma unroll
    for (int q = 0; q < 5; q++) o.F[DIR][q * fb.fstride + e] = f[q];
}
template <bool CHAR, bool BORGES, bool PHYS>
__global__ void __launch_bounds__(128, 3)
    k_op_faces(const double* __restrict__ W, const double* __restrict__ U, Box b, Consts c, OpFaces o) {
    if (blockIdx.x < o.blocks[0]) op_face<0, CHAR, BORGES, PHYS>(W, U, b, c, o, blockIdx.x);
    else if (blockIdx.x < o.blocks[0] + o.blocks[1]) op_face<1, CHAR, BORGES, PHYS>(W, U, b, c, o, blockIdx.x - o.blocks[0]);
    else op_face<2, CHAR, BORGES, PHYS>(W, U, b, c, o, blockIdx.x - o.blocks[0] - o.blocks[1]);
}

// one face of an FP32 operator call
template <int DIR, bool CHAR, bool BORGES, bool PHYS>
__device__ __forceinline__ void face_at(const double* __restrict__ W, const double* __restrict__ U,
                                        const Box& b, const Consts& c, float* __restrict__ F,
                                        const FaceBox& fb, int aa, int bb, int kk) {
    long long step;
    long long o0 = face_origin<DIR>(b, aa, bb, kk, step);
    float fL[5][5], fR[5][5], wa[5], out[5];
    face_stencil<DIR, CHAR, PHYS, float>(W, U, b, c, o0, step, fL, fR, wa);
    if constexpr (!CHAR)
        face_comp<float, BORGES>(fL, fR, out);
    else
        face_char<DIR, PHYS, float, BORGES>(fL, fR, wa, float(c.gamma), float(c.inv_gm1), out);
    long long fo = fb.at(aa, bb, kk);
#pragma unroll
    for (int q = 0; q < 5; q++) F[q * fb.fstride + fo] = out[q];
}

// FP32 faces of one (i, j) tile row of 32 k-faces per warp, 4 rows per block.  Along
// y and z the last face plane (j = ny, k = nz) is left to k_face_flux_tail: as
// a 33rd k-face or a 4th-of-4 row it would occupy a whole block for one live
// lane or warp per block.
template <int DIR, bool CHAR, bool BORGES, bool PHYS>
__global__ void __launch_bounds__(128, FaceMinBlocks<CHAR>::value)
    k_face_flux(const double* __restrict__ W, const double* __restrict__ U, Box b, Consts c,
                float* __restrict__ F, FaceBox fb) {
    int kk = blockIdx.x * 32 + threadIdx.x;
    int bb = blockIdx.y * 4 + threadIdx.y;
    int aa = blockIdx.z;
    if (kk >= fb.n2 - (DIR == 2) || bb >= fb.n1 - (DIR == 1)) return;
    face_at<DIR, CHAR, BORGES, PHYS>(W, U, b, c, F, fb, aa, bb, kk);
}

// The last face plane along y (j = ny, threads along k) or z (k = nz, threads
// along j), one face per thread.
template <int DIR, bool CHAR, bool BORGES, bool PHYS>
__global__ void __launch_bounds__(128, FaceMinBlocks<CHAR>::value)
    k_face_flux_tail(const double* __restrict__ W, const double* __restrict__ U, Box b, Consts c,
                     float* __restrict__ F, FaceBox fb) {
    static_assert(DIR > 0, "x-faces have no tail plane");
    const int r = blockIdx.x * 128 + threadIdx.x, aa = blockIdx.y;
    if (r >= (DIR == 1 ? fb.n2 : fb.n1)) return;
    const int bb = DIR == 1 ? fb.n1 - 1 : r, kk = DIR == 1 ? r : fb.n2 - 1;
    face_at<DIR, CHAR, BORGES, PHYS>(W, U, b, c, F, fb, aa, bb, kk);
}

// ---------------------------------------------------------------------------
// centered viscous terms, reference semantics (CenteredDiffusion::compute_residual,
// src/diffusion_schemes/centered_diffusion.cpp:70-182 with the stress helpers of
// diffusion_scheme.cpp:3-58; dmu = 0 terms dropped, which is exact).
//   - d2/dy2 applies the x-stencil scaled by 1/dy^2 (cd-n.cpp:77)
//   - Tauyy = tauxx (:143); the x work term uses Tauxy*dv_dy (:148);
//     the y heat-flux term multiplies by 1 where the pressure belongs (:166)
//   - 2D terms only; rhoW untouched (:173-176)
//   - mixed derivatives differentiate first derivatives that are zero outside
//     the interior along a non-periodic axis (derivative halos are only filled
//     by the periodic exchange, :22-24)

template <int H, typename TV>
__device__ __forceinline__ void viscous_reference(const double* __restrict__ W, const Box& b,
                                                  const Consts& c, int i, int j, int k, TV r[5]) {
    const long long fs = b.fstride;
    const long long sx = (long long)b.NY * b.NZp, sy = b.NZp;
    const long long o = b.at(i + NG, j + NG, k + NG);
    TV cx1[2 * H + 1], cy1[2 * H + 1], cxx[2 * H + 1], cyy[2 * H + 1];
#pragma unroll
    for (int t = 0; t <= 2 * H; t++) {
        cx1[t] = TV(c.df[3 - H + t] * c.inv_dx);
        cy1[t] = TV(c.df[3 - H + t] * c.inv_dy);
        cxx[t] = TV(c.ddf[3 - H + t] * c.inv_dx * c.inv_dx);
        cyy[t] = TV(c.ddf[3 - H + t] * c.inv_dy * c.inv_dy);
    }
    // first and second derivatives of rho, p, u, v at the cell
    TV Dx[4], Dy[4], Dxx[4], Dyy[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        TV sx1 = 0, sy1 = 0, sxx = 0, syy = 0;
#pragma unroll
        for (int t = 0; t <= 2 * H; t++) {
            TV wx = TV(W[q * fs + o + (t - H) * sx]);
            TV wy = TV(W[q * fs + o + (t - H) * sy]);
            if (t != H) { sx1 += wx * cx1[t]; sy1 += wy * cy1[t]; }
            sxx += wx * cxx[t];
            syy += wx * cyy[t];
        }
        Dx[q] = sx1; Dy[q] = sy1; Dxx[q] = sxx; Dyy[q] = syy;
    }
    // mixed derivatives of u (q=2) and v (q=3)
    TV Dxy[2], Dyx[2];
#pragma unroll
    for (int v = 0; v < 2; v++) {
        const int q = 2 + v;
        TV sxy = 0, syx = 0;
#pragma unroll
        for (int s = 0; s <= 2 * H; s++) {
            if (s == H) continue;
            // The loads run unconditionally from the wrapped (always valid) row or
            // column, so that they issue together; a term outside a non-periodic
            // axis is then dropped by a select.
            // d/dy of (d/dx W) at row j+s-H
            const int jj = j + s - H;
            {
                const int jw = fold(jj, b.ny, 1);
                const long long ob = b.at(i + NG, jw + NG, k + NG);
                TV dx = 0;
#pragma unroll
                for (int t = 0; t <= 2 * H; t++)
                    if (t != H) dx += TV(W[q * fs + ob + (t - H) * sx]) * cx1[t];
                if ((jj >= 0 && jj < b.ny) || c.periodic[1]) sxy += dx * cy1[s];
            }
            // d/dx of (d/dy W) at column i+s-H
            const int ii = i + s - H;
            {
                const int iw = c.ext_x ? ii : fold(ii, b.nx, 1);
                const long long ob = b.at(iw + NG, j + NG, k + NG);
                TV dy = 0;
#pragma unroll
                for (int t = 0; t <= 2 * H; t++)
                    if (t != H) dy += TV(W[q * fs + ob + (t - H) * sy]) * cy1[t];
                if (x_inside(ii, b.nx, c)) syx += dy * cx1[s];
            }
        }
        Dxy[v] = sxy; Dyx[v] = syx;
    }
    viscous_reference_terms<TV>(Dx, Dy, Dxx, Dyy, Dxy, Dyx, TV(W[2 * fs + o]), TV(W[3 * fs + o]),
                                TV(W[1 * fs + o]), TV(W[o]), c, r);
}

// Physical semantics: full 3D viscous stress and heat flux with constant mu
// (no reference counterpart).  Derivatives along one axis read the
// boundary-filled W as it is (ghost cells included); a mixed derivative also
// reads edge and corner cells, which no fill writes, so its offsets are folded
// back into the interior along each axis (periodic wrap or Neumann clamp; a
// slab's x ghost planes are the neighbours' cells and stay).  All axis loops
// unroll at compile time (2D skips the z terms at run time) and the folded
// offsets are formed once per axis.
template <int H, typename TV>
__device__ __forceinline__ void viscous_physical(const double* __restrict__ W, const Box& b,
                                                 const Consts& c, int i, int j, int k, TV r[5]) {
    constexpr int NS = 2 * H + 1;
    const long long fs = b.fstride;
    const long long st3[3] = {(long long)b.NY * b.NZp, (long long)b.NZp, 1};
    const long long o = b.at(i + NG, j + NG, k + NG);
    const bool three = c.dim == 3;
    const double inv[3] = {c.inv_dx, c.inv_dy, c.inv_dz};
    const int n3[3] = {b.nx, b.ny, b.nz};
    const int c3[3] = {i, j, k};
    // offsets of the folded stencil cells along each axis, and the CD coefficients
    long long off[3][NS];
    TV c1[3][NS], c2[3][NS];
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int t = 0; t < NS; t++) {
            const int v = c3[a] + t - H;
            const int f = (a == 0) ? fold_x(v, n3[0], c) : fold(v, n3[a], c.periodic[a]);
            off[a][t] = (long long)(f - c3[a]) * st3[a];
            c1[a][t] = TV(c.df[3 - H + t] * inv[a]);
            c2[a][t] = TV(c.ddf[3 - H + t] * inv[a] * inv[a]);
        }
    TV gu[3][3], lap[3], gdiv[3], lapT = 0;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        lap[a] = 0;
        gdiv[a] = 0;
#pragma unroll
        for (int bx = 0; bx < 3; bx++) gu[a][bx] = 0;
    }
#pragma unroll
    for (int bx = 0; bx < 3; bx++) {
        if (bx == 2 && !three) continue;
#pragma unroll
        for (int t = 0; t < NS; t++) {
            const long long oo = o + (t - H) * st3[bx];
            const TV T = TV(W[1 * fs + oo]) / TV(W[oo]);
#pragma unroll
            for (int a = 0; a < 3; a++) {
                const TV va = TV(W[(2 + a) * fs + oo]);
                if (t != H) gu[a][bx] += va * c1[bx][t];
                lap[a] += va * c2[bx][t];
                if (a == bx) gdiv[a] += va * c2[bx][t];
            }
            lapT += T * c2[bx][t];
        }
    }
    // grad(div u)_a += d/dx_a (d u_b / dx_b) for b != a
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int bx = 0; bx < 3; bx++) {
            if (a == bx || ((a == 2 || bx == 2) && !three)) continue;
            TV acc = 0;
#pragma unroll
            for (int s = 0; s < NS; s++) {
                if (s == H) continue;
                TV inner = 0;
#pragma unroll
                for (int t = 0; t < NS; t++) {
                    if (t == H) continue;
                    inner += TV(W[(2 + bx) * fs + o + off[a][s] + off[bx][t]]) * c1[bx][t];
                }
                acc += inner * c1[a][s];
            }
            gdiv[a] += acc;
        }
    const TV mu = TV(c.mu), lamb = TV(c.lamb);
    const TV uv[3] = {TV(W[2 * fs + o]), TV(W[3 * fs + o]), TV(W[4 * fs + o])};
    const TV div = gu[0][0] + gu[1][1] + gu[2][2];
    TV work = 0, diss = 0, mom[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        mom[a] = mu * lap[a] + (mu + lamb) * gdiv[a];
        work += uv[a] * mom[a];
    }
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int bx = 0; bx < 3; bx++) {
            const TV tab = mu * (gu[a][bx] + gu[bx][a]) + (a == bx ? lamb * div : TV(0));
            diss += tab * gu[a][bx];
        }
    r[2] -= mom[0];
    r[3] -= mom[1];
    r[4] -= mom[2];
    r[1] -= work + diss + TV(c.heat) * mu * lapT;
}

// ---------------------------------------------------------------------------
// cell update: R = sum_d (f_d(+) - f_d(-))/d  (+ viscous), then
//   MODE_STAGE: U = U0*m1 + U*m2 + R*(mc*dt)    (TimeScheme::substep, time_scheme.cpp:72-96)
//   MODE_RHS  : Rout += R
// dt = CFL * min(1e10, reduced minimum) (time_scheme.cpp:98-136).

// The update kernel is memory-latency bound; 8 resident blocks (64 registers)
// matched the compiler's own choice and beat looser bounds in a B200 sweep.
#ifndef NS_UPDATE_MINB
#define NS_UPDATE_MINB 8
#endif
template <int MODE, int H, bool PHYS, typename TF, typename TV>
__global__ void __launch_bounds__(128, NS_UPDATE_MINB) k_update(const double* __restrict__ W, double* __restrict__ U,
                                                const double* __restrict__ U0,
                                                const TF* __restrict__ Fx, const TF* __restrict__ Fy,
                                                const TF* __restrict__ Fz, Box b, FaceBox fx,
                                                FaceBox fy, FaceBox fz, Consts c, int flags,
                                                const unsigned long long* __restrict__ slot,
                                                double m1, double m2, double mc,
                                                double* __restrict__ Rout, double* __restrict__ clock) {
    int k = blockIdx.x * 32 + threadIdx.x;
    int j = blockIdx.y * 4 + threadIdx.y;
    int i = blockIdx.z;
    if (k >= b.nz || j >= b.ny) return;
    double r[5] = {0, 0, 0, 0, 0};
    if (flags & UPD_CONV) {
#pragma unroll
        for (int q = 0; q < 5; q++) {
            r[q] += (double(Fx[q * fx.fstride + fx.at(i + 1, j, k)]) -
                     double(Fx[q * fx.fstride + fx.at(i, j, k)])) * c.inv_dx;
            r[q] += (double(Fy[q * fy.fstride + fy.at(i, j + 1, k)]) -
                     double(Fy[q * fy.fstride + fy.at(i, j, k)])) * c.inv_dy;
            if (flags & UPD_CONVZ)
                r[q] += (double(Fz[q * fz.fstride + fz.at(i, j, k + 1)]) -
                         double(Fz[q * fz.fstride + fz.at(i, j, k)])) * c.inv_dz;
        }
    }
    if constexpr (H > 0) {
        TV rv[5] = {0, 0, 0, 0, 0};
        if constexpr (PHYS)
            viscous_physical<H, TV>(W, b, c, i, j, k, rv);
        else
            viscous_reference<H, TV>(W, b, c, i, j, k, rv);
#pragma unroll
        for (int q = 1; q < 5; q++) r[q] += double(rv[q]);
    }
    long long o = b.at(i + NG, j + NG, k + NG);
    if constexpr (MODE == MODE_STAGE) {
        double mn = __longlong_as_double((long long)*slot);
        double dt = fmin(1e10, mn) * c.cfl;
        double m3 = mc * dt;
        if (clock && (blockIdx.x | blockIdx.y | blockIdx.z | threadIdx.x | threadIdx.y) == 0) {
            clock[0] = dt;
            clock[1] += dt;
        }
#pragma unroll
        for (int q = 0; q < 5; q++) {
            long long a = q * b.fstride + o;
            U[a] = (U0[a] * m1) + (U[a] * m2) + (r[q] * m3);
        }
    } else {
        if (flags & UPD_OVERWRITE) {
#pragma unroll
            for (int q = 0; q < 5; q++) Rout[q * b.fstride + o] = r[q];
        } else {
#pragma unroll
            for (int q = 0; q < 5; q++) Rout[q * b.fstride + o] += r[q];
        }
    }
}

// ---------------------------------------------------------------------------
// error bounds of div_pos_nr against the IEEE quotient and of rsqrt_pos_nr
// against CUDA's rsqrt: n pairs with x log-uniform in [1e-3, 1e3] and d
// log-uniform in [1e-60, 1e60] (SplitMix64 draws); max_ulp[0], max_ulp[1]
// receive the largest distances in units in the last place

__device__ __forceinline__ unsigned long long splitmix64(unsigned long long z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__global__ void k_div_check(long long n, unsigned long long seed, unsigned long long* __restrict__ max_ulp) {
    unsigned long long worst = 0, worst_r = 0;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const double u = (splitmix64(seed + 2 * e) >> 11) * 0x1.0p-53;
        const double v = (splitmix64(seed + 2 * e + 1) >> 11) * 0x1.0p-53;
        const double x = exp10(-3.0 + 6.0 * u), d = exp10(-60.0 + 120.0 * v);
        const long long a = __double_as_longlong(div_pos_nr(x, d)), b = __double_as_longlong(x / d);
        const unsigned long long dist = (unsigned long long)(a > b ? a - b : b - a);
        if (dist > worst) worst = dist;
        // 1/sqrt(d) against CUDA's rsqrt (itself within an ulp)
        const long long ra = __double_as_longlong(rsqrt_pos_nr(d)), rb = __double_as_longlong(rsqrt(d));
        const unsigned long long rdist = (unsigned long long)(ra > rb ? ra - rb : rb - ra);
        if (rdist > worst_r) worst_r = rdist;
    }
    atomicMax(max_ulp, worst);
    atomicMax(max_ulp + 1, worst_r);
}

cudaError_t launch_div_check(long long n, unsigned long long seed, unsigned long long* max_ulp, cudaStream_t s) {
    k_div_check<<<256, 256, 0, s>>>(n, seed, max_ulp);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// host <-> device layout transposes (reference AoS [i][j][k][q], unpadded
// (nx+6)(ny+6)(nz+6) x 5  <->  device SoA planes)

__global__ void __launch_bounds__(128) k_aos_to_soa(const double* __restrict__ A, double* __restrict__ S,
                                                    Box b, int ih0) {
    int kh = blockIdx.x * 32 + threadIdx.x;
    int jh = blockIdx.y * 4 + threadIdx.y;
    int ih = blockIdx.z + ih0;
    int NZ = b.nz + 2 * NG;
    if (kh >= NZ || jh >= b.NY) return;
    long long a = (((long long)ih * b.NY + jh) * NZ + kh) * 5;
    long long o = b.at(ih, jh, kh);
#pragma unroll
    for (int q = 0; q < 5; q++) S[q * b.fstride + o] = A[a + q];
}

__global__ void __launch_bounds__(128) k_soa_to_aos(const double* __restrict__ S, double* __restrict__ A,
                                                    Box b, int ih0) {
    int kh = blockIdx.x * 32 + threadIdx.x;
    int jh = blockIdx.y * 4 + threadIdx.y;
    int ih = blockIdx.z + ih0;
    int NZ = b.nz + 2 * NG;
    if (kh >= NZ || jh >= b.NY) return;
    long long a = (((long long)ih * b.NY + jh) * NZ + kh) * 5;
    long long o = b.at(ih, jh, kh);
#pragma unroll
    for (int q = 0; q < 5; q++) A[a + q] = S[q * b.fstride + o];
}

// ---------------------------------------------------------------------------
// slab halo exchange (Communicator::communicate_x_direction, src/communicator.cpp:16-57,
// with the slices of src/containers/array_4d.cpp:39-84): the outer three interior
// planes of one side packed as [q][layer][j][k], interior j and k; unpack writes
// the same layout into the ghost planes of that side.
__global__ void __launch_bounds__(128) k_slab_pack(const double* __restrict__ U, Box b, int side,
                                                   double* __restrict__ buf) {
    const long long n = 3LL * b.ny * b.nz, t = (long long)blockIdx.x * 128 + threadIdx.x;
    if (t >= 5 * n) return;
    const int q = (int)(t / n);
    const long long r = t % n;
    const int layer = (int)(r / ((long long)b.ny * b.nz)), j = (int)((r / b.nz) % b.ny), k = (int)(r % b.nz);
    const int i = side ? b.nx - NG + layer : layer;
    buf[t] = U[q * b.fstride + b.at(i + NG, j + NG, k + NG)];
}

__global__ void __launch_bounds__(128) k_slab_unpack(double* __restrict__ U, Box b, int side,
                                                     const double* __restrict__ buf) {
    const long long n = 3LL * b.ny * b.nz, t = (long long)blockIdx.x * 128 + threadIdx.x;
    if (t >= 5 * n) return;
    const int q = (int)(t / n);
    const long long r = t % n;
    const int layer = (int)(r / ((long long)b.ny * b.nz)), j = (int)((r / b.nz) % b.ny), k = (int)(r % b.nz);
    const int i = side ? b.nx + layer : layer - NG;
    U[q * b.fstride + b.at(i + NG, j + NG, k + NG)] = buf[t];
}

// ---------------------------------------------------------------------------
// global diagnostics over the interior (FP64): sums of conserved variables,
// kinetic energy, enstrophy (second-order central curl), non-finite count.
__global__ void __launch_bounds__(128) k_diagnostics(const double* __restrict__ U, Box b, Consts c,
                                                     double* __restrict__ acc) {
    int k = blockIdx.x * 32 + threadIdx.x;
    int j = blockIdx.y * 4 + threadIdx.y;
    int i = blockIdx.z;
    double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (k < b.nz && j < b.ny) {
        long long o = b.at(i + NG, j + NG, k + NG);
        double u[5];
        bool bad = false;
#pragma unroll
        for (int q = 0; q < 5; q++) {
            u[q] = U[q * b.fstride + o];
            bad |= !isfinite(u[q]);
        }
        double dV = c.dx * c.dy * c.dz;
        v[0] = u[0] * dV;
        v[1] = u[2] * dV;
        v[2] = u[3] * dV;
        v[3] = u[4] * dV;
        v[4] = u[1] * dV;
        v[5] = 0.5 * (u[2] * u[2] + u[3] * u[3] + u[4] * u[4]) / u[0] * dV;
        // velocity of neighbours through the periodic/clamped index map
        auto vel = [&](int ii, int jj, int kk, int a) {
            ii = fold_x(ii, b.nx, c);
            jj = fold(jj, b.ny, c.periodic[1]);
            kk = fold(kk, b.nz, c.periodic[2]);
            long long oo = b.at(ii + NG, jj + NG, kk + NG);
            return U[(2 + a) * b.fstride + oo] / U[oo];
        };
        double dwdy = (vel(i, j + 1, k, 2) - vel(i, j - 1, k, 2)) * 0.5 * c.inv_dy;
        double dvdz = (vel(i, j, k + 1, 1) - vel(i, j, k - 1, 1)) * 0.5 * c.inv_dz;
        double dudz = (vel(i, j, k + 1, 0) - vel(i, j, k - 1, 0)) * 0.5 * c.inv_dz;
        double dwdx = (vel(i + 1, j, k, 2) - vel(i - 1, j, k, 2)) * 0.5 * c.inv_dx;
        double dvdx = (vel(i + 1, j, k, 1) - vel(i - 1, j, k, 1)) * 0.5 * c.inv_dx;
        double dudy = (vel(i, j + 1, k, 0) - vel(i, j - 1, k, 0)) * 0.5 * c.inv_dy;
        double wx = dwdy - dvdz, wy = dudz - dwdx, wz = dvdx - dudy;
        v[6] = 0.5 * u[0] * (wx * wx + wy * wy + wz * wz) * dV;
        v[7] = bad ? 1.0 : 0.0;
    }
    __shared__ double red[8][4];
    int warp = threadIdx.y;  // blockDim = (32,4): one warp per row
#pragma unroll
    for (int m = 0; m < 8; m++) {
        double x = v[m];
        for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
        if (threadIdx.x == 0) red[m][warp] = x;
    }
    __syncthreads();
    if (threadIdx.y == 0 && threadIdx.x < 8) {
        int m = threadIdx.x;
        atomicAdd(&acc[m], red[m][0] + red[m][1] + red[m][2] + red[m][3]);
    }
}

// ---------------------------------------------------------------------------
// state check (no reference counterpart: the reference lets NaN propagate,
// src/time_scheme.cpp:104-117): counts the interior cells whose values are not
// all finite or whose density or pressure is not positive.  PRIM: A is W
// (pressure read directly), else A is U (pressure from the equation of state).
template <bool PRIM>
__global__ void __launch_bounds__(128) k_check_state(const double* __restrict__ A, Box b, Consts c,
                                                     unsigned long long* __restrict__ count) {
    const int k = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 4 + threadIdx.y, i = blockIdx.z;
    bool bad = false;
    if (k < b.nz && j < b.ny) {
        const long long o = b.at(i + NG, j + NG, k + NG);
        double v[5];
        bool fin = true;
#pragma unroll
        for (int q = 0; q < 5; q++) {
            v[q] = A[q * b.fstride + o];
            fin &= isfinite(v[q]);
        }
        double pr = v[1];
        if (!PRIM) {
            double w[5];
            prim_from_cons(v, c.gm1, w);
            pr = w[1];
        }
        bad = !fin || !(v[0] > 0.0) || !(pr > 0.0);
    }
    const unsigned m = __ballot_sync(0xffffffffu, bad);
    if (threadIdx.x == 0 && m) atomicAdd(count, (unsigned long long)__popc(m));
}

// ---------------------------------------------------------------------------
// host launchers

static dim3 cell_grid(const Box& b, const Planes& pl = Planes()) {  // all halo'd cells (of planes pl)
    return dim3((b.nz + 2 * NG + 31) / 32, (b.NY + 3) / 4, pl.n < 0 ? b.NX : pl.n);
}
static dim3 interior_grid(const Box& b) {
    return dim3((b.nz + 31) / 32, (b.ny + 3) / 4, b.nx);
}

void launch_step_begin(bool from_u, bool phys, double* W, double* U, double* U0, const Box& b,
                       const Consts& c, unsigned long long* slot, cudaStream_t s, Planes pl) {
    const dim3 blk(32, 4), g = cell_grid(b, pl);
    if (from_u) {
        if (phys) k_step_begin<true, true><<<g, blk, 0, s>>>(W, U, U0, b, c, slot, pl.lo);
        else k_step_begin<true, false><<<g, blk, 0, s>>>(W, U, U0, b, c, slot, pl.lo);
    } else {
        if (phys) k_step_begin<false, true><<<g, blk, 0, s>>>(W, U, U0, b, c, slot, pl.lo);
        else k_step_begin<false, false><<<g, blk, 0, s>>>(W, U, U0, b, c, slot, pl.lo);
    }
}

void launch_prim_all(double* W, const double* U, const Box& b, const Consts& c, cudaStream_t s, Planes pl) {
    k_prim_all<<<cell_grid(b, pl), dim3(32, 4), 0, s>>>(W, U, b, c, pl.lo);
}

void launch_cons_all(const double* W, double* U, const Box& b, const Consts& c, cudaStream_t s) {
    k_cons_all<<<cell_grid(b), dim3(32, 4), 0, s>>>(W, U, b, c);
}

void launch_min_dt(bool phys, const double* W, const Box& b, const Consts& c, unsigned long long* slot,
                   cudaStream_t s) {
    if (phys) k_min_dt<true><<<interior_grid(b), dim3(32, 4), 0, s>>>(W, b, c, slot);
    else k_min_dt<false><<<interior_grid(b), dim3(32, 4), 0, s>>>(W, b, c, slot);
}

void launch_fill_prim(double* W, double* U, const Box& b, const Consts& c, cudaStream_t s) {
    k_fill_prim<<<cell_grid(b), dim3(32, 4), 0, s>>>(W, U, b, c);
}

void launch_fill_w(bool phys, double* W, const double* U, const Box& b, const Consts& c, cudaStream_t s, Planes pl) {
    const dim3 g = cell_grid(b, pl), blk(32, 4);
    if (phys) k_fill_w<true, false><<<g, blk, 0, s>>>(W, U, b, c, pl.lo);
    else k_fill_w<false, false><<<g, blk, 0, s>>>(W, U, b, c, pl.lo);
}

void launch_fill_shell(bool phys, double* W, const double* U, const Box& b, const Consts& c, cudaStream_t s) {
    const long long NZ = b.nz + 2 * NG;
    const long long n = 2 * NG * std::max(std::max(b.NY * NZ, b.nx * NZ), (long long)b.nx * b.ny);
    const dim3 g((unsigned)((n + 127) / 128), 3);
    if (phys) k_fill_w<true, true><<<g, 128, 0, s>>>(W, U, b, c, 0);
    else k_fill_w<false, true><<<g, 128, 0, s>>>(W, U, b, c, 0);
}

void launch_fill_uhalo(double* U, const double* Us, const Box& b, const Consts& c, cudaStream_t s) {
    const long long nxe = b.nx + (c.ext_x ? 2 * NG : 0);  // slabs: y/z ghost rows of the x ghost planes too
    const long long area = std::max(std::max((long long)b.ny * b.nz, nxe * b.nz), nxe * b.ny);
    k_fill_uhalo<<<dim3((unsigned)((3 * area + 127) / 128), 6), 128, 0, s>>>(U, Us, b, c);
}

template <int DIR, bool CHAR, bool BORGES, bool PHYS>
static void face_one(const double* W, const double* U, const Box& b, const Consts& c, void* F,
                     const FaceBox& fb, cudaStream_t s) {
    const dim3 grid((fb.n2 - (DIR == 2) + 31) / 32, (fb.n1 - (DIR == 1) + 3) / 4, fb.n0);
    k_face_flux<DIR, CHAR, BORGES, PHYS><<<grid, dim3(32, 4), 0, s>>>(W, U, b, c, (float*)F, fb);
    if constexpr (DIR > 0) {
        const dim3 tail(((DIR == 1 ? fb.n2 : fb.n1) + 127) / 128, fb.n0);
        k_face_flux_tail<DIR, CHAR, BORGES, PHYS><<<tail, 128, 0, s>>>(W, U, b, c, (float*)F, fb);
    }
}

template <bool CHAR, bool BORGES, bool PHYS>
static int faces_one(bool fp32, int dims, const double* W, const double* U, const Box& b, const Consts& c, void* const F[3],
                     const FaceBox fb[3], cudaStream_t s) {
    if (fp32) {
        face_one<0, CHAR, BORGES, PHYS>(W, U, b, c, F[0], fb[0], s);
        face_one<1, CHAR, BORGES, PHYS>(W, U, b, c, F[1], fb[1], s);
        if (dims == 3) face_one<2, CHAR, BORGES, PHYS>(W, U, b, c, F[2], fb[2], s);
        return dims == 3 ? 5 : 3;
    }
    OpFaces o;
    unsigned blocks = 0;
    for (int d = 0; d < 3; d++) {
        o.F[d] = (double*)F[d];
        o.fb[d] = fb[d];
        o.blocks[d] = d < dims ? (unsigned)(((long long)fb[d].n0 * fb[d].n1 * fb[d].n2 + 127) / 128) : 0;
        blocks += o.blocks[d];
    }
    k_op_faces<CHAR, BORGES, PHYS><<<blocks, 128, 0, s>>>(W, U, b, c, o);
    return 1;
}

int launch_faces(bool chr, bool borges, bool phys, bool fp32, int dims, const double* W, const double* U, const Box& b,
                 const Consts& c, void* const F[3], const FaceBox fb[3], cudaStream_t s) {
    if (chr) {
        if (borges) return phys ? faces_one<true, true, true>(fp32, dims, W, U, b, c, F, fb, s)
                                : faces_one<true, true, false>(fp32, dims, W, U, b, c, F, fb, s);
        return phys ? faces_one<true, false, true>(fp32, dims, W, U, b, c, F, fb, s)
                    : faces_one<true, false, false>(fp32, dims, W, U, b, c, F, fb, s);
    }
    if (borges) return phys ? faces_one<false, true, true>(fp32, dims, W, U, b, c, F, fb, s)
                            : faces_one<false, true, false>(fp32, dims, W, U, b, c, F, fb, s);
    return phys ? faces_one<false, false, true>(fp32, dims, W, U, b, c, F, fb, s)
                : faces_one<false, false, false>(fp32, dims, W, U, b, c, F, fb, s);
}

template <int MODE, int H, bool PHYS, typename TF, typename TV>
static void update_one(const UpdateArgs& a, cudaStream_t s) {
    k_update<MODE, H, PHYS, TF, TV><<<interior_grid(a.b), dim3(32, 4), 0, s>>>(
        a.W, a.U, a.U0, (const TF*)a.F[0], (const TF*)a.F[1], (const TF*)a.F[2], a.b, a.fb[0],
        a.fb[1], a.fb[2], a.c, a.flags, a.slot, a.m1, a.m2, a.mc, a.Rout, a.clock);
}

template <int MODE, bool PHYS, typename TF, typename TV>
static void update_h(int h, const UpdateArgs& a, cudaStream_t s) {
    switch (h) {
        case 0: update_one<MODE, 0, PHYS, TF, TV>(a, s); break;
        case 1: update_one<MODE, 1, PHYS, TF, TV>(a, s); break;
        case 2: update_one<MODE, 2, PHYS, TF, TV>(a, s); break;
        default: update_one<MODE, 3, PHYS, TF, TV>(a, s); break;
    }
}

template <int MODE, typename T>
static void update_mode(const UpdateArgs& a, cudaStream_t s) {
    int h = a.viscous ? a.c.order / 2 : 0;
    if (a.phys) update_h<MODE, true, T, T>(h, a, s);
    else update_h<MODE, false, T, T>(h, a, s);
}

void launch_update(const UpdateArgs& a, cudaStream_t s) {
    if (a.mode == MODE_STAGE) update_mode<MODE_STAGE, double>(a, s);  // FP32 steps are fused (ns_fused.cuh)
    else if (a.fp32) update_mode<MODE_RHS, float>(a, s);
    else update_mode<MODE_RHS, double>(a, s);
}

void launch_check_state(const double* A, bool prim, const Box& b, const Consts& c,
                        unsigned long long* count, cudaStream_t s) {
    if (prim) k_check_state<true><<<interior_grid(b), dim3(32, 4), 0, s>>>(A, b, c, count);
    else k_check_state<false><<<interior_grid(b), dim3(32, 4), 0, s>>>(A, b, c, count);
}

void launch_slab_pack(const double* U, const Box& b, int side, double* buf, cudaStream_t s) {
    const long long n = 15LL * b.ny * b.nz;
    k_slab_pack<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(U, b, side, buf);
}
void launch_slab_unpack(double* U, const Box& b, int side, const double* buf, cudaStream_t s) {
    const long long n = 15LL * b.ny * b.nz;
    k_slab_unpack<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(U, b, side, buf);
}

void launch_aos_to_soa(const double* A, double* S, const Box& b, cudaStream_t s, Planes pl) {
    k_aos_to_soa<<<cell_grid(b, pl), dim3(32, 4), 0, s>>>(A, S, b, pl.lo);
}
void launch_soa_to_aos(const double* S, double* A, const Box& b, cudaStream_t s, Planes pl) {
    k_soa_to_aos<<<cell_grid(b, pl), dim3(32, 4), 0, s>>>(S, A, b, pl.lo);
}
void launch_diagnostics(const double* U, const Box& b, const Consts& c, double* acc, cudaStream_t s) {
    k_diagnostics<<<interior_grid(b), dim3(32, 4), 0, s>>>(U, b, c, acc);
}

// The bounded wait of the tensor-core kernels, on a phase that no
// arrival or transaction completes: it must give up after `polls` polls.
__global__ void k_wait_probe(unsigned polls, unsigned long long* __restrict__ out) {
    __shared__ __align__(8) unsigned long long bar;
    if (threadIdx.x == 0) tc::mbar_init(tc::smem_u32(&bar), 1);
    __syncthreads();
    const bool done = tc::mbar_wait(tc::smem_u32(&bar), 0, polls);
    if (__syncthreads_or(done)) {
        if (threadIdx.x == 0) out[0] = 0;
    } else if (threadIdx.x == 0) {
        out[0] = 1;
    }
}

cudaError_t launch_wait_probe(unsigned polls, unsigned long long* out, cudaStream_t s) {
    k_wait_probe<<<1, 32, 0, s>>>(polls, out);
    return cudaGetLastError();
}

}  // namespace nsb

// ---------------------------------------------------------------------------
// FMA throughput probe: the measured denominator of the compute roofline.
// Every thread runs 8 independent FMA chains (enough to cover the pipe's
// latency); the result is written only if it is NaN so the work is kept.
namespace nsb {
template <typename T>
__global__ void __launch_bounds__(256) k_fma_probe(int iters, T seed, T* sink) {
    T a[8];
#pragma unroll
    for (int c = 0; c < 8; c++) a[c] = seed + T(threadIdx.x + c);
    const T m = T(0.999999), k = T(1e-7);
    for (int it = 0; it < iters; it++) {
#pragma unroll
        for (int c = 0; c < 8; c++) a[c] = a[c] * m + k;
    }
    T s = a[0] + a[1] + a[2] + a[3] + a[4] + a[5] + a[6] + a[7];
    if (s != s) *sink = s;
}

cudaError_t launch_fma_probe(bool fp64, int blocks, int iters, void* sink, cudaStream_t s) {
    if (fp64)
        k_fma_probe<double><<<blocks, 256, 0, s>>>(iters, 1.0, (double*)sink);
    else
        k_fma_probe<float><<<blocks, 256, 0, s>>>(iters, 1.0f, (float*)sink);
    return cudaGetLastError();
}
}  // namespace nsb
