// ns_viscous64.cu -- the centered viscous terms of an FP64 time step's stage
// (CenteredDiffusion::compute_residual, src/diffusion_schemes/centered_diffusion.cpp:70-182,
// or the full 3D terms of the physical semantics), residual components 1..4 into V.
//
// A thread marches a column (j, k) along x.  The stencils are tensor products, so
// every derivative with an x in it is an x-difference of something that belongs to
// one plane: the plane's own values and its derivatives along y and z.  Those are
// formed once per plane, as it comes into reach, and kept by the thread; a cell then
// reads no neighbour outside its plane.  (Taken literally the mixed derivatives are six
// products of 2H x 2H neighbours.)  W's ghost cells are folded along every axis, edges
// and corners too, so no cell is a special case.
//
// CD-4 and CD-6 (k_viscous) keep the planes in a private ring in shared memory and
// read neighbours from global memory.  CD-2 keeps them in registers and reads each
// plane's neighbours once, from tiles that the TMA unit loads four planes ahead
// (k_viscous_cd2_tma): the loads' latency is the bound otherwise, at 128 registers a
// thread.  Tiles are 32 cells wide, so rows of less than 16 cells go without
// (k_viscous_cd2).  ms per step before -> now (both with TMA tiles / without):
//   CD-2, physical, 384^3: 3.73 -> 2.50 / 4.67      256x256x17: 0.123 / 0.134, x8: 0.123 / 0.074
//   CD-2, reference, 256^3: 1.00 -> 0.58 / 0.79     256x256x8: 0.094 / 0.044, 512x512x1: 0.301 / 0.086
//   CD-6, physical, 101x75x130: 0.80 -> 0.25 (cells near an edge had read 250 neighbours each)
// Marching along y instead of x, or loading the next plane's rows ahead into registers,
// measured the same or slower.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "ns_common.cuh"
#include "ns_eos.cuh"
#include "ns_kernels.h"
#include "ns_tcgen05.cuh"
#include "ns_tma.cuh"
#include "ns_viscous.cuh"

namespace nsb {

template <int H, bool PHYS>
struct ViscRing {
    // physical: T, u, v, w, dv/dy + dw/dz, du/dy, du/dz; reference: rho, p, u, v,
    // d(u, v)/dy and d(u, v)/dy of the rows inside
    static constexpr int NR = PHYS ? 7 : 8, NS = 2 * H + 1;
    static constexpr size_t bytes = (size_t)NS * NR * 128 * 8;
    static constexpr int MINB = H == 2 ? 4 : 3;
    // a warp's dv/dy and dw/dy of one plane, each of its at most two runs of columns with
    // H columns on both sides
    static constexpr int RUN = 32 + 4 * H;
    static constexpr size_t shared_bytes = (size_t)4 * 2 * RUN * 8;
};

// centered first and second difference of f(-H) .. f(H), undivided
template <int H, typename Fn>
__device__ __forceinline__ double diff1(Fn f, const Consts& c) {
    double s = c.df[4] * (f(1) - f(-1));
#pragma unroll
    for (int h = 2; h <= H; h++) s = fma(c.df[3 + h], f(h) - f(-h), s);
    return s;
}
// the coefficients sum to zero, so the centre enters through the differences to it
template <int H, typename Fn>
__device__ __forceinline__ double diff2(Fn f, const Consts& c) {
    const double f0 = f(0);
    double s = c.ddf[4] * fma(-2.0, f0, f(1) + f(-1));
#pragma unroll
    for (int h = 2; h <= H; h++) s = fma(c.ddf[3 + h], fma(-2.0, f0, f(h) + f(-h)), s);
    return s;
}

// Physical semantics: the terms of a cell from the velocity gradient gu[a][b] =
// du_a/dx_b, the Laplacians of the velocity and of T, d(div u)/dx_a and the velocity
__device__ __forceinline__ void viscous_physical_terms(const double gu[3][3], const double lap[3], const double gdiv[3],
                                                       double lapT, const double vel[3], const Consts& c,
                                                       double* __restrict__ v, long long vs) {
    const double div = gu[0][0] + gu[1][1] + gu[2][2];
    double work = c.heat * c.mu * lapT, mom[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        mom[a] = c.mu * lap[a] + (c.mu + c.lamb) * gdiv[a];
        work += vel[a] * mom[a];
    }
    // dissipation tau_ab du_a/dx_b with tau_ab = mu (du_a/dx_b + du_b/dx_a) + lamb div delta_ab
    double sq = 2.0 * (gu[0][0] * gu[0][0] + gu[1][1] * gu[1][1] + gu[2][2] * gu[2][2]);
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const double g = gu[a][(a + 1) % 3] + gu[(a + 1) % 3][a];
        sq = fma(g, g, sq);
    }
    work += c.mu * sq + c.lamb * div * div;
    v[0] = -work;
#pragma unroll
    for (int a = 0; a < 3; a++) v[(1 + a) * vs] = -mom[a];
}

// SHARE (physical semantics, 3D, nz >= 32): the lanes of a warp run along z, at most once
// around the end of their rows, so d2/dydz of v and w is taken from the lanes' own d/dy of
// the plane (shared memory) and 4H columns of it at the runs' ends, which the lanes form
// besides: 12 reads of shared memory and 6 loads instead of 72 loads for CD-6, half of a
// cell's, and loads are what bounds this kernel.  ms per step without -> with: CD-6
// 101x75x130 0.301 -> 0.246, 128x128x40 0.192 -> 0.164, 384^3 12.2 -> 10.3; CD-4 0.195 ->
// 0.182, 384^3 7.78 -> 7.19.  In rows of less than 32 cells a warp has more ends than its
// lanes can serve, and each lane takes the products.
template <int H, bool PHYS, bool SHARE>
__global__ void __launch_bounds__(128, ViscRing<H, PHYS>::MINB)
    k_viscous(const double* __restrict__ W, Box b, Consts c, double* __restrict__ V, long long vs, int xlo, int xhi,
              int lx) {
    using VR = ViscRing<H, PHYS>;
    extern __shared__ double vsm[];
    const int t = threadIdx.y * 32 + threadIdx.x;
    int j, k;
    const bool mine = row_tile(b, j, k);
    if (SHARE ? !__any_sync(~0u, mine) : !mine) return;  // a lane without a column goes along in row 0
    const int x0 = xlo + blockIdx.y * lx, x1 = min(x0 + lx, xhi);
    double* ring = vsm + t;  // [NS][NR][128]
    const long long xs = (long long)b.NY * b.NZp;
    // SHARE: where this lane's d/dy goes, and the column at an end that it forms besides
    double* run = nullptr;
    double* end = nullptr;
    const double* we = nullptr;
    if constexpr (SHARE) {
        double* warp = vsm + VR::NS * VR::NR * 128 + threadIdx.y * 2 * VR::RUN;
        const int l = threadIdx.x, k0 = __shfl_sync(~0u, k, 0), j0 = __shfl_sync(~0u, j, 0);
        const int m = min(32, b.nz - k0);  // lanes of the first run
        run = warp + H + l + (l < m ? 0 : 2 * H);
        const int f = l / (4 * H), e = l % (4 * H), side = e / H, h = e % H;  // v or w; the runs' ends in turn
        // (the first lane's column exists where any does: rows rise with the lanes)
        const int je = side < 2 ? j0 : j0 + 4;
        const int ke = side == 0 ? k0 - H + h : side == 1 ? k0 + m + h : side == 2 ? h - H : 32 - m + h;
        if (f < 2 && (side < 2 || (m < 32 && je < b.ny))) {
            end = warp + f * VR::RUN + (side == 0 ? h : side == 1 ? H + m + h : side == 2 ? 2 * H + m + h : 3 * H + 32 + h);
            we = W + (3 + f) * b.fstride + b.at(x0 + NG, je + NG, ke + NG);
        }
    }
    const double* w = W + b.at(x0 - H + NG, j + NG, k + NG);
    double* v = V + ((long long)x0 * b.ny + j) * b.nz + k;
    const bool three = c.dim == 3;
    for (int p = x0 - H; p < x1 + H; p++) {
        // plane p into the ring
        double* e = ring + ((p - x0 + H) % VR::NS) * VR::NR * 128;
        {
            auto y = [&](int q) { return diff1<H>([&](int h) { return w[q * b.fstride + h * b.NZp]; }, c) * c.inv_dy; };
            auto z = [&](int q) { return diff1<H>([&](int h) { return w[q * b.fstride + h]; }, c) * c.inv_dz; };
            if constexpr (PHYS) {
                e[0] = w[5 * b.fstride];
#pragma unroll
                for (int a = 0; a < 3; a++) e[(1 + a) * 128] = w[(2 + a) * b.fstride];
                e[4 * 128] = three ? y(3) + z(4) : y(3);
                e[5 * 128] = y(2);
                e[6 * 128] = three ? z(2) : 0.0;
            } else {
                // first derivatives are zero outside the domain along an axis that is not
                // periodic (derivative halos are only filled by the periodic exchange,
                // centered_diffusion.cpp:22-24): dW/dy of an outside plane, and the rows that
                // d/dy of dW/dx reaches
#pragma unroll
                for (int q = 0; q < 4; q++) e[q * 128] = w[q * b.fstride];
                const bool in = x_inside(p, b.nx, c);
#pragma unroll
                for (int q = 2; q < 4; q++) {
                    const double d = y(q);
                    e[(2 + q) * 128] = in ? d : 0.0;
                    double m = d;
                    if (!c.periodic[1] && (j < H || j >= b.ny - H)) {
                        m = 0.0;
#pragma unroll
                        for (int h = -H; h <= H; h++)
                            if (h != 0 && j + h >= 0 && j + h < b.ny) m = fma(c.df[3 + h], w[q * b.fstride + h * b.NZp], m);
                        m *= c.inv_dy;
                    }
                    e[(4 + q) * 128] = m;
                }
            }
        }
        w += xs;
        if (p < x0 + H) continue;
        const int i = p - H;
        const double* wi = w - (H + 1) * xs;  // plane i
        // quantity r of plane i + h
        auto X = [&](int r, int h) { return ring[((i + h - x0 + H) % VR::NS) * VR::NR * 128 + r * 128]; };
        auto dx = [&](int r) { return diff1<H>([&](int h) { return X(r, h); }, c) * c.inv_dx; };
        auto Y = [&](int q, int h) { return wi[q * b.fstride + h * b.NZp]; };
        if constexpr (PHYS) {
            const double ix2 = c.inv_dx * c.inv_dx, iy2 = c.inv_dy * c.inv_dy, iz2 = c.inv_dz * c.inv_dz;
            auto Z = [&](int q, int h) { return wi[q * b.fstride + h]; };
            auto dxx = [&](int r) { return diff2<H>([&](int h) { return X(r, h); }, c) * ix2; };
            auto dyy = [&](int q) { return diff2<H>([&](int h) { return Y(q, h); }, c) * iy2; };
            auto dzz = [&](int q) { return diff2<H>([&](int h) { return Z(q, h); }, c) * iz2; };
            auto dyz = [&](int q) {
                return diff1<H>([&](int h) {
                           return diff1<H>([&](int g) { return wi[q * b.fstride + h * b.NZp + g]; }, c);
                       }, c) * (c.inv_dy * c.inv_dz);
            };
            // gradient of u along each axis, Laplacians, d(div u)/dx_a
            double gu[3][3], lap[3], gdiv[3], lapT = dxx(0) + dyy(5);
            if (three) lapT += dzz(5);
            const double uxx = dxx(1), vyy = dyy(3);
            gu[0][0] = dx(1);
            gu[1][0] = dx(2);
            gu[2][0] = dx(3);
            gu[0][1] = X(5, 0);
            const double v_y = diff1<H>([&](int h) { return Y(3, h); }, c), w_y = diff1<H>([&](int h) { return Y(4, h); }, c);
            gu[1][1] = v_y * c.inv_dy;
            gu[2][1] = w_y * c.inv_dy;
            gu[0][2] = gu[1][2] = gu[2][2] = 0.0;
            lap[0] = uxx + dyy(2);
            lap[1] = dxx(2) + vyy;
            lap[2] = dxx(3) + dyy(4);
            gdiv[0] = uxx + dx(4);
            gdiv[1] = vyy + dx(5);
            gdiv[2] = 0.0;
            if (three) {
                const double wzz = dzz(4);
                gu[0][2] = X(6, 0);
                gu[1][2] = diff1<H>([&](int h) { return Z(3, h); }, c) * c.inv_dz;
                gu[2][2] = diff1<H>([&](int h) { return Z(4, h); }, c) * c.inv_dz;
                lap[0] += dzz(2);
                lap[1] += dzz(3);
                lap[2] += wzz;
                if constexpr (SHARE) {
                    run[0] = v_y;
                    run[VR::RUN] = w_y;
                    if (end) *end = diff1<H>([&](int h) { return we[h * b.NZp]; }, c);
                    __syncwarp();
                    const double s = c.inv_dy * c.inv_dz;
                    gdiv[1] += diff1<H>([&](int h) { return run[VR::RUN + h]; }, c) * s;
                    gdiv[2] = wzz + dx(6) + diff1<H>([&](int h) { return run[h]; }, c) * s;
                    __syncwarp();
                    if (end) we += xs;
                } else {
                    gdiv[1] += dyz(4);
                    gdiv[2] = wzz + dx(6) + dyz(3);
                }
            }
            const double vel[3] = {X(1, 0), X(2, 0), X(3, 0)};
            if (!SHARE || mine) viscous_physical_terms(gu, lap, gdiv, lapT, vel, c, v, vs);
        } else {
            double Dx[4], Dy[4], Dxx[4], Dyy[4], Dxy[2], Dyx[2], r[5] = {0, 0, 0, 0, 0};
            const double ix2 = c.inv_dx * c.inv_dx, iy2 = c.inv_dy * c.inv_dy;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                Dx[q] = dx(q);
                Dy[q] = diff1<H>([&](int h) { return Y(q, h); }, c) * c.inv_dy;
                const double d = diff2<H>([&](int h) { return X(q, h); }, c);
                Dxx[q] = d * ix2;
                Dyy[q] = d * iy2;  // d2/dy2 takes the x-stencil (cd-n.cpp:77)
            }
#pragma unroll
            for (int a = 0; a < 2; a++) {
                Dyx[a] = dx(4 + a);
                Dxy[a] = dx(6 + a);
            }
            viscous_reference_terms<double>(Dx, Dy, Dxx, Dyy, Dxy, Dyx, X(2, 0), X(3, 0), X(1, 0), X(0, 0), c, r);
#pragma unroll
            for (int q = 1; q < 5; q++) v[(q - 1) * vs] = r[q];
        }
        v += (long long)b.ny * b.nz;
    }
}

// CD-2, physical semantics: the march of a column with the ring in registers (three
// planes, moved on by one a cell); each plane's neighbours are read once, when the
// plane enters.
struct ViscCd2 {
    // of planes i-1, i, i+1: T, u, v, w, dv/dy + dw/dz, du/dy, du/dz
    double Q[3][7];
    // of plane i+1, then of plane i: dv/dy, dw/dy, dv/dz, dw/dz, the y- and z-parts of the
    // Laplacians of T, u, v, w, d2v/dy2, d2w/dz2, d2v/dydz, d2w/dydz
    double N[12], C[12];
    double hx, hy, hz, ix2, iy2, iz2;
    bool three;

    __device__ __forceinline__ ViscCd2(const Consts& c, const Box&, int) {
        three = c.dim == 3;
        hx = 0.5 * c.inv_dx;
        hy = 0.5 * c.inv_dy;
        hz = three ? 0.5 * c.inv_dz : 0.0;
        ix2 = c.inv_dx * c.inv_dx;
        iy2 = c.inv_dy * c.inv_dy;
        iz2 = three ? c.inv_dz * c.inv_dz : 0.0;
#pragma unroll
        for (int q = 0; q < 12; q++) N[q] = 0.0;
#pragma unroll
        for (int h = 0; h < 3; h++)
#pragma unroll
            for (int q = 0; q < 7; q++) Q[h][q] = 0.0;
    }
    // the next plane: at(f, y, z) is field f of u, v, w, T beside the column in it
    template <typename At>
    __device__ __forceinline__ void enter(At at, bool) {
#pragma unroll
        for (int q = 0; q < 7; q++) {
            Q[0][q] = Q[1][q];
            Q[1][q] = Q[2][q];
        }
#pragma unroll
        for (int q = 0; q < 12; q++) C[q] = N[q];
        Q[2][0] = at(3, 0, 0);
        N[4] = iy2 * fma(-2.0, Q[2][0], at(3, 1, 0) + at(3, -1, 0));
        if (three) N[4] = fma(iz2, fma(-2.0, Q[2][0], at(3, 0, 1) + at(3, 0, -1)), N[4]);
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const double f = at(a, 0, 0), yp = at(a, 1, 0), ym = at(a, -1, 0);
            Q[2][1 + a] = f;
            const double d = hy * (yp - ym), e = iy2 * fma(-2.0, f, yp + ym);
            double dz = 0.0, ez = 0.0;
            if (three) {
                const double zp = at(a, 0, 1), zm = at(a, 0, -1);
                dz = hz * (zp - zm);
                ez = iz2 * fma(-2.0, f, zp + zm);
                if (a > 0) N[9 + a] = (hy * hz) * ((at(a, 1, 1) - at(a, 1, -1)) - (at(a, -1, 1) - at(a, -1, -1)));
            }
            N[5 + a] = e + ez;
            if (a == 0) {
                Q[2][5] = d;
                Q[2][6] = dz;
            } else {
                N[a - 1] = d;   // dv/dy, dw/dy
                N[1 + a] = dz;  // dv/dz, dw/dz
                if (a == 1) N[8] = e;
                else N[9] = ez;
            }
        }
        Q[2][4] = N[0] + N[3];
    }
    // the terms of the middle plane's cell
    __device__ __forceinline__ void cell(const Consts& c, double* __restrict__ v, long long vs) const {
        double gu[3][3], lap[3], gdiv[3], xx[4];
#pragma unroll
        for (int q = 0; q < 4; q++) xx[q] = ix2 * fma(-2.0, Q[1][q], Q[2][q] + Q[0][q]);
#pragma unroll
        for (int a = 0; a < 3; a++) {
            gu[a][0] = hx * (Q[2][1 + a] - Q[0][1 + a]);
            lap[a] = xx[1 + a] + C[5 + a];
        }
        gu[0][1] = Q[1][5];
        gu[0][2] = Q[1][6];
        gu[1][1] = C[0];
        gu[2][1] = C[1];
        gu[1][2] = C[2];
        gu[2][2] = C[3];
        gdiv[0] = fma(hx, Q[2][4] - Q[0][4], xx[1]);
        gdiv[1] = C[8] + fma(hx, Q[2][5] - Q[0][5], C[11]);
        gdiv[2] = C[9] + fma(hx, Q[2][6] - Q[0][6], C[10]);
        viscous_physical_terms(gu, lap, gdiv, xx[0] + C[4], &Q[1][1], c, v, vs);
    }
};

// the same for the reference semantics
struct ViscCd2Ref {
    // of planes i-1, i, i+1: rho, p, u, v; d(u, v)/dy where the plane lies inside; d(u, v)/dy
    // of the rows inside (k_viscous)
    double Q[3][8];
    double N[4], C[4];  // d(rho, p, u, v)/dy of planes i+1 and i
    double hx, hy, ix2, iy2;
    bool lo, hi;        // the row below or above lies outside and does not count

    __device__ __forceinline__ ViscCd2Ref(const Consts& c, const Box& b, int j) {
        hx = 0.5 * c.inv_dx;
        hy = 0.5 * c.inv_dy;
        ix2 = c.inv_dx * c.inv_dx;
        iy2 = c.inv_dy * c.inv_dy;
        lo = j == 0 && !c.periodic[1];
        hi = j == b.ny - 1 && !c.periodic[1];
#pragma unroll
        for (int q = 0; q < 4; q++) N[q] = 0.0;
#pragma unroll
        for (int h = 0; h < 3; h++)
#pragma unroll
            for (int q = 0; q < 8; q++) Q[h][q] = 0.0;
    }
    // the next plane: at(f, y, z) is field f of rho, p, u, v; inside: whether it lies inside
    template <typename At>
    __device__ __forceinline__ void enter(At at, bool inside) {
#pragma unroll
        for (int q = 0; q < 8; q++) {
            Q[0][q] = Q[1][q];
            Q[1][q] = Q[2][q];
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
            C[q] = N[q];
            Q[2][q] = at(q, 0, 0);
            const double yp = at(q, 1, 0), ym = at(q, -1, 0);
            N[q] = hy * (yp - ym);
            if (q >= 2) {
                Q[2][2 + q] = inside ? N[q] : 0.0;
                Q[2][4 + q] = hy * ((hi ? 0.0 : yp) - (lo ? 0.0 : ym));
            }
        }
    }
    __device__ __forceinline__ void cell(const Consts& c, double* __restrict__ v, long long vs) const {
        double Dx[4], Dxx[4], Dyy[4], Dxy[2], Dyx[2], r[5] = {0, 0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < 4; q++) {
            Dx[q] = hx * (Q[2][q] - Q[0][q]);
            const double d = fma(-2.0, Q[1][q], Q[2][q] + Q[0][q]);
            Dxx[q] = d * ix2;
            Dyy[q] = d * iy2;  // d2/dy2 takes the x-stencil (cd-n.cpp:77)
        }
#pragma unroll
        for (int a = 0; a < 2; a++) {
            Dyx[a] = hx * (Q[2][4 + a] - Q[0][4 + a]);
            Dxy[a] = hx * (Q[2][6 + a] - Q[0][6 + a]);
        }
        viscous_reference_terms<double>(Dx, C, Dxx, Dyy, Dxy, Dyx, Q[1][2], Q[1][3], Q[1][1], Q[1][0], c, r);
#pragma unroll
        for (int q = 1; q < 5; q++) v[(q - 1) * vs] = r[q];
    }
};

template <bool PHYS>
struct Cd2;
template <>
struct Cd2<true> {
    using March = ViscCd2;
    static constexpr int F0 = 2;  // plane of its first field
};
template <>
struct Cd2<false> {
    using March = ViscCd2Ref;
    static constexpr int F0 = 0;
};

// straight from global memory
template <bool PHYS>
__global__ void __launch_bounds__(128, 5)
    k_viscous_cd2(const double* __restrict__ W, Box b, Consts c, double* __restrict__ V, long long vs, int xlo, int xhi,
                  int lx) {
    int j, k;
    if (!row_tile(b, j, k)) return;
    const int x0 = xlo + blockIdx.y * lx, x1 = min(x0 + lx, xhi);
    const double* w = W + b.at(x0 - 1 + NG, j + NG, k + NG) + Cd2<PHYS>::F0 * b.fstride;
    double* v = V + ((long long)x0 * b.ny + j) * b.nz + k;
    typename Cd2<PHYS>::March m(c, b, j);
    for (int p = x0 - 1; p <= x1; p++) {
        m.enter([&](int f, int y, int z) { return w[f * b.fstride + y * b.NZp + z]; }, x_inside(p, b.nx, c));
        w += (long long)b.NY * b.NZp;
        if (p <= x0) continue;  // the first cell's own plane
        m.cell(c, v, vs);
        v += (long long)b.ny * b.nz;
    }
}

// through a ring of tiles that the TMA unit fills: a block owns 4 rows x 32 columns, and
// a plane's box is four fields of rows j0-1 .. j0+4 and columns k0-1 .. k0+32
struct ViscTile {
    static constexpr int BZ = 34, BY = 6, ELEMS = 4 * BY * BZ;
    static constexpr int STRIDE = (ELEMS + 15) / 16 * 16;  // 128-byte aligned slots
    static constexpr int NS = 4;
    static constexpr size_t smem = (size_t)NS * STRIDE * 8 + NS * 8;
    static constexpr int MINB = 3;
};
template <bool PHYS>
__global__ void __launch_bounds__(128, ViscTile::MINB)
    k_viscous_cd2_tma(const __grid_constant__ CUtensorMap map, Box b, Consts c, double* __restrict__ V, long long vs,
                      unsigned long long* __restrict__ err, int xlo, int xhi, int lx) {
    using VT = ViscTile;
    extern __shared__ __align__(128) double vsm[];  // [NS][4][BY][BZ], then NS mbarriers
    unsigned long long* full = reinterpret_cast<unsigned long long*>(vsm + VT::NS * VT::STRIDE);
    const int lane = threadIdx.x, ty = threadIdx.y, t = ty * 32 + lane;
    if (tc::smem_u32(vsm) & 127u) {  // a TMA destination must be 128-byte aligned: report, touch nothing
        if (t == 0) atomicOr(err, 2ull);
        return;
    }
    const int k0 = blockIdx.x * 32, j0 = blockIdx.y * 4, x0 = xlo + blockIdx.z * lx, x1 = min(x0 + lx, xhi);
    const int k = k0 + lane, j = j0 + ty;
    const bool live = k < b.nz && j < b.ny;
    // plane p (x0 - 1 <= p <= x1) is the (p - x0 + 1)-th load of the block
    auto slot = [&](int p) { return (p - x0 + 1) % VT::NS; };
    auto bar = [&](int p) { return tc::smem_u32(&full[slot(p)]); };
    auto issue = [&](int p) {
        mbar_expect_tx(bar(p), VT::ELEMS * 8);
        tma_load_4d(tc::smem_u32(vsm + slot(p) * VT::STRIDE), &map, k0 + 2, j0 + NG - 1, p + NG, Cd2<PHYS>::F0, bar(p));
    };
    if (t == 0)
        for (int q = 0; q < VT::NS; q++) tc::mbar_init(tc::smem_u32(&full[q]), 1);
    __syncthreads();
    if (t == 0)
        for (int p = x0 - 1; p <= min(x0 - 2 + VT::NS, x1); p++) issue(p);
    const int cc = (ty + 1) * VT::BZ + lane + 1;
    double* v = V + ((long long)x0 * b.ny + j) * b.nz + k;
    typename Cd2<PHYS>::March m(c, b, j);
    for (int p = x0 - 1; p <= x1; p++) {
        const bool ok = tc::mbar_wait(bar(p), (uint32_t)(((p - x0 + 1) / VT::NS) & 1), kTilePolls);
        if (ok) {
            const double* P = vsm + slot(p) * VT::STRIDE + cc;
            m.enter([&](int f, int y, int z) { return P[f * (VT::BY * VT::BZ) + y * VT::BZ + z]; }, x_inside(p, b.nx, c));
        }
        // every thread has read plane p (and agrees on whether a wait ran out)
        if (__syncthreads_or(!ok)) {
            if (t == 0) {
                atomicOr(err, 1ull);
                // the loads still in flight
                for (int q = p; q <= min(p - 1 + VT::NS, x1); q++)
                    tc::mbar_wait(bar(q), (uint32_t)(((q - x0 + 1) / VT::NS) & 1), kTilePolls);
            }
            __syncthreads();
            return;
        }
        if (t == 0 && p + VT::NS <= x1) issue(p + VT::NS);
        if (p <= x0) continue;  // the first cell's own plane
        if (live) m.cell(c, v, vs);
        v += (long long)b.ny * b.nz;
    }
}

// ---------------------------------------------------------------------------
// host side

static PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }();
    return fn;
}

bool visc_tma_encode(VTmaMap* m, const double* W, const Box& b, int planes) {
    m->W = nullptr;
    PFN_cuTensorMapEncodeTiled_v12000 enc = encode_fn();
    if (!enc) return false;
    // dimensions innermost first: z (padded row), y, x, field
    const cuuint64_t dims[4] = {(cuuint64_t)b.NZp, (cuuint64_t)b.NY, (cuuint64_t)b.NX, (cuuint64_t)planes};
    const cuuint64_t strides[3] = {(cuuint64_t)b.NZp * 8, (cuuint64_t)b.NY * b.NZp * 8, (cuuint64_t)b.fstride * 8};
    const cuuint32_t estr[4] = {1, 1, 1, 1}, box[4] = {ViscTile::BZ, ViscTile::BY, 1, 4};
    if (enc(reinterpret_cast<CUtensorMap*>(m->map), CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, const_cast<double*>(W), dims,
            strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    m->W = W;
    return true;
}

template <bool PHYS>
static void viscous_cd2(const VTmaMap* m, const double* W, const Box& b, const Consts& c, double* V, long long vs,
                        unsigned long long* err, int sms, cudaStream_t s, Planes pl) {
    const int x0 = pl.n < 0 ? 0 : pl.lo, np = pl.n < 0 ? b.nx : pl.n;
    if (m) {
        dim3 grid((b.nz + 31) / 32, (b.ny + 3) / 4);
        const int lx = march_length(np, (long long)grid.x * grid.y, sms * ViscTile::MINB, 2.0, 64);
        grid.z = (np + lx - 1) / lx;
        cudaFuncSetAttribute(k_viscous_cd2_tma<PHYS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ViscTile::smem);
        k_viscous_cd2_tma<PHYS><<<grid, dim3(32, 4), ViscTile::smem, s>>>(
            *reinterpret_cast<const CUtensorMap*>(m->map), b, c, V, vs, err, x0, x0 + np, lx);
        return;
    }
    const long long blocks = row_tiles(b);
    const int lx = march_length(np, blocks, sms * 5, 2.0, 32);
    k_viscous_cd2<PHYS><<<dim3((unsigned)blocks, (np + lx - 1) / lx), dim3(32, 4), 0, s>>>(W, b, c, V, vs, x0, x0 + np,
                                                                                             lx);
}

template <int H, bool PHYS, bool SHARE>
static void viscous_one(const double* W, const Box& b, const Consts& c, double* V, long long vs, int sms,
                        cudaStream_t s, Planes pl) {
    using VR = ViscRing<H, PHYS>;
    // the attribute is per device; a refusal surfaces as the launch's error
    constexpr size_t bytes = VR::bytes + (SHARE ? VR::shared_bytes : 0);
    cudaFuncSetAttribute(k_viscous<H, PHYS, SHARE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    const int x0 = pl.n < 0 ? 0 : pl.lo, np = pl.n < 0 ? b.nx : pl.n;
    const long long blocks = row_tiles(b);
    // a segment costs its cells and 2H planes of the ring, about half a cell's work each
    const int lx = march_length(np, blocks, sms * VR::MINB, 1.0 + H, 32);
    k_viscous<H, PHYS, SHARE><<<dim3((unsigned)blocks, (np + lx - 1) / lx), dim3(32, 4), bytes, s>>>(
        W, b, c, V, vs, x0, x0 + np, lx);
}

void launch_viscous(int h, bool phys, const VTmaMap* m, const double* W, const Box& b, const Consts& c, double* V,
                    long long vs, unsigned long long* err, int sms, cudaStream_t s, Planes pl) {
    if (h == 1) {
        if (phys) viscous_cd2<true>(m, W, b, c, V, vs, err, sms, s, pl);
        else viscous_cd2<false>(m, W, b, c, V, vs, err, sms, s, pl);
    } else if (phys) {
        const bool share = c.dim == 3 && b.nz >= 32;
        if (h == 2 && share) viscous_one<2, true, true>(W, b, c, V, vs, sms, s, pl);
        else if (h == 2) viscous_one<2, true, false>(W, b, c, V, vs, sms, s, pl);
        else if (share) viscous_one<3, true, true>(W, b, c, V, vs, sms, s, pl);
        else viscous_one<3, true, false>(W, b, c, V, vs, sms, s, pl);
    } else {
        if (h == 2) viscous_one<2, false, false>(W, b, c, V, vs, sms, s, pl);
        else viscous_one<3, false, false>(W, b, c, V, vs, sms, s, pl);
    }
}

}  // namespace nsb
