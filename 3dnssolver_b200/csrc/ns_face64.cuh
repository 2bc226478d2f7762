// ns_face64.cuh -- FP64 WENO-5 face flux of one face (device functions).
//
// A face along axis DIR lies between cells a and a+1; its 6-cell stencil is
// a-2..a+3.  The numerical flux is WENO5_left(fL) + WENO5_right(fR) of the
// Lax-Friedrichs split fL = (F + alpha U)/2 (cells a-2..a+2), fR = (F - alpha U)/2
// (cells a-1..a+3), component-wise (Weno5::x/y/z_sweep,
// src/convection_schemes/weno-5.cpp:75-220) or in characteristic variables
// (Weno5cw::compute_num_flux, src/convection_schemes/weno-5cw.cpp:4-28).
//
// The face kernels are bound by the FP64 pipe, so the flux is arranged for few
// FP64 operations (about 650 characteristic-wise where the formulas taken
// literally need about 1000).  All of it is exact algebra; results differ from
// the literal form by rounding only:
//   - A WENO-5 value is its centre cell plus a combination of the stencil's four
//     differences: smoothness indicators and candidates depend on differences
//     alone (weno5_diff).  So differences are what is formed and projected, 4
//     columns a side instead of 5, and they are taken before the projection,
//     where they cancel least.
//   - The centre cells' share fL(a) + fR(a+1) needs no projection: R L = I.
//   - The right-biased reconstruction is the left-biased one on the reversed
//     stencil.
//   - The projection rows share their terms: with m = (momentum) - u (density) and
//     h = (energy) - u.m - |u|^2/2 (density), L f = (K/(2c^2) h -+ m_n/(2c), m_t,
//     density - K/c^2 h).  The acoustic fields are taken 2c times as large (WENO is
//     homogeneous when its epsilon is scaled with them), the tangential ones up to
//     their sign.
//   - Everything is formed for the doubled flux F +- alpha U; the candidates' 1/6 is
//     applied once, at the end, and the 1/2 left to the flux differences' 1/dx.
//
// Measured on B200 against the literal form (6 U/F/2 and ten projected columns a
// face, weights on the stencil values) in the kernels of the time, ms per step of 3
// stages: Taylor-Green 384^3 physical characteristic-wise y/z faces 12.40/12.54 ->
// 9.53/9.56, x-march 15.18 -> 12.76; shear layer 256^3 reference characteristic-wise
// 3.10/3.04 -> 2.33/2.18, x-march 4.34 -> 3.71; Sod 512x128x128 component-wise 1.23/1.22
// -> 0.95/0.92.  A further 25 operations (third-order reciprocals, factors left to the
// caller) took the shear layer from 8.46 to 8.30 ms a step, faces 2.25/2.15 -> 2.18/2.09.
// The error of the right-hand side against 80-bit arithmetic falls too, 1.1 to 25 times in
// 44 of 48 combinations of form and flow (smooth, rough, Taylor-Green, shear, Sod, SI
// units), and is within 3e-16 of it in the others.  (Figures before the quotient's
// scaling, weno5_pair_diff, which adds 5 operations and changes no bit of these.)
#pragma once

#include "ns_common.cuh"
#include "ns_eos.cuh"
#include "ns_face.cuh"

namespace nsb {

// Smoothness indicators are kept at 12/13 of their value (the coefficient 13/12 of
// the second difference becomes 1), which the epsilon follows; the doubled flux
// makes them 4 times as large.
constexpr double kWenoEpsScale = 4.0 * 12.0 / 13.0;
template <bool BORGES>
struct WenoEps {
    static constexpr double value = kWenoEpsScale * (BORGES ? 1e-14 : 1e-6);
};

// WENO-5 (weno-5.cpp:222-322) from the differences d0..d3 of the stencil
// (d0 = b - a .. d3 = e - d): 6 (value - c) = d1 + 2 d2 + 2 num/den.  The candidates
// are taken relative to the central one: 6 (f0 - f1) = 2 (D0 - D1), 6 (f2 - f1) =
// D1 - D2 with the second differences D.  The nonlinear weights d_k / s_k^2 (Borges:
// d_k (1 + tau/B_k)) are multiplied by the product of all denominators.
template <bool BORGES>
__device__ __forceinline__ void weno5_diff(double d0, double d1, double d2, double d3, double eps, double& num,
                                           double& den) {
    constexpr double k = 3.0 / 13.0;  // 1/4 at the indicators' scale
    const double D0 = d1 - d0, D1 = d2 - d1, D2 = d3 - d2;
    const double t0 = fma(3.0, d1, -d0), t1 = d1 + d2, t2 = fma(3.0, d2, -d3);
    const double s0 = fma(D0, D0, fma(k * t0, t0, eps));
    const double s1 = fma(D1, D1, fma(k * t1, t1, eps));
    const double s2 = fma(D2, D2, fma(k * t2, t2, eps));
    const double p0 = s1 * s2, p1 = s0 * s2, p2 = s0 * s1;
    double x, y, z;
    if constexpr (BORGES) {
        const double tau = fabs(s0 - s2);
        x = (s0 + tau) * p0;
        y = (s1 + tau) * p1;
        z = (s2 + tau) * p2;
    } else {
        x = p0 * p0;
        y = p1 * p1;
        z = p2 * p2;
    }
    num = fma(1.5, z * (D1 - D2), x * (D0 - D1));
    den = fma(3.0, z, fma(6.0, y, x));
}

// 6 (WENO5_left(l) + WENO5_right(r) - centre cells) from the left stencil's
// differences and the reversed right stencil's, with one division: nL/dL + nR/dR =
// (nL dR + nR dL) / (dL dR).  A denominator is of the eighth order in the differences
// (Shu), so dL dR would leave the double range where these pass 1e18: half or, for the
// acoustic fields (2c times as large), a small fraction of what the literal form bears.
// Both terms therefore take dL at the exponent of [2, 4), and dR times the same power of two
// f; being a power of two it changes no bit of the quotient, and differences up to 1e33
// pass.  One multiplication a field, 0.6 to 1.4% of a step (Taylor-Green 384^3 168.6 ->
// 170.4 ms a pass of 4 steps, shear layer 256^3 8.23 -> 8.34 ms a step).  A check of the
// exponents that forms a face again where it fails cost nearly as much, 8.31, for twice
// the code.  (f is 0 for a dL that is not finite, which makes the denominator and so the
// result NaN.)
template <bool BORGES>
__device__ __forceinline__ double weno5_pair_diff(const double l[4], const double r[4], double eps) {
    double nL, dL, nR, dR;
    weno5_diff<BORGES>(l[0], l[1], l[2], l[3], eps, nL, dL);
    weno5_diff<BORGES>(r[0], r[1], r[2], r[3], eps, nR, dR);
    const int hi = __double2hiint(dL);
    const double f = __hiloint2double(0x7ff00000 - (hi & 0x7ff00000), 0);
    const double fdL = __hiloint2double((hi & 0x000fffff) | 0x40000000, __double2loint(dL));
    const double fdR = f * dR;
    const double lin = fma(2.0, l[2] + r[2], l[1] + r[1]);
    return fma(2.0, div_pos_nr(fma(nL, fdR, nR * fdL), dL * fdR), lin);
}

// U and the Euler flux along DIR of one cell (ConvectionFlux::form_flux,
// convection_flux.cpp:23-61).  WONLY: U = cons(W), formed here; else u holds the
// caller's U and the flux is W's alone.
template <int DIR, bool WONLY>
__device__ __forceinline__ void cell_flux(const double w[5], double inv_gm1, double u[5], double f[5]) {
    const double m[3] = {w[0] * w[2], w[0] * w[3], w[0] * w[4]};
    const double k2 = fma(m[2], w[4], fma(m[1], w[3], m[0] * w[2]));
    const double e = fma(0.5, k2, w[1] * inv_gm1);
    const double qn = w[2 + DIR];
    if constexpr (WONLY) {
        u[0] = w[0];
        u[1] = e;
        u[2] = m[0];
        u[3] = m[1];
        u[4] = m[2];
    }
    f[0] = m[DIR];
    f[1] = qn * (e + w[1]);
#pragma unroll
    for (int a = 0; a < 3; a++) f[2 + a] = a == DIR ? fma(m[a], qn, w[1]) : m[a] * qn;
}

// Twice the numerical flux of one face.  Of stencil cell s = 0..5, cell(s, u, f) gives U
// and the flux, prim(s, w) gives W (asked of cells 2 and 3), and lam(s) gives |q_n| + c
// (physical semantics).
template <int DIR, bool CHAR, bool BORGES, bool PHYS, typename Cell, typename Prim, typename Speed>
__device__ __forceinline__ void face_flux64(Cell cell, Prim prim, Speed lam, const Consts& c, double out[5]) {
    // local Lax-Friedrichs speed, the largest of the 6 cells (physical semantics; the
    // reference's is the constant 3, convection_flux.cpp:241)
    double alpha = 3.0;
    if constexpr (PHYS) {
#pragma unroll
        for (int s = 0; s < 6; s++) {
            const double a = lam(s);
            alpha = (s == 0) ? a : (a > alpha ? a : alpha);
        }
    }
    // eigensystem at the arithmetic face average (ConvectionFlux::eigenvectors,
    // convection_flux.cpp:117-175); the reference semantics' c2 is gamma/(p rho) (:139)
    double v[3], hq2 = 0, cs2 = 0, K2pc = 0, kc = 0, inv2c = 0;
    if constexpr (CHAR) {
        double wa[5], wb[5];
        prim(2, wa);
        prim(3, wb);
#pragma unroll
        for (int q = 0; q < 5; q++) wa[q] = wa[q] + wb[q];  // twice the average
#pragma unroll
        for (int a = 0; a < 3; a++) v[a] = 0.5 * wa[2 + a];
        hq2 = 0.5 * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
        double ic, cs;  // 1/c and c
        if constexpr (PHYS) {
            // rho r and gamma p r with r = 1/sqrt(gamma p rho): the doubling cancels
            const double gp = c.gamma * wa[1];
            const double r = rsqrt_pos_nr(gp * wa[0]);
            ic = wa[0] * r;
            cs = gp * r;
        } else {
            // sqrt(p rho / gamma) and sqrt(gamma / (p rho)), with p rho four times as large
            const double pr = wa[1] * wa[0];
            const double r = rsqrt_pos_nr(pr);
            ic = c.half_inv_sqrt_gamma * (pr * r);
            cs = c.two_sqrt_gamma * r;
        }
        cs2 = cs * cs;
        kc = c.gm1 * ic;    // K/c
        K2pc = kc * ic;     // K/c^2
        inv2c = 0.5 * ic;
    }
    // state index of the textbook components [rho, rho u, rho v, rho w, rho E]
    constexpr int s0 = st<PHYS>(0), s4 = st<PHYS>(4);
    constexpr int sm[3] = {st<PHYS>(1), st<PHYS>(2), st<PHYS>(3)};
    constexpr int T1 = Frame<DIR>::m_ax, T2 = Frame<DIR>::l_ax;  // tangential axes
    // L applied to one column of differences, fields (2c u-c, 2c u+c, m, l, entropy)
    auto project = [&](const double d[5], double g[5]) {
        if constexpr (!CHAR) {
#pragma unroll
            for (int q = 0; q < 5; q++) g[q] = d[q];
        } else {
            const double r = d[s0];
            double m[3];
#pragma unroll
            for (int a = 0; a < 3; a++) m[a] = fma(-v[a], r, d[sm[a]]);
            double h = fma(-hq2, r, d[s4]);
#pragma unroll
            for (int a = 0; a < 3; a++) h = fma(-v[a], m[a], h);
            g[0] = fma(kc, h, -m[DIR]);
            g[1] = fma(kc, h, m[DIR]);
            g[2] = m[T1];
            g[3] = m[T2];
            g[4] = fma(-K2pc, h, r);
        }
    };
    // the cells in order: differences of F + alpha U between cells s-1 and s (s = 1..4)
    // and, reversed, of F - alpha U (s = 2..5)
    double gl[5][4], gr[5][4], cen[5], up[5], fp[5];
#pragma unroll
    for (int s = 0; s < 6; s++) {
        double u[5], f[5];
        cell(s, u, f);
        if (s > 0) {
            double l[5], r[5], g[5];
#pragma unroll
            for (int q = 0; q < 5; q++) {
                const double du = u[q] - up[q], df = f[q] - fp[q];
                l[q] = fma(alpha, du, df);
                r[q] = fma(alpha, du, -df);
                if (s == 3) cen[q] = fma(-alpha, du, f[q] + fp[q]);  // doubled centre cells' share
            }
            if (s <= 4) {
                project(l, g);
#pragma unroll
                for (int q = 0; q < 5; q++) gl[q][s - 1] = g[q];
            }
            if (s >= 2) {
                project(r, g);
#pragma unroll
                for (int q = 0; q < 5; q++) gr[q][5 - s] = g[q];
            }
        }
#pragma unroll
        for (int q = 0; q < 5; q++) {
            up[q] = u[q];
            fp[q] = f[q];
        }
    }
    constexpr double eps = WenoEps<BORGES>::value;
    const double epsc = CHAR ? eps * (4.0 * cs2) : eps;
    double ft[5];
#pragma unroll
    for (int q = 0; q < 5; q++) ft[q] = weno5_pair_diff<BORGES>(gl[q], gr[q], q < 2 ? epsc : eps);
    constexpr double k6 = 1.0 / 6.0;
    if constexpr (!CHAR) {
#pragma unroll
        for (int q = 0; q < 5; q++) out[q] = fma(k6, ft[q], cen[q]);
    } else {
        // back-projection R ft (textbook rows of R, convection_flux.cpp:153-158)
        const double p = inv2c * (ft[0] + ft[1]), hd = 0.5 * (ft[1] - ft[0]);  // ft+ + ft-, c (ft+ - ft-)
        const double acc = p + ft[4];
        double tb[5];
        tb[0] = acc;
        tb[1 + DIR] = fma(v[DIR], acc, hd);
        tb[1 + T1] = fma(v[T1], acc, ft[2]);
        tb[1 + T2] = fma(v[T2], acc, ft[3]);
        const double H = fma(cs2, c.inv_gm1, hq2);
        tb[4] = fma(H, p, fma(v[DIR], hd, fma(v[T1], ft[2], fma(v[T2], ft[3], hq2 * ft[4]))));
#pragma unroll
        for (int t = 0; t < 5; t++) out[st<PHYS>(t)] = fma(k6, tb[t], cen[st<PHYS>(t)]);
    }
}

// The faces of a time step, twice the flux: U = cons(W), and at(q, s) gives plane q of stencil cell
// s, W in planes 0..4 and (physical semantics) the sound speed in plane 6.
template <int DIR, bool CHAR, bool BORGES, bool PHYS, typename At>
__device__ __forceinline__ void face_flux64_w(At at, const Consts& c, double out[5]) {
    auto ld = [&](int s, double w[5]) {
#pragma unroll
        for (int q = 0; q < 5; q++) w[q] = at(q, s);
    };
    auto cell = [&](int s, double u[5], double f[5]) {
        double w[5];
        ld(s, w);
        cell_flux<DIR, true>(w, c.inv_gm1, u, f);
    };
    auto lam = [&](int s) { return fabs(at(2 + DIR, s)) + at(6, s); };
    face_flux64<DIR, CHAR, BORGES, PHYS>(cell, ld, lam, c, out);
}

// the faces of an operator call: W and the caller's U in device memory, stencil
// cell 0 at o0, stride step
template <int DIR, bool CHAR, bool BORGES, bool PHYS>
__device__ __forceinline__ void face_flux64_wu(const double* __restrict__ W, const double* __restrict__ U,
                                               const Box& b, const Consts& c, long long o0, long long step,
                                               double out[5]) {
    auto ld = [&](int s, double w[5]) {
#pragma unroll
        for (int q = 0; q < 5; q++) w[q] = W[q * b.fstride + o0 + s * step];
    };
    auto cell = [&](int s, double u[5], double f[5]) {
        double w[5];
        ld(s, w);
#pragma unroll
        for (int q = 0; q < 5; q++) u[q] = U[q * b.fstride + o0 + s * step];
        cell_flux<DIR, false>(w, c.inv_gm1, u, f);
    };
    auto lam = [&](int s) {
        double w[5];
        ld(s, w);
        return fabs(w[2 + DIR]) + sound_speed(w, c.gamma);
    };
    face_flux64<DIR, CHAR, BORGES, PHYS>(cell, ld, lam, c, out);
#pragma unroll
    for (int q = 0; q < 5; q++) out[q] *= 0.5;
}

}  // namespace nsb
