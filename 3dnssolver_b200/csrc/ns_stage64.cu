// ns_stage64.cu -- the convection of an FP64 time step's stage: the y- and z-face
// fluxes, and the x-march that forms the x-faces and updates the cells.
//
// The face kernels read their stencils straight from global memory: a stencil is one
// pass over W and the sound speed plane (physical semantics), five sixths of it
// in L1.  Threads are numbered through rows and planes, so warps are full at any
// extent and no axis needs a launch for its last face plane.
//
// Bound: the FP64 pipe, 75% (y) and 81% (z) busy.  One face per thread, nothing carried:
// 16 warps per SM (128 registers) hide the stencil's latency and each other's dependent
// chains.  ms per step, y/z: Taylor-Green 384^3 12.4/12.5 -> 8.1/7.6, shear layer 256^3
// 3.10/3.04 -> 2.22/2.12 (fluxes on differences, the sound speed's plane, no tiles).
// Tried and slower on B200 (Taylor-Green 384^3, ms per step, y/z 7.94/7.58 in the same
// runs): 12 warps per SM 8.27/7.77; the sound speeds formed per face 9.47/9.50; tiles
// of W staged by TMA 8.90/9.01; flux differences instead of fluxes, y marched per
// thread and z through shared memory 9.50/8.74.
#include <cuda_runtime.h>

#include <algorithm>

#include "ns_common.cuh"
#include "ns_eos.cuh"
#include "ns_face64.cuh"
#include "ns_kernels.h"

namespace nsb {

constexpr int kFaceBlocks = 4;  // per SM

// y-faces (twice the flux): a block takes 4 face rows x 32 columns, the columns (i, k) of the x-planes
// numbered through.
template <bool CHAR, bool BORGES, bool PHYS>
__global__ void __launch_bounds__(128, kFaceBlocks)
    k_faces_y(const double* __restrict__ W, Box b, Consts c, double* __restrict__ F, FaceBox fb, int x0,
              long long columns) {
    const int jf = blockIdx.x * 4 + threadIdx.y;  // between cells jf - 1 and jf
    const long long e = (long long)blockIdx.y * 32 + threadIdx.x + (long long)blockIdx.z * 65535 * 32;
    if (e >= columns || jf > b.ny) return;
    const int i = x0 + (int)(e / b.nz), k = (int)(e % b.nz);
    const double* w = W + b.at(i + NG, jf, k + NG);  // stencil cell 0
    auto at = [&](int q, int s) { return w[q * b.fstride + s * b.NZp]; };
    double f[5];
    face_flux64_w<1, CHAR, BORGES, PHYS>(at, c, f);
    double* o = F + fb.at(i, jf, k);
#pragma unroll
    for (int q = 0; q < 5; q++) o[q * fb.fstride] = f[q];
}

// z-faces (twice the flux): one thread per face of the rows' nz + 1 faces, numbered through
template <bool CHAR, bool BORGES, bool PHYS>
__global__ void __launch_bounds__(128, kFaceBlocks)
    k_faces_z(const double* __restrict__ W, Box b, Consts c, double* __restrict__ F, FaceBox fb, int x0,
              long long faces) {
    const long long e = (long long)blockIdx.x * 128 + threadIdx.x;
    if (e >= faces) return;
    const long long row = e / (b.nz + 1);
    const int kf = (int)(e % (b.nz + 1)), i = x0 + (int)(row / b.ny), j = (int)(row % b.ny);
    const double* w = W + b.at(i + NG, j + NG, kf);  // stencil cell 0 of the face between cells kf - 1 and kf
    auto at = [&](int q, int s) { return w[q * b.fstride + s]; };
    double f[5];
    face_flux64_w<2, CHAR, BORGES, PHYS>(at, c, f);
    double* o = F + fb.at(i, j, kf);
#pragma unroll
    for (int q = 0; q < 5; q++) o[q * fb.fstride] = f[q];
}

// ---------------------------------------------------------------------------
// The FP64 stage's x-march: x-face fluxes formed along x together with the cell
// update of each cell as soon as both of its x-faces are known, so the x-faces
// never reach HBM.  One thread per column (j, k), the columns numbered through so
// that warps are full at any extent, marching lx cells.  A thread's stencil is its
// own column's alone, so each keeps a private ring of 7 planes in shared memory, filled
// with cp.async: planes i-2 .. i+3 feed the x-face between cells i and i+1 while plane
// i+4 is in flight, with no barrier between the threads.  The ring holds the stage's
// input U itself, which the update reads from it as well, and what a face needs besides:
// p, 1/rho and (in registers) |u| + c, formed once as a plane arrives (the same W = prim(U) that the
// other kernels read, and a cell's flux takes 6 operations instead of 13).  U0 of the
// update comes by cp.async too; the face fluxes of the other axes and the viscous terms
// are read at the update.  Ghost planes are U's folded planes.  Uout is a second
// buffer: neighbouring segments still read U.
//
// LAST (third stage): the next step's start as well -- W = prim(U_out) for its
// CFL minimum (time_scheme.cpp:69, 98-136) into slot_next and U0 = cons(W)
// (the W -> U round trip of time_scheme.cpp:124); U_out itself stays the raw
// stage result, as the reference's U holds it between steps.  In the first stage U
// and U0 are one buffer, only read, and only once; U0 is written in the third stage
// only, where it is not U (so the restrict qualifiers hold).
//
// Bound: memory (291 bytes a cell measured, 7.6 ms a step at 384^3 at the copy rate:
// 66% of it) and the FP64 pipe (61% busy) together, at 12 warps per SM.  Three blocks per SM hold
// the ring without spills.  ms per step (Taylor-Green 384^3 / shear layer 256^3 / Sod
// 512x128x128 component-wise): this 11.3 / 3.28 / 1.54; a ring of W and U read besides
// 12.0 / 3.31 / 1.58; planes of W through TMA on mbarriers with a block barrier per cell
// 12.3 / 3.51 / 1.69; with the faces' operands staged too 13.2 / 3.65 / 1.75; U0 not staged
// 15.3 / 4.53 / 2.18; four blocks of 128 registers 15.7 / 3.61 / 1.60.  |u| + c in the ring
// instead of in registers: 13.6 at 384^3 (7 KB less L1 for the operands read at the update).
//
// IMAGES: each cell's W also goes to the ghost cells that fold onto it, over edges and
// corners too, so that the next stage needs no launch of its own for them.
constexpr int kXMarchBlocks = 3;  // per SM
struct XMarchLayout {
    static constexpr int NF = 7, NS = 7;  // U, p, 1/rho
    static constexpr size_t bytes = (size_t)(NS * NF + 5 + 5) * 128 * 8;
};

// The ghost indices -3 .. -1 (bits 0..2) and n .. n+2 (bits 3..5) that fold onto index a
// of an axis of n cells, and a itself (bit 6).
__device__ __forceinline__ unsigned images(int a, int n, int periodic) {
    unsigned m = 64;
    if (periodic) {
        for (int g = 0; g < 6; g++)
            if (fold(g < 3 ? g - 3 : n + g - 3, n, 1) == a) m |= 1u << g;
    } else {
        if (a == 0) m |= 7;
        if (a == n - 1) m |= 56;
    }
    return m;
}
__device__ __forceinline__ int image(int bit, int a, int n) { return bit == 6 ? a : (bit < 3 ? bit - 3 : n + bit - 3); }
template <bool CHAR, bool BORGES, bool PHYS, bool LAST, bool IMAGES>
__global__ void __launch_bounds__(128, kXMarchBlocks)
    k_xmarch(const double* __restrict__ U, double* __restrict__ U0,
             double* __restrict__ Uout, double* __restrict__ Wn, const double* __restrict__ Fy,
             const double* __restrict__ Fz, const double* __restrict__ V, long long vs, Box b, FaceBox fy, FaceBox fz,
             Consts c, const unsigned long long* __restrict__ slot, unsigned long long* __restrict__ slot_next,
             double m1, double m2, double mc, double* __restrict__ clock, unsigned long long* __restrict__ slot_reset,
             int xlo, int xhi, int lx) {
    constexpr int NF = XMarchLayout::NF, NS = XMarchLayout::NS;
    extern __shared__ double xsm[];
    const int t = threadIdx.y * 32 + threadIdx.x;
    double* ring = xsm + t;                // [NS][NF][128]
    double* fprev = ring + NS * NF * 128;  // [5][128]
    double* opnd = fprev + 5 * 128;        // [5][128]: U0 of the cell
    int j, k;
    const bool live = row_tile(b, j, k);
    // threads outside the grid march no cells but join the block reduction of LAST
    const int x0 = xlo + blockIdx.y * lx, x1 = live ? min(x0 + lx, xhi) : x0 - 1;
    double best = INFINITY;
    const double dt = fmin(1e10, __longlong_as_double((long long)*slot)) * c.cfl;
    const double m3 = mc * dt;
    if (clock && (blockIdx.x | blockIdx.y | t) == 0) {
        clock[0] = dt;
        clock[1] += dt;
        *slot_reset = ~0ull;  // for the third stage
    }
    // the column's images along y and z (in 2D no stencil runs along z)
    unsigned mj = 64, mk = 64;
    if constexpr (IMAGES) {
        mj = images(j, b.ny, c.periodic[1]);
        if (c.dim == 3) mk = images(k, b.nz, c.periodic[2]);
    }
    const bool first = U == U0;  // the first stage's input is the step's start
    auto slot_of = [&](int p) { return ring + ((p - x0 + 3) % NS) * NF * 128; };
    auto load_plane = [&](int p) {
        const double* u = U + b.at(fold_x(p, b.nx, c) + NG, j + NG, k + NG);
        double* d = slot_of(p);
#pragma unroll
        for (int q = 0; q < 5; q++) cp_async8(d + q * 128, u + q * b.fstride);
    };
    double win[6] = {0, 0, 0, 0, 0, 0};  // |u| + c of planes i-2 .. i+3 (physical semantics)
    auto arrived = [&](int p) {  // p, 1/rho and |u| + c of a plane
        double* d = slot_of(p);
        double u[5], w[5];
#pragma unroll
        for (int q = 0; q < 5; q++) u[q] = d[q * 128];
        prim_from_cons(u, c.gm1, w);
        d[5 * 128] = w[1];
        d[6 * 128] = 1.0 / u[0];
        if constexpr (PHYS) {
#pragma unroll
            for (int s = 0; s < 5; s++) win[s] = win[s + 1];
            win[5] = fabs(w[2]) + sound_speed(w, c.gamma);
        }
    };
    if (live)
        for (int p = x0 - 3; p < x0 + 3; p++) load_plane(p);
    cp_async_commit();
    cp_async_wait_all();
    if (live)
        for (int p = x0 - 3; p < x0 + 2; p++) arrived(p);
    for (int i = x0 - 1; i < x1; i++) {
        const long long o = b.at(i + NG, j + NG, k + NG);
        if (i + 4 <= x1 + 2) load_plane(i + 4);
        if (i >= x0 && !first) {
#pragma unroll
            for (int q = 0; q < 5; q++) cp_async8(opnd + q * 128, U0 + q * b.fstride + o);
        }
        cp_async_commit();
        // plane i + 3 has landed (beyond the first cell by the update's wait, which drains
        // plane i + 4 with U0: the next plane's latency is covered by one face, not two)
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        arrived(i + 3);
        const double* P[6];
#pragma unroll
        for (int s = 0; s < 6; s++) P[s] = slot_of(i - 2 + s);
        auto cell = [&](int s, double u[5], double g[5]) {
            const double* d = P[s];
#pragma unroll
            for (int q = 0; q < 5; q++) u[q] = d[q * 128];
            const double pr = d[5 * 128], vel = u[2] * d[6 * 128];
            g[0] = u[2];
            g[1] = (u[1] + pr) * vel;
            g[2] = fma(u[2], vel, pr);
            g[3] = u[3] * vel;
            g[4] = u[4] * vel;
        };
        auto prim = [&](int s, double w[5]) {
            const double* d = P[s];
            const double ir = d[6 * 128];
            w[0] = d[0];
            w[1] = d[5 * 128];
#pragma unroll
            for (int a = 0; a < 3; a++) w[2 + a] = d[(2 + a) * 128] * ir;
        };
        auto lam = [&](int s) { return win[s]; };
        double f[5];
        face_flux64<0, CHAR, BORGES, PHYS>(cell, prim, lam, c, f);
        if (i < x0) {
#pragma unroll
            for (int q = 0; q < 5; q++) fprev[q * 128] = f[q];
            continue;
        }
        cp_async_wait_all();
        const double* py = Fy + fy.at(i, j, k);
        const double* pz = Fz + fz.at(i, j, k);
        const double* pv = V + ((long long)i * b.ny + j) * b.nz + k;
        double un[5], w[5];
#pragma unroll
        for (int q = 0; q < 5; q++) {
            // the residual in k_update's order: x, y, z differences, then the viscous terms
            // (the faces hold twice the flux)
            double r = (f[q] - fprev[q * 128]) * c.half_inv[0];
            fprev[q * 128] = f[q];
            r += (py[q * fy.fstride + b.nz] - py[q * fy.fstride]) * c.half_inv[1];
            if (Fz) r += (pz[q * fz.fstride + 1] - pz[q * fz.fstride]) * c.half_inv[2];
            if (q && V) r += pv[(q - 1) * vs];
            const double u = P[2][q * 128], u0 = first ? u : opnd[q * 128];
            un[q] = (u0 * m1) + (u * m2) + (r * m3);
            Uout[q * b.fstride + o] = un[q];
        }
        prim_from_cons(un, c.gm1, w);  // the next stage's W
        if constexpr (LAST) {
            double u0[5];
            const double d = PHYS ? local_dt_physical(w, c) : local_dt(w, c);
            if (d < best) best = d;  // NaN never lowers the minimum
            cons_from_prim(w, c.inv_gm1, u0);
#pragma unroll
            for (int q = 0; q < 5; q++) U0[q * b.fstride + o] = u0[q];
            prim_from_cons(u0, c.gm1, w);  // the next step's first stage reads prim(U0)
        }
        store_w<PHYS>(Wn, b.fstride, o, w, c.gamma);
        if constexpr (IMAGES) {
            const unsigned mi = i < NG || i >= b.nx - NG ? images(i, b.nx, c.periodic[0]) : 64;
            if ((mi | mj | mk) == 64) continue;
            for (unsigned x = mi; x; x &= x - 1)
                for (unsigned y = mj; y; y &= y - 1) {
                    const long long row = b.at(image(__ffs(x) - 1, i, b.nx) + NG, image(__ffs(y) - 1, j, b.ny) + NG, NG);
                    for (unsigned z = mk; z; z &= z - 1) {
                        const long long g = row + image(__ffs(z) - 1, k, b.nz);
                        if (g != o) store_w<PHYS>(Wn, b.fstride, g, w, c.gamma);
                    }
                }
        }
    }
    cp_async_wait_all();
    if constexpr (LAST) block_min_to(best, slot_next);
}

// ---------------------------------------------------------------------------
// host side

// Cells per thread of a march over n cells with `blocks` blocks across: the length
// whose waves cost least, a segment costing its cells and `extra` more (its first
// face, and the first planes' latency).  Long segments where the grid fills the GPU
// many times over, short ones where it does not: with 64 cells throughout, the 64^3
// x-march was 32 blocks on 148 SMs, 0.40 ms a step where it now takes 0.084.  Beyond
// eight waves a partly filled last one hardly matters, and more segments only cost.
// `longest`: longer marches drift apart and lose the planes that blocks share in L2
// (viscous march, Taylor-Green 384^3: 3.73 ms a step at 32 cells, 4.13 at 128).
int march_length(int n, long long blocks, int resident, double extra, int longest) {
    int best = n;
    double cost = 1e300;
    for (int most = std::min(n, longest); most >= 1; most--) {
        const int seg = (n + most - 1) / most, len = (n + seg - 1) / seg;
        const long long waves = (blocks * seg + resident - 1) / resident;
        const double w = waves > 8 ? (double)blocks * seg / resident : (double)waves;
        if (w * (len + extra) < cost * (1 - 1e-9)) {
            cost = w * (len + extra);
            best = len;
        }
        if (waves > 8) break;
    }
    return best;
}

template <bool CHAR, bool BORGES, bool PHYS>
static void step_faces_one(int dir, const double* W, const Box& b, const Consts& c, double* F, const FaceBox& fb,
                           cudaStream_t s, Planes pl) {
    const int x0 = pl.n < 0 ? 0 : pl.lo, xn = pl.n < 0 ? b.nx : pl.n;
    if (dir == 1) {
        const long long columns = (long long)xn * b.nz, blocks = (columns + 31) / 32;
        const dim3 grid((b.ny + 1 + 3) / 4, (unsigned)std::min(blocks, 65535ll), (unsigned)((blocks + 65534) / 65535));
        k_faces_y<CHAR, BORGES, PHYS><<<grid, dim3(32, 4), 0, s>>>(W, b, c, F, fb, x0, columns);
    } else {
        const long long faces = (long long)xn * b.ny * (b.nz + 1);
        k_faces_z<CHAR, BORGES, PHYS><<<(unsigned)((faces + 127) / 128), 128, 0, s>>>(W, b, c, F, fb, x0, faces);
    }
}

void launch_step_faces(int dir, bool chr, bool borges, bool phys, const double* W, const Box& b, const Consts& c,
                       double* F, const FaceBox& fb, cudaStream_t s, Planes pl) {
    if (chr) {
        if (borges) {
            if (phys) step_faces_one<true, true, true>(dir, W, b, c, F, fb, s, pl);
            else step_faces_one<true, true, false>(dir, W, b, c, F, fb, s, pl);
        } else {
            if (phys) step_faces_one<true, false, true>(dir, W, b, c, F, fb, s, pl);
            else step_faces_one<true, false, false>(dir, W, b, c, F, fb, s, pl);
        }
    } else {
        if (borges) {
            if (phys) step_faces_one<false, true, true>(dir, W, b, c, F, fb, s, pl);
            else step_faces_one<false, true, false>(dir, W, b, c, F, fb, s, pl);
        } else {
            if (phys) step_faces_one<false, false, true>(dir, W, b, c, F, fb, s, pl);
            else step_faces_one<false, false, false>(dir, W, b, c, F, fb, s, pl);
        }
    }
}

template <bool CHAR, bool BORGES, bool PHYS, bool LAST, bool IMAGES>
static void xmarch_one(const XMarchArgs& a, cudaStream_t s, Planes pl) {
    constexpr size_t bytes = XMarchLayout::bytes;
    auto kern = k_xmarch<CHAR, BORGES, PHYS, LAST, IMAGES>;
    // the attribute is per device; a refusal surfaces as the launch's error
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    const int x0 = pl.n < 0 ? 0 : pl.lo, np = pl.n < 0 ? a.b.nx : pl.n;
    const long long blocks = row_tiles(a.b);
    // a segment costs its cells, its first face and the latency of its first planes
    const int lx = march_length(np, blocks, a.sms * kXMarchBlocks, 2.0, 64);
    kern<<<dim3((unsigned)blocks, (np + lx - 1) / lx), dim3(32, 4), bytes, s>>>(
        a.U, a.U0, a.Uout, a.Wnext, a.Fy, a.Fz, a.V, a.vs, a.b, a.fy, a.fz, a.c, a.slot,
        LAST ? a.slot_next : nullptr, a.m1, a.m2, a.mc, a.clock, a.slot_reset, x0, x0 + np, lx);
}

template <bool CHAR, bool BORGES, bool PHYS>
static void xmarch_last(const XMarchArgs& a, cudaStream_t s, Planes pl) {
    if (a.images) {
        if (a.slot_next) xmarch_one<CHAR, BORGES, PHYS, true, true>(a, s, pl);
        else xmarch_one<CHAR, BORGES, PHYS, false, true>(a, s, pl);
    } else {
        if (a.slot_next) xmarch_one<CHAR, BORGES, PHYS, true, false>(a, s, pl);
        else xmarch_one<CHAR, BORGES, PHYS, false, false>(a, s, pl);
    }
}

void launch_xmarch(bool chr, bool borges, bool phys, const XMarchArgs& a, cudaStream_t s, Planes pl) {
    if (chr) {
        if (borges) { if (phys) xmarch_last<true, true, true>(a, s, pl); else xmarch_last<true, true, false>(a, s, pl); }
        else { if (phys) xmarch_last<true, false, true>(a, s, pl); else xmarch_last<true, false, false>(a, s, pl); }
    } else {
        if (borges) { if (phys) xmarch_last<false, true, true>(a, s, pl); else xmarch_last<false, true, false>(a, s, pl); }
        else { if (phys) xmarch_last<false, false, true>(a, s, pl); else xmarch_last<false, false, false>(a, s, pl); }
    }
}

}  // namespace nsb
