// ns_kernels.h -- host-side launchers of the device kernels (internal).
#pragma once

#include <cuda_runtime.h>

#include "ns_common.cuh"

namespace nsb {

enum { MODE_STAGE = 0, MODE_RHS = 1 };
enum { UPD_CONV = 1, UPD_CONVZ = 2, UPD_OVERWRITE = 4 };

struct UpdateArgs {
    const double* W;
    double* U;
    const double* U0;
    const void* F[3];
    Box b;
    FaceBox fb[3];
    Consts c;
    int flags;       // UPD_*
    int mode;        // MODE_*
    bool viscous;
    bool phys;
    bool fp32;
    const unsigned long long* slot;  // reduced CFL minimum of this step
    double m1, m2, mc;               // U = U0*m1 + U*m2 + R*(mc*dt)
    double* Rout;                    // MODE_RHS target (halo'd SoA)
    double* clock;                   // [last dt, accumulated time], updated once per step (nullable)
};

// the x-march of an FP64 stage (launch_xmarch)
struct XMarchArgs {
    const double* U;    // the stage's input (on a slab with its exchanged ghost planes)
    double* U0;         // the step's start
    double* Uout;       // the stage's output buffer
    double* Wnext;      // receives the next stage's W (interior)
    const double* Fy;   // y- and z-face fluxes (Fz null in 2D)
    const double* Fz;
    const double* V;    // viscous terms of components 1..4 (null without): planes of stride
    long long vs;       // vs of the interior cells ((i ny + j) nz + k)
    Box b;
    FaceBox fy, fz;
    Consts c;
    const unsigned long long* slot;  // CFL minimum of this step
    unsigned long long* slot_next;   // third stage: the next step's CFL minimum (U0 then receives
                                     // the next step's start), else null
    double m1, m2, mc;               // U = U0*m1 + U*m2 + R*(mc*dt)
    double* clock;                   // first stage: [last dt, accumulated time]
    unsigned long long* slot_reset;  // first stage: the slot that the third stage reduces into
    bool images;                     // Wnext's ghost cells too (not on a slab)
    int sms;                         // multiprocessors of the device
};

// per-face flags of the learned sensor (1 = characteristic-wise), FaceBox order
struct Gate {
    const unsigned char* m[3];
    FaceBox fb[3];
};

// The learned sensor's flags of a step in the form the correction passes read:
// per axis the flag bytes and a compacted list of the flagged faces (FaceBox
// indices), and the cells next to a flagged face (one byte per cell, and a
// compacted list of interior indices (i ny + j) nz + k).  Counts on the device.
struct GateLists {
    const unsigned* face_list[3];
    const unsigned* face_count;  // [3]
    const unsigned* cell_list;
    const unsigned* cell_count;
    const unsigned char* touched;
    const unsigned char* mask[3];
};

// one fused SSP-RK3 stage (ns_fused.cu)
struct FusedArgs {
    const double* Uin;
    double* U0;
    double* Uout;
    Box b;
    Consts c;
    int conv_dims;   // 0 (no convection), 2 or 3
    int visc_h;      // half width of the CD stencil, 0 without diffusion
    bool fp32, chr, borges, last;
    bool phys;                        // physical semantics (local LF speed, textbook eigensystem,
                                      // 3D viscous terms, multi-dimensional CFL)
    double m1, m2, mc;
    const unsigned long long* slot;   // CFL minimum of this step
    unsigned long long* slot_next;    // last stage: CFL minimum of the next step
    double* clock;                    // first stage: [last dt, accumulated time]
    int sms;                          // multiprocessors of the device
    const unsigned char* skip;        // last stage: cells (interior order) whose next-step start a
                                      // correction pass forms instead (nullable)
};
cudaError_t launch_stage_fused(const FusedArgs& a, cudaStream_t s);
// the learned sensor's correction of a fused FP32 stage (ns_gate.cu); F: per-axis
// float face arrays for the flagged faces' flux differences
cudaError_t gate_correct(const FusedArgs& a, const GateLists& L, void* const F[3], const FaceBox fb[3], int sms,
                         cudaStream_t s);

cudaError_t launch_fma_probe(bool fp64, int blocks, int iters, void* sink, cudaStream_t s);

// A range of x-planes [lo, lo + n) for the launchers that take one (n < 0: all
// planes).  The cell kernels (step begin, prim, fill, layout transposes) count
// halo'd planes (0 .. nx+5); the sweeps and marches of a stage count interior
// planes (0 .. nx-1).
struct Planes {
    int lo = 0, n = -1;
};
// cells per thread of a march over n cells with `blocks` blocks across, of which
// `resident` fit the device at once; a segment costs `extra` cells besides its own
int march_length(int n, long long blocks, int resident, double extra, int longest);

void launch_step_begin(bool from_u, bool phys, double* W, double* U, double* U0, const Box& b,
                       const Consts& c, unsigned long long* slot, cudaStream_t s, Planes pl = Planes());
void launch_prim_all(double* W, const double* U, const Box& b, const Consts& c, cudaStream_t s,
                     Planes pl = Planes());
void launch_cons_all(const double* W, double* U, const Box& b, const Consts& c, cudaStream_t s);
void launch_min_dt(bool phys, const double* W, const Box& b, const Consts& c, unsigned long long* slot,
                   cudaStream_t s);
// U's face halos from its interior, then W = prim(U) on every cell (operator calls,
// and steps without convection or in FP32)
void launch_fill_prim(double* W, double* U, const Box& b, const Consts& c, cudaStream_t s);
// W (and, phys, its two further planes) of an FP64 stage from the stage's input U, on
// every cell (of planes pl) or on the ghost cells alone
void launch_fill_w(bool phys, double* W, const double* U, const Box& b, const Consts& c, cudaStream_t s,
                   Planes pl = Planes());
void launch_fill_shell(bool phys, double* W, const double* U, const Box& b, const Consts& c, cudaStream_t s);
// U's face halos after an FP64 step, from the third stage's input Us
void launch_fill_uhalo(double* U, const double* Us, const Box& b, const Consts& c, cudaStream_t s);
// face fluxes of an operator call along the first `dims` axes, from W and U; returns
// the kernels launched
int launch_faces(bool chr, bool borges, bool phys, bool fp32, int dims, const double* W, const double* U, const Box& b,
                 const Consts& c, void* const F[3], const FaceBox fb[3], cudaStream_t s);
// the y- (dir 1) or z-faces (dir 2) of an FP64 stage, from W (and the sound speed plane) alone
void launch_step_faces(int dir, bool chr, bool borges, bool phys, const double* W, const Box& b, const Consts& c,
                       double* F, const FaceBox& fb, cudaStream_t s, Planes pl = Planes());
// largest ulp distance between div_pos_nr and the IEEE quotient over n draws
cudaError_t launch_div_check(long long n, unsigned long long seed, unsigned long long* max_ulp, cudaStream_t s);
// one block waits (bounded) on an mbarrier phase nothing completes; out[0] = 1
// if the wait gave up, 0 if it claimed completion
cudaError_t launch_wait_probe(unsigned polls, unsigned long long* out, cudaStream_t s);
void launch_update(const UpdateArgs& a, cudaStream_t s);
// x-faces + update of an FP64 stage in one march
void launch_xmarch(bool chr, bool borges, bool phys, const XMarchArgs& a, cudaStream_t s, Planes pl = Planes());
// TMA tensor map of a stage's W (of 5 or 7 planes) for the CD-2 viscous march (a
// CUtensorMap: 128 bytes, 64-byte aligned); false if none can be made
struct VTmaMap {
    alignas(64) unsigned char map[128];
    const double* W = nullptr;
};
bool visc_tma_encode(VTmaMap* m, const double* W, const Box& b, int planes);
// viscous terms (components 1..4) of every interior cell into V (as XMarchArgs's) from
// a stage's W; half-width h = 1, 2, 3 of the centered scheme; m: W's map (nullable);
// *err receives 1 if a wait ran out
void launch_viscous(int h, bool phys, const VTmaMap* m, const double* W, const Box& b, const Consts& c, double* V,
                    long long vs, unsigned long long* err, int sms, cudaStream_t s, Planes pl = Planes());
// slab halo exchange: pack the outer interior planes of a side / unpack into its ghost planes
void launch_slab_pack(const double* U, const Box& b, int side, double* buf, cudaStream_t s);
void launch_slab_unpack(double* U, const Box& b, int side, const double* buf, cudaStream_t s);
void launch_aos_to_soa(const double* A, double* S, const Box& b, cudaStream_t s, Planes pl = Planes());
void launch_soa_to_aos(const double* S, double* A, const Box& b, cudaStream_t s, Planes pl = Planes());
// interior cells of A (W if prim, else U) that are non-finite or have rho <= 0 or p <= 0,
// added to *count
void launch_check_state(const double* A, bool prim, const Box& b, const Consts& c,
                        unsigned long long* count, cudaStream_t s);
void launch_diagnostics(const double* U, const Box& b, const Consts& c, double* acc, cudaStream_t s);

}  // namespace nsb
