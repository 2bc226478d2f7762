// ns_tma.cu -- tensor maps of W for the Tensor Memory Accelerator (the viscous
// march's planes, ns_kernels.cu) and the self-test of the bounded device waits.
//
// Boxes: 4D (z, y, x, field) of the halo'd SoA array.  TMA wants the innermost
// start x 8 bytes and the box's innermost extent x 8 bytes to be multiples of 16.
// A box that reaches past the array (the last z tile of an nz that is not a
// multiple of 32) is zero-filled by the TMA unit and only feeds cells that do
// not exist.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstdint>

#include "ns_common.cuh"
#include "ns_kernels.h"
#include "ns_tcgen05.cuh"
#include "ns_tma.cuh"

namespace nsb {

// The bounded wait of every TMA and tensor-core kernel, on a phase that no
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

bool w_tma_encode(WTmaMaps* m, const double* W, const Box& b, int planes) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = encode_fn();
    if (!enc) return false;
    // dimensions innermost first: z (padded row), y, x, field
    const cuuint64_t dims[4] = {(cuuint64_t)b.NZp, (cuuint64_t)b.NY, (cuuint64_t)b.NX, (cuuint64_t)planes};
    const cuuint64_t strides[3] = {(cuuint64_t)b.NZp * 8, (cuuint64_t)b.NY * b.NZp * 8, (cuuint64_t)b.fstride * 8};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const cuuint32_t boxv1[4] = {ViscTile<1>::BZ, ViscTile<1>::BY, 1, 5};
    const cuuint32_t boxv2[4] = {ViscTile<2>::BZ, ViscTile<2>::BY, 1, 5};
    const cuuint32_t boxv3[4] = {ViscTile<3>::BZ, ViscTile<3>::BY, 1, 5};
    const cuuint32_t* boxes[3] = {boxv1, boxv2, boxv3};
    for (int d = 0; d < 3; d++) {
        CUresult r = enc(reinterpret_cast<CUtensorMap*>(m->map[d]), CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4,
                         const_cast<double*>(W), dims, strides, boxes[d], estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return false;
    }
    m->W = W;
    return true;
}

}  // namespace nsb
