// geometry.cu -- the element geometry table: B^-1 and det B of every element,
// formed once per mesh.
//
// The FP32 element kernels all start from B^-1 (each entry the FP64 value
// rounded once to FP32) and det B of their element (geometry_fp64).  A handle's
// mesh never changes, so the table is part of its mesh layout like the slot
// maps: 40 bytes per element, structure of arrays, read back coalesced.
// Forming it in every element kernel cost about 55 FP64 operations per element
// on a pipe that takes 20 cycles per warp instruction, and twelve gathered
// coordinates.
#include "kernels.cuh"

namespace fedd {
namespace {

__global__ void __launch_bounds__(128) k_geometry(const double *__restrict__ xyz, const int32_t *__restrict__ conn,
                                                  int64_t ne, float *__restrict__ geo) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= ne) return;
    float Bi[9];
    const float det = d2f_rn(geometry_fp64(xyz, conn[e], conn[ne + e], conn[2 * ne + e], conn[3 * ne + e], Bi));
#pragma unroll
    for (int k = 0; k < 9; k++) geo[k * ne + e] = Bi[k];
    geo[9 * ne + e] = det;
}

}  // namespace

void launch_geometry(const double *xyz, const int32_t *conn, int64_t ne, float *geo, cudaStream_t s) {
    if (ne == 0) return;
    k_geometry<<<ceil_div(ne, 128), 128, 0, s>>>(xyz, conn, ne, geo);
    FEDD_CUDA(cudaGetLastError());
}

}  // namespace fedd
