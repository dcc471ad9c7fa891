// The resident kernels of the E_z engine, with conductivity, magnetic cells, maps, poles and plane-wave boxes (a file of their own to compile beside the others).
#include "fdtd2d_resident_kernel.cuh"

cudaError_t res2d_launch_ez_gen(int shape, const Res2DJob &job, size_t smem, cudaStream_t stream) {
    return res_launch_any<false, true>(shape, job, smem, stream);
}
