// Shape choice and launch of the resident 2D kernels (fdtd2d_resident_kernel.cuh).
#include "fdtd2d_resident_kernel.cuh"

cudaError_t res2d_launch_ez_plain(int shape, const Res2DJob &job, size_t smem, cudaStream_t stream);
cudaError_t res2d_launch_ez_gen(int shape, const Res2DJob &job, size_t smem, cudaStream_t stream);
cudaError_t res2d_launch_hz_plain(int shape, const Res2DJob &job, size_t smem, cudaStream_t stream);
cudaError_t res2d_launch_hz_gen(int shape, const Res2DJob &job, size_t smem, cudaStream_t stream);

int res2d_shape(int ny, int max_rows, bool blocked_takes_it) {
    for (int s = 0; s < RES_N_SHAPES; ++s)
        if (!(blocked_takes_it && RES_SHAPES[s].blocked_is_faster) && max_rows <= RES_SHAPES[s].rt &&
            (ny + RES_SHAPES[s].c - 1) / RES_SHAPES[s].c <= RES_SHAPES[s].nt)
            return s;
    return -1;
}

int res2d_columns(int shape) { return RES_SHAPES[shape].c; }

size_t res2d_smem_bytes(const Res2DJob &job, int i0, int i1, int layer_e, int layer_h, int shape) {
    return sizeof(Res2DJob) + (size_t)(i1 - i0 + 2) * sizeof(ResRow) +
           (size_t)job.n_poles * sizeof(ResPoleRows) +
           res_strip_floats(job, i0, i1, layer_e, layer_h, RES_SHAPES[shape].c, RES_SHAPES[shape].rt) * sizeof(float);
}

size_t res2d_mail_words(int hz, int ny, int n_cta) {
    return (size_t)n_cta * 2 * res_mail_rows(hz) * (size_t)res_pitch(ny);
}

bool res2d_general(const Res2DJob &job) {
    // a uniform da other than 1 has no array, but scales H all the same: the general kernels multiply by it
    return job.ca || job.da || job.da_u != 1.0f || job.n_maps || job.n_poles || job.n_tfsf;
}

cudaError_t res2d_launch(int shape, const Res2DJob &job, size_t smem, cudaStream_t stream) {
    const bool gen = res2d_general(job);
    if (job.hz) return gen ? res2d_launch_hz_gen(shape, job, smem, stream) : res2d_launch_hz_plain(shape, job, smem, stream);
    return gen ? res2d_launch_ez_gen(shape, job, smem, stream) : res2d_launch_ez_plain(shape, job, smem, stream);
}
