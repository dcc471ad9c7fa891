// The resident form of the 2D step: one cooperative launch runs a whole chunk of steps with the fields held in
// registers, for grids that fit the chip (fdtd2d_resident_kernel.cuh has the kernel and the reasons).  This header: the parameter
// block of one simulation and the launch entry points.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#define RES_MAX_LINES 16
#define RES_MAX_MONS 8
#define RES_MAX_PROBES 8
#define RES_MAX_MAPS 4
#define RES_MAX_POLES 12
#define RES_MAX_TFSF 2

struct ResLine {
    int32_t axis, position, lo, hi;   // axis 0: cells (i, position), axis 1: cells (position, j)
    const float *profile;
};

struct ResMon {
    int32_t normal_axis, position, lo, hi;
    float *stage;                     // (samples of the chunk, 2, hi - lo)
};

struct ResProbe {
    int32_t ix, iy, comp, pad;
    float *row;                       // the probe's row: value of step n at row[n - 1]
    int64_t start;                    // first recorded row
};

struct ResMap {
    int32_t x0, y0, ds, mx, my, nf;
    const float *ph_e, *ph_h;         // this chunk's phases (samples, nf, 2): E-time, and H_z-time (H_z engines)
    float *acc;
};

struct ResPole {
    int32_t kind, comp, i0, i1, j0, j1;
    float damping, restoring;
    const float *drive;
    float *a, *b;
};

struct ResTfsf {
    int32_t x0, x1, y0, y1, aux_x0, aux_n, source_index, pad;
    float coef_h[4], coef_e[4], mur_lo, mur_hi;
    float *aux_e, *aux_h;             // the incident line: E_z and H_y (E_z engines), E_y and H_z (H_z engines)
    const float *aux_coef_h, *aux_coef_e;
    const float *values;              // this chunk's soft-source values, one per step
};

// One simulation.  f / a / b: E_z, H_x, H_y of an E_z engine; H_z, E_x, E_y of an H_z engine (updated in place).
struct __align__(16) Res2DJob {
    int32_t hz, nx, ny, px, py, npml, cpml_mask, n_cta;
    float *f, *a, *b;
    const float *ca, *cb, *ca_y, *cb_y;   // E_z: ca, cb of E_z; H_z: of E_x and E_y.  ca NULL: 1
    const float *da, *db;                 // NULL: the uniform values
    float da_u, db_u;
    const float *inv_dx_e, *inv_dx_h, *inv_dy_e, *inv_dy_h;
    const float *cpml_rows[4];            // b_e, a_e, inv_e, b_h, a_h, inv_h (npml each)
    float *psi_e[4], *psi_h[4];
    const int32_t *row_start;             // n_cta + 1 first rows of the blocks' strips
    uint64_t *mail;                       // boundary rows of the strips (res2d_mail_words)
    uint32_t *arrived;                    // blocks that ever finished loading their state, this launch's ending at `arrivals`
    uint32_t epoch;                       // number of this chunk's first boundary rows
    uint32_t arrivals;
    int64_t n_steps, n0, m;               // steps of this chunk, steps before it, DFT sample interval
    int64_t q_first;                      // first sample of the chunk (staging slot 0)
    int64_t q_table;                      // first sample of the phase tables
    const float *line_values;             // row l: this chunk's values of line l, rows values_stride apart
    int64_t values_stride;
    int32_t n_lines, n_mons, n_probes, n_maps, n_poles, n_tfsf;
    int32_t n_drude, pad1;                // Drude poles
    float inv_dt;
    ResLine lines[RES_MAX_LINES];
    ResMon mons[RES_MAX_MONS];
    ResProbe probes[RES_MAX_PROBES];
    ResMap maps[RES_MAX_MAPS];
    ResPole poles[RES_MAX_POLES];         // Drude poles first, each kind in add order
    ResTfsf tfsf[RES_MAX_TFSF];
    float *rec;                           // E_z engines: E_z of a cell box after every step (step, box), or NULL
    int32_t rec_i0, rec_i1, rec_j0, rec_j1;
    int32_t *err;
    int64_t stall_probe_ns;               // test hook of the bounded waits (0: off)
};
static_assert(sizeof(Res2DJob) % 16 == 0, "Res2DJob lies in front of 16-byte vectors in shared memory");

// Kernel shape for strips of max_rows rows of ny columns, -1 when they fit none (or, for a run that the blocked kernels
// take too, none that is faster than those).
int res2d_shape(int ny, int max_rows, bool blocked_takes_it);
// Columns a thread of a shape.
int res2d_columns(int shape);
// Shared memory of the block of rows [i0, i1), layer_e / layer_h of them in the E / H kind's x-side CPML.
size_t res2d_smem_bytes(const Res2DJob &job, int i0, int i1, int layer_e, int layer_h, int shape);
// 64-bit words of a simulation's mail.
size_t res2d_mail_words(int hz, int ny, int n_cta);
// Whether the job runs in the kernels with conductivity, magnetic cells, maps, poles and plane-wave boxes.
bool res2d_general(const Res2DJob &job);
// Launches one simulation (n_cta blocks of `smem` bytes, the largest strip's).
cudaError_t res2d_launch(int shape, const Res2DJob &job, size_t smem, cudaStream_t stream);
