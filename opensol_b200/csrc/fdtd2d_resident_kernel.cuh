// Resident 2D step: one cooperative launch advances a simulation by a whole chunk of Yee steps.
//
// The grid is cut into strips of rows, one block each.  A thread owns C adjacent columns of its block's strip and keeps
// their three fields in registers for the whole chunk (RT rows at most, unrolled); material words, CPML psi and pole
// state sit in shared memory.  A step has two phases with a block barrier after each (E_z: H_x and H_y, then E_z; H_z:
// H_z, then E_x and E_y): vertical neighbours are the thread's own registers, horizontal ones come by warp shuffle and,
// between warps, through small shared arrays of the warps' edge columns.  Strips exchange one boundary row per
// direction and step through global memory ("mail"): each word carries a float and the number of the step that
// produced it, so a reader polls the word itself and needs no fence, flag or grid barrier.  The one value of the
// neighbour's new half step a strip needs (H_y of the row above for E_z, H_z of the row below for H_z) is computed
// again from the mailed old values, so one exchange per step is enough.  Two slots per word are enough: a strip can mail
// step s + 2 only after it received its neighbour's step s + 1, which the neighbour mailed after reading step s.
//
// Every cell is evaluated in open_sol's order on the same operands as the other forms (fdtd_ez_2d_kernels.py:23-122,
// fdtd_hz_2d_kernels.py:28-174, boundaries.py:27-37), so the results are the same bits.  Differences and products run
// packed (two columns an instruction); every add of a product is scalar, since the code generator would merge a packed
// multiply into a packed add.  Sources, plane-wave boxes, poles, probes, field maps and the flux lines' samples are
// handled inside the step; the flux lines' running sums are folded once per chunk from the staged samples.
//
// What bounds it: small strips (270 x 120 cells) wait for the mail, about 1 us from store to poll across L2, plus two
// block barriers (6.6 % of the issue slots used); large ones (1075 x 1075) the latency of the row updates at the 17 warps a
// multiprocessor that the registers leave (80 instructions per row of two columns and phase, 44 % of the issue slots, a fifth
// of a warp's time at the barriers).  Measured on a B200, device time per step against the launches per step before it: 270 x
// 120 cells 2.2 us (15), 441 x 393 lossy 3.6 us (20), 1075 x 1075 5.7 us (17), 930 x 730 H_z 5.2 us (18).  Fields in shared memory instead of registers (one cell at a time) took 18 us at
// 1075 x 1075; so did polling one mailed word after the other (an L2 round trip each).
//
// GEN adds what plain lossless runs do not need: ca / da / db words, field maps, poles, plane-wave boxes.
//
// Every poll is bounded by %globaltimer: 2 s for a neighbour's mail, 120 s for all blocks to be placed at the start (other
// streams' kernels may hold multiprocessors until then).  When it runs out the block sets the engine's error flag and
// leaves, and the others follow when they see the flag or their own bound.
#pragma once

#include "fdtd2d_resident.cuh"
#include "mbarrier.cuh"

enum { RSX_LO = 0, RSX_HI = 1, RSY_LO = 2, RSY_HI = 3 };
enum { RF_MAP = 1, RF_TFSF = 2, RF_EDGE = 4 };

// Facts of one row: index r + 1 of the table for strip row r; 0: the row above the strip, R + 1: the row below it.
struct __align__(16) ResRow {
    float ixe, ixh;                       // 1 / spacing of the centre and hi face
    int32_t xe, xh;                       // x-side CPML: place of the row's psi among the strip's (-1: none)
    float b_e, a_e, i_e, unused_e;        // and its recursion
    float b_h, a_h, i_h, unused_h;
    int32_t i, flags;                     // physical row, RF_* bits
    uint32_t poles;                       // poles on the row
    int32_t pad;
};
static_assert(sizeof(ResRow) % 16 == 0, "the row table is followed by vectors");

__host__ __device__ static inline int res_pitch(int ny) { return (ny + 3) & ~3; }
__host__ __device__ static inline int res_coef_arrays(const Res2DJob &p) {
    return (p.hz ? 2 : 1) + (p.ca ? (p.hz ? 2 : 1) : 0) + (p.da ? 2 : 0);
}
__host__ __device__ static inline size_t res_mail_rows(int hz) { return hz ? 3 : 2; }

// A pole's rows in shared memory: the columns of the threads (c each) its box reaches, drive and state (2 or 3 arrays).
__host__ __device__ static inline int res_pole_width(const ResPole &q, int c) {
    return ((q.j1 + c - 1) / c - q.j0 / c) * c;
}
__host__ __device__ static inline int res_pole_floats(const ResPole &q, int i0, int i1, int c) {
    const int a = q.i0 > i0 ? q.i0 : i0, b = q.i1 < i1 ? q.i1 : i1;
    return b > a ? (b - a) * res_pole_width(q, c) * (q.kind == 0 ? 2 : 3) : 0;
}

__device__ __forceinline__ float2 rs_sub(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ float2 rs_mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 rs_add_p(float2 a, float2 b) {
    return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y));
}
__device__ __forceinline__ float2 rs_sub_p(float2 a, float2 b) {
    return make_float2(__fadd_rn(a.x, -b.x), __fadd_rn(a.y, -b.y));
}
__device__ __forceinline__ float2 rs_pair(float v) { return make_float2(v, v); }

// Component c of a thread's columns (unrolled selects keep the arrays in registers).
template <int H>
__device__ __forceinline__ float rs_get(const float2 (&v)[H], int c) {
    float out = v[0].x;
#pragma unroll
    for (int k = 0; k < 2 * H; ++k)
        if (k == c) out = (k & 1) ? v[k >> 1].y : v[k >> 1].x;
    return out;
}
template <int H>
__device__ __forceinline__ void rs_set(float2 (&v)[H], int c, float x) {
#pragma unroll
    for (int k = 0; k < 2 * H; ++k)
        if (k == c) {
            if (k & 1) v[k >> 1].y = x;
            else v[k >> 1].x = x;
        }
}

__device__ __forceinline__ void res_send(uint64_t *at, float v, uint32_t epoch) {
    const uint64_t w = ((uint64_t)epoch << 32) | (uint64_t)__float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(at), "l"(w) : "memory");
}
__device__ __forceinline__ uint64_t res_peek(const uint64_t *at) {
    uint64_t w;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(at) : "memory");
    return w;
}
#define RES_START_WAIT_NS 120000000000ull
// Whether a poll that started at t0 gives up: its time is over, or another thread or block gave up (then *dead is set).
static __device__ __noinline__ bool res_give_up(uint64_t t0, uint64_t wait_ns, int *err, int *dead) {
    if (*(volatile int *)dead) return true;
    if (!*(volatile int *)err && tb_globaltimer() - t0 <= wait_ns) return false;
    atomicExch(err, 1);
    *(volatile int *)dead = 1;
    return true;
}

// This block has loaded its state, and: have all.
__device__ __forceinline__ void res_arrive(uint32_t *arrived) {
    __threadfence();
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrived) : "memory");
}
static __device__ __noinline__ void res_wait_all(const uint32_t *arrived, uint32_t arrivals, int *err, int *dead) {
    const uint64_t t0 = tb_globaltimer();
    for (int tries = 0;; ++tries) {
        uint32_t n;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(arrived) : "memory");
        if ((int32_t)(n - arrivals) >= 0) return;
        if ((tries & 63) == 63 && res_give_up(t0, RES_START_WAIT_NS, err, dead)) return;
    }
}

__device__ __forceinline__ float res_wrap_hi(float w) { return w * 1.0f + w * 0.0f; }
__device__ __forceinline__ float res_wrap_lo(float w) { return w * 1.0f - w * 0.0f; }

// CPML side and slab row of H (hi-face) / E (centre) row r of an axis of n cells (lo: the axis's lo side).
__device__ __forceinline__ int res_h_side(int lo, int mask, int r, int n, int npml, int &k) {
    k = r;
    if (((mask >> lo) & 1) && r < npml) return lo;
    k = r - (n - npml - 1);
    if (((mask >> (lo + 1)) & 1) && k >= 0 && k < npml) return lo + 1;
    return -1;
}
__device__ __forceinline__ int res_e_side(int lo, int mask, int r, int n, int npml, int &k) {
    k = r - 1;
    if (((mask >> lo) & 1) && k >= 0 && k < npml) return lo;
    k = r - (n - npml - 1);
    if (((mask >> (lo + 1)) & 1) && k >= 0 && k < npml) return lo + 1;
    return -1;
}

// One term of a field map's running sum (complex64 arithmetic, as ez2d_dft_map_kernel).
__device__ __forceinline__ void res_map_add(float *acc, const float *ph, float v) {
    const float pr = __ldg(ph), pi = __ldg(ph + 1), zero = 0.0f;
    float2 s = *reinterpret_cast<float2 *>(acc);
    s.x = s.x + (pr * v - pi * zero);
    s.y = s.y + (pr * zero + pi * v);
    *reinterpret_cast<float2 *>(acc) = s;
}
// Sample index of (i, j) in a map, -1 when it is not sampled.
__device__ __forceinline__ int64_t res_map_index(const ResMap &d, int i, int j) {
    const int di = i - d.x0, dj = j - d.y0;
    if (di < 0 || dj < 0 || di % d.ds || dj % d.ds) return -1;
    const int x = di / d.ds, y = dj / d.ds;
    return x < d.mx && y < d.my ? (int64_t)x * d.my + y : -1;
}
static __device__ __noinline__ void res_maps_ez(const Res2DJob &p, int i, int j, int64_t n, float v) {
    for (int k = 0; k < p.n_maps; ++k) {
        const ResMap &d = p.maps[k];
        const int64_t c = res_map_index(d, i, j);
        if (c < 0) continue;
        const float *ph = d.ph_e + (size_t)(n / p.m - p.q_table) * d.nf * 2;
        for (int f = 0; f < d.nf; ++f) res_map_add(d.acc + 2 * ((size_t)f * d.mx * d.my + c), ph + 2 * f, v);
    }
}
// H_z maps (monitors.py:296-322): H_z, and E_x / E_y collocated to the cell centre from their lo partners.
static __device__ __noinline__ void res_maps_hz(const Res2DJob &p, int i, int j, int64_t n, float hz, float ex,
                                                float ex_lo, float ey, float ey_lo) {
    const float half = 0.5f;
    for (int k = 0; k < p.n_maps; ++k) {
        const ResMap &d = p.maps[k];
        const int64_t c = res_map_index(d, i, j);
        if (c < 0) continue;
        const size_t s = (size_t)(n / p.m - p.q_table) * d.nf * 2, per_f = (size_t)d.mx * d.my, total = per_f * d.nf;
        for (int f = 0; f < d.nf; ++f) {
            const size_t at = (size_t)f * per_f + c;
            res_map_add(d.acc + 2 * at, d.ph_h + s + 2 * f, hz);
            res_map_add(d.acc + 2 * (total + at), d.ph_e + s + 2 * f, half * (ex + ex_lo));
            res_map_add(d.acc + 2 * (2 * total + at), d.ph_e + s + 2 * f, half * (ey + ey_lo));
        }
    }
}

extern __shared__ __align__(16) unsigned char res_smem[];   // the block's shared memory (functions that are not inlined
                                                            // address it by offset, so their accesses stay shared ones)

// Plane-wave boxes: each box's incident line in shared memory is four arrays of aux_n floats at `at`: E cells, H cells
// and their coefficients.  The corrections of the boxes' x sides on a thread's columns j0 .. j0 + C - 1 of row i (the y
// sides are ResStrip::tfsf_ab's): `v` is H_y after the H update or E_z after the E update of an E_z engine, H_z after
// its update or E_y after the E update of an H_z engine.
template <int C>
static __device__ __noinline__ float4 res_tfsf_row(const Res2DJob &p, int at, bool e_phase, int i, int j0, float4 in) {
    float v[4] = {in.x, in.y, in.z, in.w};
#pragma unroll 1
    for (int k = 0; k < p.n_tfsf; ++k) {
        const ResTfsf &t = p.tfsf[k];
        const float *e = reinterpret_cast<const float *>(res_smem) + at, *h = e + t.aux_n;
        const int last = t.aux_x0 + (t.x1 - 1 - t.x0);
        float lo = 0.0f, hi = 0.0f;   // signed terms of the two sides
        bool on_lo, on_hi;
        if (!p.hz && !e_phase) {
            on_lo = i == t.x0 - 1, lo = -(t.coef_h[0] * e[t.aux_x0]);
            on_hi = i == t.x1 - 1, hi = t.coef_h[1] * e[last];
        } else if (!p.hz) {
            on_lo = i == t.x0, lo = -(t.coef_e[0] * h[t.aux_x0 - 1]);
            on_hi = i == t.x1 - 1, hi = t.coef_e[1] * h[last];
        } else if (!e_phase) {
            on_lo = i == t.x0, lo = t.coef_h[0] * e[t.aux_x0 - 1];
            on_hi = i == t.x1 - 1, hi = -(t.coef_h[1] * e[last]);
        } else {
            on_lo = i == t.x0 - 1, lo = t.coef_e[0] * h[t.aux_x0];
            on_hi = i == t.x1 - 1, hi = -(t.coef_e[1] * h[last]);
        }
#pragma unroll
        for (int c = 0; c < C; ++c) {
            if (j0 + c < t.y0 || j0 + c >= t.y1) continue;
            if (on_lo) v[c] = v[c] + lo;
            if (on_hi) v[c] = v[c] + hi;
        }
        at += 4 * t.aux_n;
    }
    return make_float4(v[0], v[1], v[2], v[3]);
}
// The incident lines' half steps, by every block for itself (first phase: H from E, second: E from H, the soft source
// and the Mur ends).  An H_z engine's H cells are shifted by one: H_z[k] from E_y[k] - E_y[k - 1], k >= 1.
static __device__ __noinline__ void res_aux_h(const Res2DJob &p, int at, int tid, int nt) {
    for (int k = 0; k < p.n_tfsf; ++k) {
        const int n = p.tfsf[k].aux_n;
        float *e = reinterpret_cast<float *>(res_smem) + at, *h = e + n + (p.hz ? 1 : 0);
        const float *coef = e + 2 * n;
        for (int a = tid; a < n - 1; a += nt) h[a] = h[a] + coef[a] * (e[a + 1] - e[a]);
        at += 4 * n;
    }
}
static __device__ __noinline__ void res_aux_e(const Res2DJob &p, int at, int64_t k_step, int tid, int nt) {
    for (int k = 0; k < p.n_tfsf; ++k) {
        const ResTfsf &t = p.tfsf[k];
        const int n = t.aux_n;
        float *e = reinterpret_cast<float *>(res_smem) + at;
        const float *h = e + n + (p.hz ? 1 : 0), *coef = e + 3 * n;
        for (int a = 1 + tid; a < n - 1; a += nt) {
            const float old = e[a];
            float v = old + coef[a] * (h[a] - h[a - 1]);
            if (a == t.source_index) v = v + __ldg(t.values + k_step);
            e[a] = v;
            if (a == 1) e[0] = old + t.mur_lo * (v - e[0]);
            if (a == n - 2) e[n - 1] = old + t.mur_hi * (v - e[n - 1]);
        }
        at += 4 * n;
    }
}

// A pole's rows in the strip (floats from res_smem): drive, a, and b of a Lorentz pole, n floats apart, rows of w floats
// from column c0; strip rows from `first`; the box's columns [j0, j1).
struct __align__(16) ResPoleRows {
    int32_t at, n, first, w;
    int32_t c0, j0, j1, kind;
    float damping, restoring;
    int32_t comp, pad;
};
// Poles `mask` of the strip's table on a thread's columns of strip row r: the update from the fields before the step
// (fdtd_ez_2d.py:318-345): e0 is E_z, or E_x and e1 E_y.  The table lists Drude poles first, each kind in add order.
template <int C>
static __device__ __noinline__ void res_pole_update(int tab, uint32_t mask, int r, int j0, float4 e0, float4 e1) {
#pragma unroll 1
    for (; mask; mask &= mask - 1) {
        const ResPoleRows q = reinterpret_cast<const ResPoleRows *>(res_smem + tab)[__ffs(mask) - 1];
        const float4 e4 = q.comp ? e1 : e0;
        const float e[4] = {e4.x, e4.y, e4.z, e4.w};
        float2 *drive = reinterpret_cast<float2 *>(reinterpret_cast<float *>(res_smem) + q.at + (r - q.first) * q.w +
                                                   (j0 - q.c0));
        float2 *a = drive + q.n / 2, *b = a + q.n / 2;
        float2 d2[C / 2], a2[C / 2], b2[C / 2];
#pragma unroll
        for (int k = 0; k < C / 2; ++k) {
            d2[k] = drive[k], a2[k] = a[k];
            if (q.kind) b2[k] = b[k];
        }
#pragma unroll
        for (int c = 0; c < C; ++c) {
            if (j0 + c < q.j0 || j0 + c >= q.j1) continue;
            const float dr = (c & 1) ? d2[c >> 1].y : d2[c >> 1].x;
            float &av = (c & 1) ? a2[c >> 1].y : a2[c >> 1].x;
            if (q.kind == 0) {
                av = av + (q.damping * av + dr * e[c]);
            } else {
                float &bv = (c & 1) ? b2[c >> 1].y : b2[c >> 1].x;
                bv = bv + (q.damping * bv - q.restoring * av + dr * e[c]);
                av = av + bv;
            }
        }
#pragma unroll
        for (int k = 0; k < C / 2; ++k) {
            a[k] = a2[k];
            if (q.kind) b[k] = b2[k];
        }
    }
}
// Correction of the updated field of component comp (E_z: 0).  E_z: the Drude total (the J itself when there is one
// Drude pole, else summed from 0 in add order), then each Lorentz pole (fdtd_ez_2d.py:347-358; cells in no Drude box keep
// v, which is v - cb * 0).  H_z: Drude sets, then Lorentz sets (fdtd_hz_2d.py:311-325).
template <int C>
static __device__ __noinline__ float4 res_pole_correct(int tab, uint32_t mask, bool hz, int comp, bool one_drude,
                                                       float inv_dt, int r, int j0, float4 v4, float4 cb4) {
    float v[4] = {v4.x, v4.y, v4.z, v4.w}, total[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    const float cb[4] = {cb4.x, cb4.y, cb4.z, cb4.w};
    bool sum = !hz;   // the Drude total is still being summed
#pragma unroll 1
    for (;; mask &= mask - 1) {
        const ResPoleRows q = reinterpret_cast<const ResPoleRows *>(res_smem + tab)[mask ? __ffs(mask) - 1 : 0];
        if (sum && (!mask || q.kind == 1)) {
#pragma unroll
            for (int c = 0; c < C; ++c) v[c] = v[c] - cb[c] * total[c];
            sum = false;
        }
        if (!mask) break;
        if (q.comp != comp) continue;
        const float2 *s2 = reinterpret_cast<const float2 *>(reinterpret_cast<const float *>(res_smem) + q.at +
                                                            (q.kind == 0 ? q.n : 2 * q.n) + (r - q.first) * q.w +
                                                            (j0 - q.c0));
        const float scale = q.kind == 0 ? 1.0f : inv_dt;
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const float s = (c & 1) ? s2[c >> 1].y : s2[c >> 1].x;
            if (j0 + c < q.j0 || j0 + c >= q.j1) continue;
            if (sum) total[c] = one_drude ? s : total[c] + s;
            else v[c] = v[c] - cb[c] * scale * s;
        }
    }
    return make_float4(v[0], v[1], v[2], v[3]);
}

// A thread's columns as one value (C = 2: the first two).
template <int H>
__device__ __forceinline__ float4 res_from(const float2 (&v)[H]) {
    return make_float4(v[0].x, v[0].y, H > 1 ? v[H - 1].x : 0.0f, H > 1 ? v[H - 1].y : 0.0f);
}
template <int H>
__device__ __forceinline__ void res_to(float2 (&v)[H], float4 x) {
    v[0] = make_float2(x.x, x.y);
    if (H > 1) v[H - 1] = make_float2(x.z, x.w);
}

template <bool HZ, bool GEN, int C, int RT>
struct ResStrip {
    static constexpr int H = C / 2, COLS = C;
    const Res2DJob &p;
    // block
    int i0, R, P, ny, mail_p;      // P: row pitch in shared memory (every thread's columns), mail_p: in the mail
    bool has_up, has_dn, wrap_up, wrap_dn, py, odd;   // odd: column ny - 1 is not the last of its thread's
    const uint64_t *from_up, *from_dn;
    uint64_t *to_me;
    // thread
    int lane, warp, j0, cl;        // cl: component of column ny - 1 (-1: not this thread's)
    bool end_warp, take_lo;        // the warp of column ny - 1; the thread's right neighbour comes from `lo`
    uint32_t lines, mons, probes;  // of p.lines / p.mons / p.probes, those on this thread's cells
    bool yh, ye, edge_col;
    bool records;                  // the thread's columns reach the recorded box
    uint32_t pole_mask;            // poles on the thread's columns
    int y_at;                      // place of the thread's columns in the rows of y-side psi and recursion
    float db_u, da_u;
    float2 iye[H], iyh[H];
    // shared memory
    ResRow *rows;
    // [RT][34] per warp edge: lo[w]: first column of warp w (behind the last warp: of column 0, wrapped); hi[w]: last
    // column of warp w - 1 (w = 0: of column ny - 1, wrapped, or 0); last: column ny - 1
    float *lo, *hi, *last;
    float *cx, *cy, *cax, *cay, *da, *db;   // coefficient rows (R, P)
    float *xe, *xh, *gx;           // x-side psi rows; the recomputed row's
    float *yeq, *yhq, *gy;         // y-side psi (R, Y: the layer threads' columns); the recomputed row's
    float *yrec;                   // y-side recursion: b, a, inv of the E kind, then of the H kind (Y each)
    int Y;
    int aux, pole_tab;             // incident lines (floats from res_smem), the pole table (bytes)
    float *pole;
    int *dead;
    // fields
    float2 f[RT][H], a[RT][H], b[RT][H];
    float2 g[H];                   // the recomputed row: H_y above (E_z), H_z below (H_z)

    __device__ __forceinline__ ResStrip(const Res2DJob &job) : p(job) {}

    // The mailed values of N rows at the thread's columns (at[n] NULL: none), and one more word (extra, when extra_at).
    // All words are loaded at once and again until every one has arrived, so a wait costs one L2 round trip and not
    // one per word.
    template <int N>
    __device__ __forceinline__ void receive(float2 (&v)[N][H], const uint64_t *const (&at)[N], float &extra,
                                            const uint64_t *extra_at, uint32_t epoch) {
        const uint64_t none = (uint64_t)epoch << 32;
        uint64_t t0 = 0;
        for (int tries = 0;; ++tries) {
            uint64_t w[N][C], x = none;
#pragma unroll
            for (int n = 0; n < N; ++n)
#pragma unroll
                for (int c = 0; c < C; ++c) w[n][c] = at[n] && j0 + c < ny ? res_peek(at[n] + j0 + c) : none;
            if (extra_at) x = res_peek(extra_at);
            bool here = (uint32_t)(x >> 32) == epoch;
#pragma unroll
            for (int n = 0; n < N; ++n)
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    here = here && (uint32_t)(w[n][c] >> 32) == epoch;
                    if (c & 1) v[n][c >> 1].y = __uint_as_float((uint32_t)w[n][c]);
                    else v[n][c >> 1].x = __uint_as_float((uint32_t)w[n][c]);
                }
            extra = __uint_as_float((uint32_t)x);
            if (here) return;
            if (tries == 0) t0 = tb_globaltimer();
            if ((tries & 63) == 63 && res_give_up(t0, TB_WAIT_NS, p.err, dead)) return;
        }
    }
    __device__ __forceinline__ void send(uint64_t *at, const float2 (&v)[H], uint32_t epoch) {
#pragma unroll
        for (int c = 0; c < C; ++c)
            if (j0 + c < ny) res_send(at + j0 + c, (c & 1) ? v[c >> 1].y : v[c >> 1].x, epoch);
    }
    __device__ __forceinline__ size_t slot(uint32_t epoch) const {
        return (size_t)(epoch & 1) * res_mail_rows(HZ) * mail_p;
    }
    // boundary rows of the present state (E_z: E_z up and down; H_z: E_x, E_y up, E_y down)
    __device__ __forceinline__ void mail(uint32_t epoch) {
        uint64_t *m = to_me + slot(epoch);
        if (has_up) {
            send(m, HZ ? a[0] : f[0], epoch);
            if (HZ) send(m + mail_p, b[0], epoch);
        }
        if (has_dn) {
            float2 x[H];
            get(x, HZ ? b : f, R - 1);
            send(m + (HZ ? 2 : 1) * mail_p, x, epoch);
        }
    }

    // v[c + 1] of every column: the next column's value of this row (column ny - 1 of an open y: its own)
    __device__ __forceinline__ void right(float2 (&out)[H], const float2 (&v)[H], int r) {
        const float shifted = __shfl_down_sync(0xffffffffu, v[0].x, 1), edge = lo[r * 34 + warp + 1];
        const float next = take_lo ? edge : shifted;
#pragma unroll
        for (int k = 0; k < H; ++k) out[k] = make_float2(v[k].y, k + 1 < H ? v[k + 1 < H ? k + 1 : k].x : next);
        if (end_warp && (odd || !py)) {
            if (cl >= 0) rs_set(out, cl, py ? lo[r * 34 + warp + 1] : rs_get(v, cl));
        }
    }
    // v[c - 1] (column 0: the wrapped last one, or 0)
    __device__ __forceinline__ void left(float2 (&out)[H], const float2 (&v)[H], int r) {
        const float shifted = __shfl_up_sync(0xffffffffu, v[H - 1].y, 1), edge = hi[r * 34 + warp];
        const float prev = lane == 0 ? edge : shifted;
#pragma unroll
        for (int k = 0; k < H; ++k) out[k] = make_float2(k ? v[k ? k - 1 : 0].y : prev, v[k].x);
    }
    __device__ __forceinline__ void publish_lo(const float2 (&v)[RT][H]) {
        if (lane == 0) {
#pragma unroll
            for (int r = 0; r < RT; ++r)
                if (r < R) lo[r * 34 + warp] = v[r][0].x;
            if (warp == 0) {
#pragma unroll
                for (int r = 0; r < RT; ++r)
                    if (r < R) lo[r * 34 + (blockDim.x >> 5)] = res_wrap_hi(v[r][0].x);
            }
        }
    }
    __device__ __forceinline__ void publish_hi(const float2 (&v)[RT][H]) {
        if (lane == 31) {
#pragma unroll
            for (int r = 0; r < RT; ++r)
                if (r < R) hi[r * 34 + warp + 1] = v[r][H - 1].y;
        }
        if (end_warp && py && cl >= 0) {
#pragma unroll
            for (int r = 0; r < RT; ++r)
                if (r < R) {
                    const float x = rs_get(v[r], cl);
                    hi[r * 34] = res_wrap_lo(x);
                    last[r] = x;
                }
        }
    }
    __device__ __forceinline__ void coef(float2 (&v)[H], const float *base, int r) const {
        const float2 *s = reinterpret_cast<const float2 *>(base + r * P + j0);
#pragma unroll
        for (int k = 0; k < H; ++k) v[k] = s[k];
    }
    // the dead last column of an open y keeps its value
    __device__ __forceinline__ void keep_last(float2 (&v)[H], const float2 (&old)[H]) {
        if (end_warp && !py) {
            if (cl >= 0) rs_set(v, cl, rs_get(old, cl));
        }
    }

    // a row of a field by its number (selects: the arrays stay in registers)
    __device__ __forceinline__ void get(float2 (&out)[H], const float2 (&v)[RT][H], int r) const {
#pragma unroll
        for (int q = 0; q < RT; ++q)
#pragma unroll
            for (int k = 0; k < H; ++k)
                if (q == 0 || q == r) out[k] = v[q][k];
    }
    __device__ __forceinline__ void put(float2 (&v)[RT][H], const float2 (&x)[H], int r) const {
#pragma unroll
        for (int q = 0; q < RT; ++q)
#pragma unroll
            for (int k = 0; k < H; ++k)
                if (q == r) v[q][k] = x[k];
    }

    // CPML of a row, field += sign * coefficient * psi with psi = b psi + a d inv: on a thread's columns of a y layer
    // (columns outside it keep their value) ...
    __device__ __forceinline__ void y_layer(float *psi_row, bool e_rows, const float2 (&d)[H], const float2 (&c)[H],
                                            bool negative, float2 (&v)[H]) {
        float2 *s = reinterpret_cast<float2 *>(psi_row + y_at);
        const float2 *rec = reinterpret_cast<const float2 *>(yrec + (e_rows ? 0 : 3 * Y) + y_at);
        const int y2 = Y / 2;
#pragma unroll
        for (int k = 0; k < H; ++k) {
            const float2 rb = rec[k], ra = rec[y2 + k], ri = rec[2 * y2 + k];
            float2 w = s[k];
            w.x = w.x * rb.x;
            w.y = w.y * rb.y;
            w.x += ra.x * d[k].x * ri.x;
            w.y += ra.y * d[k].y * ri.y;
            s[k] = w;
            const float x = v[k].x + (negative ? -c[k].x : c[k].x) * w.x;
            const float y = v[k].y + (negative ? -c[k].y : c[k].y) * w.y;
            if (ri.x != 0.0f) v[k].x = x;   // 1 / spacing: 0 marks a column outside the layer
            if (ri.y != 0.0f) v[k].y = y;
        }
    }
    // ... and on an x-layer row.
    __device__ __forceinline__ void x_layer(float *psi_row, float rb, float ra, float ri, const float2 (&d)[H],
                                            const float2 (&c)[H], bool negative, float2 (&v)[H]) {
        float2 *s = reinterpret_cast<float2 *>(psi_row + j0);
#pragma unroll
        for (int k = 0; k < H; ++k) {
            float2 w = s[k];
            w.x = w.x * rb;
            w.y = w.y * rb;
            w.x += ra * d[k].x * ri;
            w.y += ra * d[k].y * ri;
            s[k] = w;
            v[k].x += (negative ? -c[k].x : c[k].x) * w.x;
            v[k].y += (negative ? -c[k].y : c[k].y) * w.y;
        }
    }

    // ---------------------------------------------------------------------------------------------- E_z
    __device__ __forceinline__ void ez_hy(int r, const ResRow &row, const float2 (&e)[H], const float2 (&ed)[H],
                                          const float2 (&dbv)[H], const float2 (&dav)[H], float *psi_row,
                                          float2 (&v)[H]) {
        float2 d[H];
#pragma unroll
        for (int k = 0; k < H; ++k) {
            d[k] = rs_sub(ed[k], e[k]);
            const float2 t = rs_mul(rs_mul(dbv[k], d[k]), rs_pair(row.ixh));
            v[k] = rs_add_p(GEN ? rs_mul(dav[k], v[k]) : v[k], t);
        }
        if (row.xh >= 0) x_layer(psi_row, row.b_h, row.a_h, row.i_h, d, dbv, false, v);
    }
    __device__ __forceinline__ void coef_h(float2 (&dav)[H], float2 (&dbv)[H], int r) const {
#pragma unroll
        for (int k = 0; k < H; ++k) dav[k] = rs_pair(da_u), dbv[k] = rs_pair(db_u);
        if (GEN && p.da) coef(dav, da, r), coef(dbv, db, r);
    }
    __device__ __forceinline__ void ez_h(uint32_t epoch) {
#pragma unroll
        for (int r = 0; r < RT; ++r) {
            if (r >= R) break;
            const ResRow &row = rows[r + 1];
            float2 er[H], d[H], dav[H], dbv[H], old[H];
            coef_h(dav, dbv, r);
            right(er, f[r], r);
#pragma unroll
            for (int k = 0; k < H; ++k) {
                old[k] = a[r][k];
                d[k] = rs_sub(er[k], f[r][k]);
                const float2 t = rs_mul(rs_mul(dbv[k], d[k]), iyh[k]);
                a[r][k] = rs_sub_p(GEN ? rs_mul(dav[k], a[r][k]) : a[r][k], t);
            }
            if (yh) y_layer(yhq + r * Y, false, d, dbv, true, a[r]);
            keep_last(a[r], old);
            if (r + 1 < RT && r + 1 < R) ez_hy(r, row, f[r], f[r + 1 < RT ? r + 1 : r], dbv, dav, xh + row.xh * P, b[r]);
        }
        float2 got[2][H];   // E_z of the row above and of the row below
        {
            const uint64_t *const at[2] = {has_up ? from_up + slot(epoch) + mail_p : nullptr,
                                           has_dn ? from_dn + slot(epoch) : nullptr};
            float none;
            receive(got, at, none, nullptr, epoch);
        }
        if (has_dn) {
#pragma unroll
            for (int k = 0; k < H; ++k)
                if (wrap_dn) got[1][k] = make_float2(res_wrap_hi(got[1][k].x), res_wrap_hi(got[1][k].y));
            const ResRow &row = rows[R];
            float2 dav[H], dbv[H], e[H], v[H];
            coef_h(dav, dbv, R - 1);
            get(e, f, R - 1);
            get(v, b, R - 1);
            ez_hy(R - 1, row, e, got[1], dbv, dav, xh + row.xh * P, v);
            put(b, v, R - 1);
        }
        if (has_up) {   // H_y of the row above, again
            const ResRow &row = rows[0];
            float2 ed[H], dav[H], dbv[H];
#pragma unroll
            for (int k = 0; k < H; ++k)
                ed[k] = wrap_up ? make_float2(res_wrap_hi(f[0][k].x), res_wrap_hi(f[0][k].y)) : f[0][k];
            coef_h(dav, dbv, -1);
            ez_hy(-1, row, got[0], ed, dbv, dav, gx, g);
        }
        if (GEN && p.n_tfsf) {
            tfsf_ab();
            if (has_up && (rows[0].flags & RF_EDGE)) res_to(g, res_tfsf_row<C>(p, aux, false, rows[0].i, j0, res_from(g)));
        }
        publish_hi(a);
    }

    // plane-wave box corrections of the in-plane fields: b on the boxes' edge rows, a on their edge columns (from the
    // incident E after the H update of an E_z engine, from the incident H after the E update of an H_z engine)
    __device__ __forceinline__ void tfsf_ab() {
#pragma unroll 1
        for (int r = 0; r < R; ++r) {
            if (!(rows[r + 1].flags & RF_EDGE)) continue;
            float2 y[H];
            get(y, b, r);
            res_to(y, res_tfsf_row<C>(p, aux, HZ, i0 + r, j0, res_from(y)));
            put(b, y, r);
        }
        if (!edge_col) return;
        const float *line = reinterpret_cast<const float *>(res_smem) + aux;
#pragma unroll 1
        for (int k = 0; k < p.n_tfsf; ++k) {
            const ResTfsf &t = p.tfsf[k];
            const float *incident = line + (HZ ? t.aux_n : 0) + t.aux_x0 + (i0 - t.x0);
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                const int at = (side ? t.y1 : t.y0) - 1 - j0;
                if (at < 0 || at >= C) continue;
                const float coef = HZ ? t.coef_e[2 + side] : t.coef_h[2 + side];
                const bool minus = HZ ? side == 0 : side == 1;
#pragma unroll
                for (int r = 0; r < RT; ++r) {
                    if (r >= R || i0 + r < t.x0 || i0 + r >= t.x1) continue;
                    const float term = coef * incident[r], x = rs_get(a[r], at);
                    rs_set(a[r], at, minus ? x - term : x + term);
                }
            }
            line += 4 * t.aux_n;
        }
    }

    // poles on the strip's pole rows: the updates from E^n before the E update (u: E_z or E_x, w: E_y of an H_z engine) ...
    __device__ __forceinline__ void pole_updates(const float2 (&u)[RT][H], const float2 (&w)[RT][H]) {
#pragma unroll 1
        for (int r = 0; r < R; ++r) {
            const uint32_t mask = rows[r + 1].poles & pole_mask;
            if (!mask) continue;
            float2 x[H], y[H];
            get(x, u, r);
            get(y, w, r);
            res_pole_update<C>(pole_tab, mask, r, j0, res_from(x), res_from(y));
        }
    }
    // ... and the corrections after it
    __device__ __forceinline__ void pole_corrections(float2 (&v)[RT][H], int comp, const float *cb_rows) {
#pragma unroll 1
        for (int r = 0; r < R; ++r) {
            const uint32_t mask = rows[r + 1].poles & pole_mask;
            if (!mask) continue;
            float2 x[H], cb[H];
            get(x, v, r);
            coef(cb, cb_rows, r);
            res_to(x, res_pole_correct<C>(pole_tab, mask, HZ, comp, p.n_drude == 1, p.inv_dt, r, j0, res_from(x),
                                          res_from(cb)));
            put(v, x, r);
        }
    }

    __device__ __forceinline__ void ez_e(int64_t step, uint32_t epoch) {
        if (GEN && pole_mask) pole_updates(f, f);
#pragma unroll
        for (int r = 0; r < RT; ++r) {
            if (r >= R) break;
            const ResRow &row = rows[r + 1];
            float2 hl[H], cb[H], dx[H], dy[H], ca[H];
            coef(cb, cx, r);
            if (GEN && p.ca) coef(ca, cax, r);
            left(hl, a[r], r);
#pragma unroll
            for (int k = 0; k < H; ++k) {
                float2 below = r ? b[r ? r - 1 : 0][k] : g[k];   // H_y of the row above in the array
                if (r == 0 && wrap_up) below = make_float2(res_wrap_lo(below.x), res_wrap_lo(below.y));
                dx[k] = rs_sub(b[r][k], below);
                dy[k] = rs_sub(a[r][k], hl[k]);
                const float2 curl = rs_sub_p(rs_mul(dx[k], rs_pair(row.ixe)), rs_mul(dy[k], iye[k]));
                f[r][k] = rs_add_p(GEN && p.ca ? rs_mul(ca[k], f[r][k]) : f[r][k], rs_mul(cb[k], curl));
            }
            if (row.xe >= 0) x_layer(xe + row.xe * P, row.b_e, row.a_e, row.i_e, dx, cb, false, f[r]);
            if (ye) y_layer(yeq + r * Y, true, dy, cb, true, f[r]);
        }
        if (GEN && pole_mask) pole_corrections(f, 0, cx);
        if (lines) sources(-1, step - 1, f);
        if (GEN && p.n_tfsf) {
#pragma unroll 1
            for (int r = 0; r < R; ++r) {
                if (!(rows[r + 1].flags & RF_TFSF)) continue;
                float2 x[H];
                get(x, f, r);
                res_to(x, res_tfsf_row<C>(p, aux, true, i0 + r, j0, res_from(x)));
                put(f, x, r);
            }
        }
        mail(epoch);
        publish_lo(f);
    }

    // ---------------------------------------------------------------------------------------------- H_z
    __device__ __forceinline__ void hz_update(int r, const ResRow &row, const float2 (&ex)[H], const float2 (&exl)[H],
                                              const float2 (&ey)[H], const float2 (&eyd)[H], float *px, float *py_psi,
                                              float2 (&v)[H]) {
        float2 dx[H], dy[H], dav[H], dbv[H];
        coef_h(dav, dbv, r);
#pragma unroll
        for (int k = 0; k < H; ++k) {
            dy[k] = rs_sub(ex[k], exl[k]);
            dx[k] = rs_sub(ey[k], eyd[k]);
            const float2 curl = rs_sub_p(rs_mul(dy[k], iye[k]), rs_mul(dx[k], rs_pair(row.ixe)));
            v[k] = rs_add_p(GEN ? rs_mul(dav[k], v[k]) : v[k], rs_mul(dbv[k], curl));
        }
        if (row.xe >= 0) x_layer(px, row.b_e, row.a_e, row.i_e, dx, dbv, true, v);
        if (ye) y_layer(py_psi, true, dy, dbv, false, v);
        if (GEN && (row.flags & RF_TFSF)) res_to(v, res_tfsf_row<C>(p, aux, false, row.i, j0, res_from(v)));
    }
    // fold >= 0: the step before was a sample step of the field maps, whose E partners have arrived now
    __device__ __forceinline__ void hz_h(uint32_t epoch, int64_t fold, bool update) {
        const uint64_t *mu = has_up ? from_up + slot(epoch) + 2 * mail_p : nullptr, *md = from_dn + slot(epoch);
        if (GEN && fold >= 0) {
            const uint64_t *const at[1] = {mu};
            float2 up[1][H];
            float none;
            receive(up, at, none, nullptr, epoch);
#pragma unroll 1
            for (int r = 0; r < R; ++r) {
                float2 h[H], x[H], xl[H], y[H], yl[H];
                get(x, a, r);
                left(xl, x, r);
                if (!(rows[r + 1].flags & RF_MAP)) continue;
                get(h, f, r);
                get(y, b, r);
                get(yl, b, r ? r - 1 : 0);
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    if (j0 + c >= ny) continue;
                    // the lo partner of column 0 is the wrapped face unscaled, or the face itself
                    const float lo_x = j0 + c ? rs_get(xl, c) : py ? last[r] : rs_get(x, c);
                    const float lo_y = r ? rs_get(yl, c) : has_up ? rs_get(up[0], c) : rs_get(y, c);
                    res_maps_hz(p, i0 + r, j0 + c, fold, rs_get(h, c), rs_get(x, c), lo_x, rs_get(y, c), lo_y);
                }
            }
        }
        if (!update) return;
#pragma unroll
        for (int r = RT - 1; r >= 1; --r) {   // rows that need no mail
            float2 exl[H];
            if (r < R) {
                left(exl, a[r], r);
                const ResRow &row = rows[r + 1];
                hz_update(r, row, a[r], exl, b[r], b[r ? r - 1 : 0], xe + row.xe * P, yeq + r * Y, f[r]);
            }
        }
        float2 got[3][H];   // E_y of the row above; E_x, E_y of the row below
        float prev_edge = 0.0f;
        {
            const uint64_t *const at[3] = {mu, has_dn ? md : nullptr, has_dn ? md + mail_p : nullptr};
            // E_x left of the warp's first column on the row below
            const bool edge = has_dn && lane == 0 && j0 < ny && (j0 > 0 || py);
            receive(got, at, prev_edge, edge ? md + (j0 > 0 ? j0 : ny) - 1 : nullptr, epoch);
            if (!edge) prev_edge = 0.0f;
            else if (j0 == 0) prev_edge = res_wrap_lo(prev_edge);
        }
        {
            const ResRow &row = rows[1];
            float2 exl[H];
            left(exl, a[0], 0);
#pragma unroll
            for (int k = 0; k < H; ++k) {
                if (!has_up) got[0][k] = make_float2(0.0f, 0.0f);
                if (wrap_up) got[0][k] = make_float2(res_wrap_lo(got[0][k].x), res_wrap_lo(got[0][k].y));
            }
            hz_update(0, row, a[0], exl, b[0], got[0], xe + row.xe * P, yeq, f[0]);
        }
        if (has_dn) {   // H_z of the row below, again
            const ResRow &row = rows[R + 1];
            float2 exl[H], eyd[H];
            float prev = __shfl_up_sync(0xffffffffu, got[1][H - 1].y, 1);
            if (lane == 0) prev = prev_edge;
#pragma unroll
            for (int k = 0; k < H; ++k) exl[k] = make_float2(k ? got[1][k ? k - 1 : 0].y : prev, got[1][k].x);
            get(eyd, b, R - 1);
#pragma unroll
            for (int k = 0; k < H; ++k)
                if (wrap_dn) eyd[k] = make_float2(res_wrap_lo(eyd[k].x), res_wrap_lo(eyd[k].y));
            hz_update(R, row, got[1], exl, got[2], eyd, gx, gy, g);
        }
        publish_lo(f);
    }

    __device__ __forceinline__ void hz_e(int64_t step, uint32_t epoch) {
        if (GEN && pole_mask) {
            pole_updates(a, b);
        }
#pragma unroll
        for (int r = 0; r < RT; ++r) {
            if (r >= R) break;
            const ResRow &row = rows[r + 1];
            float2 hr[H], hd[H], cbx[H], cby[H], dx[H], dy[H], old_x[H];
            coef(cbx, cx, r);
            coef(cby, cy, r);
            right(hr, f[r], r);
            const bool live_y = r + 1 < R || has_dn;
#pragma unroll
            for (int k = 0; k < H; ++k) {
                old_x[k] = a[r][k];
                float2 n = (r + 1 < RT && r + 1 < R) ? f[r + 1 < RT ? r + 1 : r][k] : g[k];
                if (r == R - 1 && wrap_dn) n = make_float2(res_wrap_hi(n.x), res_wrap_hi(n.y));
                hd[k] = n;
            }
            float2 cav[H];
            if (GEN && p.ca) coef(cav, cax, r);
#pragma unroll
            for (int k = 0; k < H; ++k) {
                dy[k] = rs_sub(hr[k], f[r][k]);
                a[r][k] = rs_add_p(GEN && p.ca ? rs_mul(cav[k], a[r][k]) : a[r][k],
                                   rs_mul(rs_mul(cbx[k], dy[k]), iyh[k]));
            }
            if (yh) y_layer(yhq + r * Y, false, dy, cbx, false, a[r]);
            keep_last(a[r], old_x);
            if (live_y) {
                if (GEN && p.ca) coef(cav, cay, r);
#pragma unroll
                for (int k = 0; k < H; ++k) {
                    dx[k] = rs_sub(hd[k], f[r][k]);
                    b[r][k] = rs_sub_p(GEN && p.ca ? rs_mul(cav[k], b[r][k]) : b[r][k],
                                       rs_mul(rs_mul(cby[k], dx[k]), rs_pair(row.ixh)));
                }
                if (row.xh >= 0) x_layer(xh + row.xh * P, row.b_h, row.a_h, row.i_h, dx, cby, true, b[r]);
            }
        }
        if (GEN && pole_mask) {
            pole_corrections(a, 0, cx);
            pole_corrections(b, 1, cy);
        }
        if (lines) {
            sources(0, step - 1, a);
            sources(1, step - 1, b);
        }
        if (GEN && p.n_tfsf) {
            tfsf_ab();
        }
        mail(epoch);
        publish_hi(a);
    }

    // ---------------------------------------------------------------------------------------------- lines, samples
    // Line sources on the thread's cells of field v (axis < 0: both axes act on it), in add order, a 0 value skipped.
    // An H_z engine's sheet does not reach the dead last faces of an open axis unless poles make it a pass of its own.
    __device__ __forceinline__ void sources(int axis, int64_t k_step, float2 (&v)[RT][H]) {
#pragma unroll 1
        for (uint32_t left_lines = lines; left_lines; left_lines &= left_lines - 1) {
            const int l = __ffs(left_lines) - 1;
            const ResLine &L = p.lines[l];
            if (axis >= 0 && L.axis != axis) continue;
            const float value = __ldg(p.line_values + (size_t)l * p.values_stride + k_step);
            if (value == 0.0f) continue;
            const int first = L.axis == 1 ? L.position - i0 : max(L.lo - i0, 0);
            const int end = L.axis == 1 ? first + 1 : min(L.hi - i0, R);
#pragma unroll 1
            for (int r = first; r < end; ++r) {
                if (HZ && L.axis == 1 && r == R - 1 && !has_dn && !p.n_poles) continue;
                float2 x[H];
                get(x, v, r);
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    const int j = j0 + c;
                    if (L.axis == 1 ? (j < L.lo || j >= L.hi) : j != L.position) continue;
                    if (HZ && L.axis == 0 && c == cl && !py && !p.n_poles) continue;
                    float &y = (c & 1) ? x[c >> 1].y : x[c >> 1].x;
                    y += value * __ldg(L.profile + (L.axis == 1 ? j - L.lo : i0 + r - L.lo));
                }
                put(v, x, r);
            }
        }
    }

    // Flux-line samples, probes and E_z maps of the state after a step.
    __device__ __forceinline__ void samples(int64_t n, bool sample) {
        if (mons && sample) {
            const size_t s = (size_t)(n / p.m - p.q_first);
#pragma unroll 1
            for (uint32_t left_mons = mons; left_mons; left_mons &= left_mons - 1) {
                const ResMon &M = p.mons[__ffs(left_mons) - 1];
                const int len = M.hi - M.lo;
                float *out = M.stage + s * 2 * (size_t)len;
                const int first = M.normal_axis == 0 ? M.position - i0 : max(M.lo - i0, 0);
                const int end = M.normal_axis == 0 ? first + 1 : min(M.hi - i0, R);
#pragma unroll 1
                for (int r = first; r < end; ++r) {
                    float2 x[H], t[H];
                    get(x, f, r);
                    if (M.normal_axis == 0) get(t, b, r);   // the in-plane component tangential to the line
                    else get(t, a, r);
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        const int j = j0 + c;
                        if (M.normal_axis == 0 ? (j < M.lo || j >= M.hi) : j != M.position) continue;
                        const int at = M.normal_axis == 0 ? j - M.lo : i0 + r - M.lo;
                        out[at] = HZ ? rs_get(t, c) : rs_get(x, c);
                        out[len + at] = HZ ? rs_get(x, c) : rs_get(t, c);
                    }
                }
            }
        }
#pragma unroll 1
        for (uint32_t left_probes = probes; left_probes; left_probes &= left_probes - 1) {
            const ResProbe &q = p.probes[__ffs(left_probes) - 1];
            if (n - 1 < q.start) continue;
            float2 x[H];
            if (q.comp == 0) get(x, f, q.ix - i0);
            else if (q.comp == 1) get(x, a, q.ix - i0);
            else get(x, b, q.ix - i0);
            q.row[n - 1] = rs_get(x, q.iy - j0);
        }
        if (!HZ && records) {
            const int w = p.rec_j1 - p.rec_j0, first = max(p.rec_i0 - i0, 0), end = min(p.rec_i1 - i0, R);
            float *out = p.rec + (size_t)(n - p.n0) * (size_t)(p.rec_i1 - p.rec_i0) * w + (j0 - p.rec_j0);
#pragma unroll 1
            for (int r = first; r < end; ++r) {
                float2 x[H];
                get(x, f, r);
#pragma unroll
                for (int c = 0; c < C; ++c)
                    if (j0 + c >= p.rec_j0 && j0 + c < p.rec_j1) out[(i0 + r - p.rec_i0) * w + c] = rs_get(x, c);
            }
        }
        if (GEN && !HZ && p.n_maps && sample) {
#pragma unroll 1
            for (int r = 0; r < R; ++r) {
                if (!(rows[r + 1].flags & RF_MAP)) continue;
                float2 x[H];
                get(x, f, r);
#pragma unroll
                for (int c = 0; c < C; ++c)
                    if (j0 + c < ny) res_maps_ez(p, i0 + r, j0 + c, n, rs_get(x, c));
            }
        }
    }
};

// Row facts of strip row r (-1 .. R); xe / xh only say whether the row lies in a layer (0, or -1).
static __device__ ResRow res_row(const Res2DJob &p, int i) {
    ResRow row = {};
    row.xe = row.xh = -1;
    if (i < 0) i += p.nx;
    if (i >= p.nx) i -= p.nx;
    row.i = i;
    row.ixe = p.inv_dx_e[i];
    row.ixh = p.inv_dx_h[i];
    int k;
    int side = res_e_side(RSX_LO, p.cpml_mask, i, p.nx, p.npml, k);
    if (side >= 0) {
        const float *c = p.cpml_rows[side];
        row.b_e = c[k], row.a_e = c[p.npml + k], row.i_e = c[2 * p.npml + k];
        row.xe = 0;
    }
    side = res_h_side(RSX_LO, p.cpml_mask, i, p.nx, p.npml, k);
    if (side >= 0) {
        const float *c = p.cpml_rows[side] + 3 * p.npml;
        row.b_h = c[k], row.a_h = c[p.npml + k], row.i_h = c[2 * p.npml + k];
        row.xh = 0;
    }
    for (int q = 0; q < p.n_poles; ++q)
        if (i >= p.poles[q].i0 && i < p.poles[q].i1) row.poles |= 1u << q;
    for (int q = 0; q < p.n_maps; ++q) {
        const int d = i - p.maps[q].x0;
        if (d >= 0 && d % p.maps[q].ds == 0 && d / p.maps[q].ds < p.maps[q].mx) row.flags |= RF_MAP;
    }
    for (int q = 0; q < p.n_tfsf; ++q) {
        if (i == p.tfsf[q].x0 || i == p.tfsf[q].x1 - 1) row.flags |= RF_TFSF;
        if (i == p.tfsf[q].x0 - 1 || i == p.tfsf[q].x1 - 1) row.flags |= RF_EDGE;
    }
    return row;
}
// Global psi row (ny floats) of physical row i, NULL outside the layers.
static __device__ float *res_psi_row(const Res2DJob &p, int i, bool e_rows) {
    int k;
    const int side = e_rows ? res_e_side(RSX_LO, p.cpml_mask, i, p.nx, p.npml, k)
                            : res_h_side(RSX_LO, p.cpml_mask, i, p.nx, p.npml, k);
    return side < 0 ? nullptr : (e_rows ? p.psi_e[side] : p.psi_h[side]) + (size_t)k * p.ny;
}
// Global y-side psi of place q of the strip's layer columns on physical row i, NULL outside the layers.
template <typename S>
static __device__ float *res_y_psi(const Res2DJob &p, const S &s, int q, int i, bool e_rows) {
    constexpr int C = S::COLS;
    const int y_lo = (p.cpml_mask >> RSY_LO) & 1 ? (p.npml / C + 1) * C : 0, first = (p.ny - p.npml - 1) / C * C;
    const int j = q < y_lo ? q : first + q - y_lo;
    if (j >= p.ny || (q >= y_lo && j < y_lo)) return nullptr;   // a thread of both layers keeps its place in the lo one
    int k;
    const int side = e_rows ? res_e_side(RSY_LO, p.cpml_mask, j, p.ny, p.npml, k)
                            : res_h_side(RSY_LO, p.cpml_mask, j, p.ny, p.npml, k);
    return side < 0 ? nullptr : (e_rows ? p.psi_e[side] : p.psi_h[side]) + (size_t)i * p.npml + k;
}
// The strip's x-side psi rows, y-side psi and pole state between the engine's arrays and shared memory.
template <typename S>
static __device__ void res_copy_psi(const Res2DJob &p, const S &s, int tid, int nt, bool out) {
    int ne = 0, nh = 0;
    for (int r = 0; r < s.R; ++r)
        for (int kind = 0; kind < 2; ++kind) {
            float *src = res_psi_row(p, s.i0 + r, kind == 0);
            if (!src) continue;
            float *dst = kind == 0 ? s.xe + ne++ * s.P : s.xh + nh++ * s.P;
            for (int j = tid; j < p.ny; j += nt) {
                if (out) src[j] = dst[j];
                else dst[j] = src[j];
            }
        }
    for (int t = tid; t < s.R * s.Y; t += nt) {
        const int r = t / s.Y, q = t - r * s.Y;
        for (int kind = 0; kind < 2; ++kind) {
            float *psi = res_y_psi(p, s, q, s.i0 + r, kind == 0), *mine = kind == 0 ? s.yeq + t : s.yhq + t;
            if (out && psi) *psi = *mine;
            if (!out) *mine = psi ? *psi : 0.0f;
        }
    }
    float *base = s.pole;
    for (int k = 0; k < p.n_poles; ++k) {
        const ResPole &q = p.poles[k];
        const int wide = q.j1 - q.j0, w = res_pole_width(q, S::COLS), pad = q.j0 - q.j0 / S::COLS * S::COLS;
        const int first = max(q.i0, s.i0), rows = max(min(q.i1, s.i0 + s.R) - first, 0), n = rows * w;
        for (int t = tid; t < n; t += nt) {
            const int r = t / w, col = t - r * w - pad;
            const bool in = col >= 0 && col < wide;
            const size_t g = (size_t)(first - q.i0 + r) * wide + col;
            if (out) {
                if (in) q.a[g] = base[n + t];
                if (in && q.kind) q.b[g] = base[2 * n + t];
            } else {
                base[t] = in ? q.drive[g] : 0.0f;
                base[n + t] = in ? q.a[g] : 0.0f;
                if (q.kind) base[2 * n + t] = in ? q.b[g] : 0.0f;
            }
        }
        base += res_pole_floats(q, s.i0, s.i0 + s.R, S::COLS);
    }
}

// Threads of a block and floats of its shared memory behind the job and the row table (the kernel lays them out).
__host__ __device__ static inline int res_threads(int ny, int c) { return ((ny + c - 1) / c + 31) & ~31; }
__host__ __device__ static inline size_t res_strip_floats(const Res2DJob &p, int i0, int i1, int layer_e, int layer_h,
                                                          int c, int rt) {
    const size_t P = (size_t)res_threads(p.ny, c) * c, R = (size_t)(i1 - i0), Y = 2 * (size_t)(p.npml + 2 * c);
    size_t n = (size_t)rt * 69 + (R + (p.da ? 2 : 0)) * P * res_coef_arrays(p) +
               ((size_t)layer_e + layer_h + 1) * P + (2 * R + 7) * Y + 16;
    for (int k = 0; k < p.n_tfsf; ++k) n += 4 * (size_t)p.tfsf[k].aux_n;
    for (int k = 0; k < p.n_poles; ++k) n += (size_t)res_pole_floats(p.poles[k], i0, i1, c);
    return n;
}

template <bool HZ, bool GEN, int C, int RT, int NT>
__global__ void __launch_bounds__(NT, 1) res2d_kernel(const __grid_constant__ Res2DJob job) {
    __shared__ int dead_flag;
    const int tid = threadIdx.x, nt = blockDim.x;
    Res2DJob &p = *reinterpret_cast<Res2DJob *>(res_smem);
    for (int w = tid; w < (int)(sizeof(Res2DJob) / 8); w += nt)
        reinterpret_cast<uint64_t *>(&p)[w] = reinterpret_cast<const uint64_t *>(&job)[w];
    if (tid == 0) dead_flag = 0;
    __syncthreads();

    ResStrip<HZ, GEN, C, RT> s(p);
    const int c = blockIdx.x, last_cta = p.n_cta - 1;
    s.i0 = p.row_start[c];
    s.R = p.row_start[c + 1] - s.i0;
    s.ny = p.ny;
    s.mail_p = res_pitch(p.ny);
    s.P = nt * C;
    s.py = p.py;
    s.odd = p.ny % C != 0;
    s.wrap_up = p.px && c == 0;
    s.wrap_dn = p.px && c == last_cta;
    s.has_up = c > 0 || p.px;
    s.has_dn = c < last_cta || p.px;
    {
        const size_t words = 2 * res_mail_rows(HZ) * (size_t)s.mail_p;
        s.from_up = p.mail + (c > 0 ? c - 1 : last_cta) * words;
        s.from_dn = p.mail + (c < last_cta ? c + 1 : 0) * words;
        s.to_me = p.mail + c * words;
    }
    s.dead = &dead_flag;
    s.lane = tid & 31;
    s.warp = tid >> 5;
    s.j0 = tid * C;
    s.cl = p.ny - 1 - s.j0;
    if (s.cl < 0 || s.cl >= C) s.cl = -1;
    s.end_warp = (p.ny - 1) / (32 * C) == s.warp;
    s.take_lo = s.lane == 31 || s.cl == C - 1;
    s.da_u = p.da_u;
    s.db_u = p.db_u;
    s.yh = s.ye = s.edge_col = false;
    s.pole_mask = 0;
#pragma unroll
    for (int q = 0; q < C; ++q) {
        const int j = s.j0 + q;
        const bool in = j < p.ny;
        rs_set(s.iye, q, in ? p.inv_dy_e[j] : 0.0f);
        rs_set(s.iyh, q, in ? p.inv_dy_h[j] : 0.0f);
        int k;
        s.ye = s.ye || (in && res_e_side(RSY_LO, p.cpml_mask, j, p.ny, p.npml, k) >= 0);
        s.yh = s.yh || (in && res_h_side(RSY_LO, p.cpml_mask, j, p.ny, p.npml, k) >= 0);
        for (int t = 0; t < p.n_tfsf; ++t) s.edge_col = s.edge_col || j == p.tfsf[t].y0 - 1 || j == p.tfsf[t].y1 - 1;
        for (int t = 0; t < p.n_poles; ++t)
            if (j >= p.poles[t].j0 && j < p.poles[t].j1) s.pole_mask |= 1u << t;
    }
    auto touches = [&](int axis_along_y, int position, int lo, int hi) {
        // cells (position, j) for lines along y, (i, position) for lines along x
        if (axis_along_y) return position >= s.i0 && position < s.i0 + s.R && lo < s.j0 + C && hi > s.j0;
        return position >= s.j0 && position < s.j0 + C && lo < s.i0 + s.R && hi > s.i0;
    };
    s.lines = s.mons = s.probes = 0;
    for (int k = 0; k < p.n_lines; ++k)
        if (touches(p.lines[k].axis == 1, p.lines[k].position, p.lines[k].lo, p.lines[k].hi)) s.lines |= 1u << k;
    for (int k = 0; k < p.n_mons; ++k)
        if (touches(p.mons[k].normal_axis == 0, p.mons[k].position, p.mons[k].lo, p.mons[k].hi)) s.mons |= 1u << k;
    for (int k = 0; k < p.n_probes; ++k)
        if (touches(1, p.probes[k].ix, p.probes[k].iy, p.probes[k].iy + 1)) s.probes |= 1u << k;

    // Y-side CPML columns: the threads of the lo layer (columns up to npml), then those of the hi layer (from
    // ny - npml - 1), each thread with all its columns
    const int y_lo = (p.cpml_mask >> RSY_LO) & 1 ? p.npml / C + 1 : 0;
    const int y_first = (p.ny - p.npml - 1) / C, y_hi = (p.cpml_mask >> RSY_HI) & 1 ? (p.ny - 2) / C - y_first + 1 : 0;
    s.Y = (y_lo + y_hi) * C;
    s.y_at = (tid < y_lo ? tid : y_lo + tid - y_first) * C;
    s.records = !HZ && p.rec && p.rec_j0 < s.j0 + C && p.rec_j1 > s.j0;
    // ---- shared memory
    s.rows = reinterpret_cast<ResRow *>(res_smem + sizeof(Res2DJob));
    for (int r = tid; r < s.R + 2; r += nt) {
        const int i = s.i0 + r - 1;
        if ((i < 0 || i >= p.nx) && !p.px) {
            s.rows[r] = ResRow{};
            s.rows[r].xe = s.rows[r].xh = -1;
        } else {
            s.rows[r] = res_row(p, i);
        }
    }
    __syncthreads();
    int n_e = 0, n_h = 0;
    for (int r = 0; r < s.R; ++r) n_e += s.rows[r + 1].xe >= 0, n_h += s.rows[r + 1].xh >= 0;
    ResPoleRows *pole_rows = reinterpret_cast<ResPoleRows *>(s.rows + s.R + 2);
    s.pole_tab = (int)(reinterpret_cast<unsigned char *>(pole_rows) - res_smem);
    float *at = reinterpret_cast<float *>(pole_rows + p.n_poles);
    const int P = s.P, rp = s.R * P;
    s.cx = at, at += rp;
    s.cy = at, at += HZ ? rp : 0;
    s.cax = at, at += p.ca ? rp : 0;
    s.cay = at, at += p.ca && HZ ? rp : 0;
    s.da = at + P, at += p.da ? rp + 2 * P : 0;   // with the rows above and below the strip
    s.db = at + P, at += p.da ? rp + 2 * P : 0;
    s.gx = at, at += P;
    s.xe = at, at += n_e * P;
    s.xh = at, at += n_h * P;
    s.yeq = at, at += s.R * s.Y;
    s.yhq = at, at += s.R * s.Y;
    s.gy = at, at += s.Y;
    s.yrec = at, at += 6 * s.Y;
    s.lo = at, at += RT * 34;
    s.hi = at, at += RT * 34;
    s.last = at, at += RT;
    s.pole = at;
    for (int k = 0; k < p.n_poles; ++k) {
        const ResPole &q = p.poles[k];
        const int first = max(q.i0, s.i0), w = res_pole_width(q, C), n = max(min(q.i1, s.i0 + s.R) - first, 0) * w;
        if (tid == 0)
            pole_rows[k] = ResPoleRows{(int)(at - reinterpret_cast<float *>(res_smem)), n, first - s.i0, w, q.j0 / C * C,
                                       q.j0, q.j1, q.kind, q.damping, q.restoring, q.comp, 0};
        at += res_pole_floats(q, s.i0, s.i0 + s.R, C);
    }
    float *const aux = at;
    s.aux = (int)(at - reinterpret_cast<float *>(res_smem));
    for (int t = tid; t < s.R * p.ny; t += nt) {
        const int r = t / p.ny, j = t - r * p.ny;
        const size_t q = (size_t)(s.i0 + r) * p.ny + j;
        s.cx[r * P + j] = p.cb[q];
        if (HZ) s.cy[r * P + j] = p.cb_y[q];
        if (p.ca) s.cax[r * P + j] = p.ca[q];
        if (HZ && p.ca) s.cay[r * P + j] = p.ca_y[q];
    }
    for (int j = p.ny + tid; j < P; j += nt)   // the pitch's padding: plain zeros
        for (int r = 0; r < s.R; ++r) {
            s.cx[r * P + j] = 0.0f;
            if (HZ) s.cy[r * P + j] = 0.0f;
            if (p.ca) s.cax[r * P + j] = 0.0f;
            if (HZ && p.ca) s.cay[r * P + j] = 0.0f;
        }
    if (p.da)
        for (int r = -1; r <= s.R; ++r)
            for (int j = tid; j < P; j += nt) {
                const bool in = j < p.ny && (r >= 0 || s.has_up) && (r < s.R || s.has_dn);
                const size_t q = in ? (size_t)s.rows[r + 1].i * p.ny + j : 0;
                s.da[r * P + j] = in ? p.da[q] : 0.0f;
                s.db[r * P + j] = in ? p.db[q] : 0.0f;
            }
    for (int j = p.ny + tid; j < P; j += nt) {
        for (int r = 0; r < n_e; ++r) s.xe[r * P + j] = 0.0f;
        for (int r = 0; r < n_h; ++r) s.xh[r * P + j] = 0.0f;
    }
    for (int t = tid; t < RT * 69; t += nt) s.lo[t] = 0.0f;
    for (int t = tid; t < 6 * s.Y; t += nt) {
        const int kind = t / (3 * s.Y), field = (t / s.Y) % 3, q = t % s.Y;
        const int j = q < y_lo * C ? q : y_first * C + q - y_lo * C;
        int k;
        const int side = kind == 0 ? res_e_side(RSY_LO, p.cpml_mask, j, p.ny, p.npml, k)
                                   : res_h_side(RSY_LO, p.cpml_mask, j, p.ny, p.npml, k);
        s.yrec[t] = side < 0 || j >= p.ny ? 0.0f : p.cpml_rows[side][(kind * 3 + field) * p.npml + k];
    }
    res_copy_psi(p, s, tid, nt, false);
    // the recomputed row: H_y above the strip (E_z), H_z below it (H_z)
    const ResRow &ghost = s.rows[HZ ? s.R + 1 : 0];
    const bool has_ghost = HZ ? s.has_dn : s.has_up;
    {
        const float *psi = has_ghost ? res_psi_row(p, ghost.i, HZ) : nullptr;
        for (int j = tid; j < P; j += nt) s.gx[j] = psi && j < p.ny ? psi[j] : 0.0f;
        for (int q = tid; q < s.Y; q += nt) {
            const float *psi_y = HZ && has_ghost ? res_y_psi(p, s, q, ghost.i, true) : nullptr;
            s.gy[q] = psi_y ? *psi_y : 0.0f;
        }
        const float *src = HZ ? p.f : p.b;
#pragma unroll
        for (int q = 0; q < C; ++q)
            rs_set(s.g, q, has_ghost && s.j0 + q < p.ny ? src[(size_t)ghost.i * p.ny + s.j0 + q] : 0.0f);
    }
    {
        float *line = aux;
        for (int k = 0; k < p.n_tfsf; ++k) {
            const ResTfsf &t = p.tfsf[k];
            const int n = t.aux_n;
            for (int q = tid; q < n; q += nt) {
                line[q] = t.aux_e[q], line[n + q] = t.aux_h[q];
                line[2 * n + q] = q < n - 1 ? t.aux_coef_h[q] : 0.0f, line[3 * n + q] = t.aux_coef_e[q];
            }
            line += 4 * n;
        }
    }
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int q = 0; q < C; ++q) {
            const bool in = r < s.R && s.j0 + q < p.ny;
            const size_t at_q = in ? (size_t)(s.i0 + r) * p.ny + s.j0 + q : 0;
            rs_set(s.f[r], q, in ? p.f[at_q] : 0.0f);
            rs_set(s.a[r], q, in ? p.a[at_q] : 0.0f);
            rs_set(s.b[r], q, in ? p.b[at_q] : 0.0f);
        }
    __syncthreads();
    if (tid == 0) {   // psi places of the layer rows
        int e = 0, h = 0;
        for (int r = 0; r < s.R; ++r) {
            if (s.rows[r + 1].xe >= 0) s.rows[r + 1].xe = e++;
            if (s.rows[r + 1].xh >= 0) s.rows[r + 1].xh = h++;
        }
    }
    if (HZ) s.publish_hi(s.a);
    else s.publish_lo(s.f);
    if (tid == 0) res_arrive(p.arrived);   // every thread's loads came before the barrier above
    if (p.stall_probe_ns && c == 0) {
        // test hook: this block sends nothing for the given time, then gives up as a real wait does
        const uint64_t t0 = tb_globaltimer();
        while (tb_globaltimer() - t0 <= (uint64_t)p.stall_probe_ns) {
        }
        if (tid == 0) atomicExch(p.err, 1);
        return;
    }
    uint32_t epoch = p.epoch;
    s.mail(epoch);
    // No block steps before all have loaded: what one reads here another overwrites later (the recomputed row and its psi
    // by their owner; the plane-wave boxes' lines, which every block reads, by block 0 at its end, and a mail travels one
    // strip a step, so a short launch's mails order block 0 behind its near strips only).
    if (tid == 0) res_wait_all(p.arrived, p.arrivals, p.err, &dead_flag);
    if (__syncthreads_or(*(volatile int *)&dead_flag)) return;

    // ---- the steps
    const bool maps = GEN && HZ && p.n_maps;
    const int64_t n_steps = p.n_steps, n0 = p.n0;
    int64_t fold = -1, to_sample = p.m - n0 % p.m;   // steps to the next DFT sample
    for (int64_t step = 1; step <= n_steps; ++step) {
        if constexpr (HZ) s.hz_h(epoch, fold, true);
        else s.ez_h(epoch);
        if (GEN && p.n_tfsf) res_aux_h(p, s.aux, tid, nt);
        if (__syncthreads_or(*(volatile int *)&dead_flag)) return;
        epoch += 1;
        if constexpr (HZ) s.hz_e(step, epoch);
        else s.ez_e(step, epoch);
        if (GEN && p.n_tfsf) res_aux_e(p, s.aux, step - 1, tid, nt);
        const bool sample = --to_sample == 0;
        if (sample) to_sample = p.m;
        s.samples(n0 + step, sample);
        fold = maps && sample ? n0 + step : -1;
        __syncthreads();
    }
    if constexpr (HZ) {
        if (maps && fold >= 0) {   // the last step was a sample step of the field maps
            s.hz_h(epoch, fold, false);
            if (__syncthreads_or(*(volatile int *)&dead_flag)) return;
        }
    }

    // ---- state out
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int q = 0; q < C; ++q)
            if (r < s.R && s.j0 + q < p.ny) {
                const size_t at_q = (size_t)(s.i0 + r) * p.ny + s.j0 + q;
                p.f[at_q] = rs_get(s.f[r], q);
                p.a[at_q] = rs_get(s.a[r], q);
                p.b[at_q] = rs_get(s.b[r], q);
            }
    res_copy_psi(p, s, tid, nt, true);
    if (c == 0) {
        const float *line = aux;
        for (int k = 0; k < p.n_tfsf; ++k) {
            const ResTfsf &t = p.tfsf[k];
            for (int q = tid; q < t.aux_n; q += nt) t.aux_e[q] = line[q], t.aux_h[q] = line[t.aux_n + q];
            line += 4 * t.aux_n;
        }
    }
}

// The kernels' shapes: C columns a thread, up to RT rows a strip, up to NT threads, in order of preference (fewest
// registers first).  The register file bounds them: NT threads have 65,536 / NT registers each (in steps of 128
// threads: 96 at 640, 128 at 512, 168 at 384, 255 at 256), of which 3 C RT hold fields and about 45 the rest.
// Four columns a thread run at about half the rate of two (fewer warps, spills).  Runs that the blocked kernels do not take
// (poles, plane-wave boxes: 30 to 60 us a step in launches per half step) use them; runs that those take do not.  With an
// earlier build's plain four-column kernels, us per step resident and blocked, E_z / H_z: up to 6 rows 530 x 1980 9.1, 13.0 /
// 12.6, 12.9 and 830 x 1430 12.6, 14.4 / 15.1, 17.8, from 8 rows 1130 x 1430 15.3, 14.4 and 1730 x 980 18.1, 13.0: a gain of up
// to 1.4 on strips of a few wide rows is left.
struct ResShape {
    int c, rt, nt;
    bool blocked_is_faster;
};
static constexpr ResShape RES_SHAPES[] = {
    {2, 4, 640, false}, {2, 8, 512, false}, {2, 8, 640, false}, {4, 4, 640, true},  {2, 16, 384, false},
    {4, 8, 512, true},  {2, 24, 256, false}, {4, 10, 384, true}, {4, 16, 256, true}};
static constexpr int RES_N_SHAPES = sizeof(RES_SHAPES) / sizeof(RES_SHAPES[0]);

template <bool HZ, bool GEN, int C, int RT, int NT>
static cudaError_t res_launch_kernel(const Res2DJob &job, size_t smem, cudaStream_t stream) {
    auto kernel = res2d_kernel<HZ, GEN, C, RT, NT>;
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    void *args[] = {const_cast<Res2DJob *>(&job)};
    return cudaLaunchCooperativeKernel((const void *)kernel, dim3((unsigned)job.n_cta),
                                       dim3((unsigned)res_threads(job.ny, C)), args, smem, stream);
}
template <bool HZ, bool GEN, int S>
static cudaError_t res_launch_shape(const Res2DJob &job, size_t smem, cudaStream_t stream) {
    constexpr ResShape sh = RES_SHAPES[S];
    if constexpr (!GEN && sh.blocked_is_faster) return cudaErrorInvalidValue;   // plain runs never ask for it
    else return res_launch_kernel<HZ, GEN, sh.c, sh.rt, sh.nt>(job, smem, stream);
}
template <bool HZ, bool GEN, int S = 0>
static cudaError_t res_launch_any(int shape, const Res2DJob &job, size_t smem, cudaStream_t stream) {
    if constexpr (S < RES_N_SHAPES) {
        if (shape == S) return res_launch_shape<HZ, GEN, S>(job, smem, stream);
        return res_launch_any<HZ, GEN, S + 1>(shape, job, smem, stream);
    } else {
        return cudaErrorInvalidValue;
    }
}
