/* Kernels of the Mamba-3 block around its SSD slot (float32), called by the host path (native.cpp) only: not part of the C ABI. */
#ifndef BM_B200_MAMBA3_HOST_H
#define BM_B200_MAMBA3_HOST_H

#include <stdint.h>

#include "../../../include/bm_b200.h"

#ifdef __cplusplus
extern "C" {
#endif

/* The block's dimensions and the small parameters its kernels read.  In-projection columns, in order:
 * z (h p) | x (h p) | B (m g r) | C (m g r) | dd_dt (h) | dd_A (h) | lambda (h) | rot (max(rope_dim / 2, 1)). */
typedef struct {
    int32_t batch, seqlen, nheads, headdim, state_rank, ngroups, mimo_rank, rope_dim;
    float range, dt_min, dt_max, a_floor, eps;
    int64_t ld;            /* elements between projection rows */
    const float* proj;
    const float* dt_bias;  /* [h] */
    const float* d;        /* [h] */
    const float* b_norm;   /* [r] */
    const float* c_norm;
    const float* b_bias;   /* [h, m, r] */
    const float* c_bias;
    const float* mimo_x;   /* [h, m, p] or NULL (ones) */
    const float* mimo_z;   /* [h, m, p], read when mimo_rank > 1 */
    const float* mimo_o;
} bmx_m3_block;

/* Per token: dt, da = dt A, gamma, scale [b, s, h] (scale_t = gamma_t + (1 - lambda_{t+1}) dt_{t+1}), v = x mimo_x [b, s, m, h, p], rot [b, s, a]. */
int32_t bmx_m3_coefficients(const bmx_m3_block* a, float* dt, float* da, float* gamma, float* scale, float* v, float* rot, void* stream);
/* h0 = ssm + (dt_0 - gamma_0) sum_m (v mimo_x_m) (x) k_m */
int32_t bmx_m3_seed(const bmx_m3_block* a, const float* dt, const float* gamma, const float* ssm, const float* k, const float* v, float* h0, void* stream);
/* D skip, gate and MIMO down-projection of y [b, s, m, h, p] -> out [b, s, h p]; also the last token's rotated B -> k_last and x -> v_last. */
int32_t bmx_m3_tail(const bmx_m3_block* a, const float* y, const float* b_rot, float* out, float* k_last, float* v_last, void* stream);
/* One token from the projection row to the out-projection's input [b, h p], caches updated in place; 0 = shape not covered. */
int32_t bmx_m3_step_covers(const bmx_m3_block* a);
int32_t bmx_m3_step(const bmx_m3_block* a, float* state, float* k_state, float* v_state, float* angle, float* out, void* stream);

#ifdef __cplusplus
}
#endif
#endif
