/* Kernels of the fused decode step, called by the host path (native.cpp) only: not part of the C ABI of bm_b200.h.
 *
 * A Mamba-2 layer's step is a chain of short kernels on one stream,
 *     norm -> in-projection -> mixer (conv, state, gate) -> out-projection              up to a batch of 8, few (batch, head) pairs
 *     norm -> in-projection -> conv -> state -> gated norm -> out-projection            up to a batch of 8
 *     norm -> [library GEMM] -> conv -> state -> gated norm -> [library GEMM]           above
 * launched with programmatic dependent launch: a kernel starts while its predecessor runs, fetches what no kernel of the
 * chain writes (weights; its own state rows), and waits for the predecessor only then.  The first kernel of a chain is
 * launched plainly, so everything enqueued before the chain is complete when any kernel of it reads memory early.
 *
 * All tensors bf16 unless said otherwise; device pointers, 16-byte aligned rows. */
#ifndef BM_B200_DECODE_H
#define BM_B200_DECODE_H

#include <stdint.h>

#include "../../../include/bm_b200.h"

#ifdef __cplusplus
extern "C" {
#endif

/* Rows [batch, >= width] that a kernel consumes: either the partial sums a split projection left, float32
 * [nslice][batch][ld] (`part`), or dense bf16 rows (`dense`). */
typedef struct {
    const float* part;
    const void* dense;
    int32_t nslice;
    int32_t reserved;
    int64_t slice;   /* elements between slices */
    int64_t ld;      /* elements between rows */
} bmx_rows;

/* The mixer between two streaming projections (state_rank 128, 4 conv taps). */
typedef struct {
    int32_t batch, nheads, headdim, ngroups, norm_before_gate, nss, planes, reserved;
    float dt_min, dt_max;
    bmx_rows proj;         /* in-projection: z | x, B, C | dt */
    float* state;          /* [b, h, p, 128] in/out */
    float* window;         /* [b, v, 4] in/out */
    const float* conv_w;
    const float* conv_b;
    const float* a;
    const float* d;
    const float* dt_bias;
    const void* gamma;     /* [d_inner] weight of the gated norm */
    void* out;             /* [planes, b, d_inner]: gated y times gamma, without the norm's row scale */
    float* ss;             /* [b, nss] partial sums of squares that scale comes from */
} bmx_mixer;

/* Status of the chains on a device: zero until a bounded wait runs out.  The partial sums of the projection that gave up are
 * then NaN.  NULL (with the thread's error text set) when there is no such word. */
int32_t* bmx_chain_status(int32_t device);
/* Returns what the word holds as a status (BM_OK or an error, reported once) and clears it; does not synchronise. */
int32_t bmx_chain_take_status(int32_t* word);
/* Number of K slices the streaming projection cuts a [k, n] weight into for this batch; 0 = the shape is not covered. */
int32_t bmx_decode_slices(int32_t batch, int32_t k, int32_t n);
/* `first` below: the kernel opens a chain and is launched plainly.
 * Rows a streaming projection reads are [planes][batch][k]: with two planes, hi and lo bf16 halves of each value.
 * part[s][b][n] = sum over slice s of x[b, k] w[k, n].  `stall` (tests): issue no copies, so that the first wait runs out. */
int32_t bmx_decode_linear(const void* x, int32_t planes, const void* w, float* part, int32_t batch, int32_t k, int32_t n, int32_t nslice, int32_t* status,
                          int32_t first, int32_t stall, void* stream);
/* x' = residual (bf16 or float32) + add (any may be missing); x32 = x_out = x' and out = x' / rms(x') * gamma where the pointers are
 * given.  `prev`: the mixer step that `add` is the out-projection of (its row scale is applied, its B / C windows slide). */
int32_t bmx_decode_norm(const void* residual, const float* residual32, const bmx_rows* add, const bmx_mixer* prev, const void* gamma, float eps, float* x32,
                        void* x_out, void* out, int32_t planes, int32_t batch, int32_t width, int32_t first, void* stream);
int32_t bmx_decode_mixer_sums(int32_t batch, int32_t nheads, int32_t headdim);   /* nss of a mixer step; 0 = take the kernels apart */
int32_t bmx_decode_mixer(const bmx_mixer* a, void* stream);
/* bm_conv_step with its input read at column `col` of `in` */
int32_t bmx_decode_conv(const bm_conv_step_args* a, const bmx_rows* in, int32_t col, void* stream);
/* bm_step2 (state_rank 128) with dt read at column `col` of `in`; needs dt_bias */
int32_t bmx_decode_state(const bm_step2_args* a, const bmx_rows* in, int32_t col, void* stream);
/* bm_rmsnorm_gated of the dense rows a->x with z read at column 0 of `z` */
int32_t bmx_decode_gated_norm(const bm_rmsnorm_gated_args* a, const bmx_rows* z, int32_t planes, void* stream);

#ifdef __cplusplus
}
#endif
#endif
