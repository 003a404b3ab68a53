// Mamba-2 state step for state_rank 128 (bm_step2 and the decode chain).
#pragma once
#include "common.cuh"
#include "host/decode.h"

namespace bm {

// Where the step's dt comes from: float32 [b, h], or a column of the in-projection's rows.
struct DtDense {
    const float* dt;
    int nheads;
    __device__ __forceinline__ float load(int b, int h) const { return dt[(int64_t)b * nheads + h]; }
};
// Slices are summed in order, eight requested at a time (a loop over them waits on memory once per slice: 1.5 us of a
// 3-slice sum under load).
__device__ __forceinline__ float rows_value(const bmx_rows& r, int64_t row, int64_t col) {
    if (r.part == nullptr) return __bfloat162float(static_cast<const __nv_bfloat16*>(r.dense)[row * r.ld + col]);
    float v = 0.f;
    const float* p = r.part + row * r.ld + col;
    for (int s0 = 0; s0 < r.nslice; s0 += 8) {
        float t[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) t[i] = s0 + i < r.nslice ? p[(s0 + i) * r.slice] : 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) v += t[i];
    }
    return v;
}
struct DtRows {
    bmx_rows rows;
    int col;
    __device__ __forceinline__ float load(int b, int h) const { return rows_value(rows, b, col + h); }
};

__device__ __forceinline__ float4 step2_ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 step2_ld4(const __nv_bfloat16* p) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    return make_float4(a.x, a.y, b.x, b.y);
}

// Sums v[j] over the warp for NR values at once; lane l ends up with the sum of value l / (32 / NR) in v[0].  A lane keeps
// the half of its values whose index bit matches its own lane bit, then the plain butterfly runs inside the group.
template <int NR>
__device__ __forceinline__ void transposed_sum(float (&v)[NR], int lane) {
    int o = 16;
#pragma unroll
    for (int n = NR / 2; n >= 1; n >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int k = 0; k < n; ++k) {
            const float send = up ? v[k] : v[k + n], keep = up ? v[k + n] : v[k];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
#pragma unroll
    for (int q = 16 / NR; q >= 1; q >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], q);
}

// h = exp(dt A) h + dt x (x) B, y = C . h + D x (src/mamba2/mamba2.rs:907-991).  A lane owns four state columns; a warp
// holds NR rows, all of them requested before anything waits (they are this step's own: no kernel of a chain writes them
// before it).  The NR row sums are reduced together by a transposing butterfly.  Bound by HBM: the state in and out.
// NR = 8 (64 rows per CTA) when there are more (batch, head) pairs than SMs, else 2, which makes four times the CTAs.  bf16 P 64,
// 2 / 8 rows: 80 pairs 4.1 / 4.8 us, 128 5.3 / 6.2, 160 to 240 6.2 / 6.2, 288 7.0 / 6.3, 320 to 400 8.2 / 8.2, 1280 18.2 / 18.3.
template <typename T, int NR, typename DT>
__global__ void __launch_bounds__(256) step2_rows_kernel(bm_step2_args a, DT dtsrc, int nsplit) {
    constexpr int R = 128, G = 32 / NR;
    pdl_launch_dependents();
    const int sp = blockIdx.x % nsplit, bh = blockIdx.x / nsplit, b = bh / a.nheads, h = bh % a.nheads, P = a.headdim;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int p0 = (sp * 8 + warp) * NR;
    float* st = a.state + ((int64_t)bh * P + p0) * R + lane * 4;
    float4 hv[NR];
#pragma unroll
    for (int j = 0; j < NR; ++j)
        if (p0 + j < P) hv[j] = step2_ld4(st + j * R);
    const float ah = a.a[h], dskip = a.d ? a.d[h] : 0.f, bias = a.dt_bias ? a.dt_bias[h] : 0.f;
    pdl_wait();
    if (p0 >= P) return;
    const int64_t bc = ((int64_t)b * a.ngroups + h / (a.nheads / a.ngroups)) * R + lane * 4;
    const float4 bq = step2_ld4(static_cast<const T*>(a.b) + bc), cq = step2_ld4(static_cast<const T*>(a.c) + bc);
    const int myrow = lane / G;   // the row whose sum this lane ends up with
    const T* xv = static_cast<const T*>(a.x) + (int64_t)bh * P + p0;
    const float xl = p0 + myrow < P ? to_f32(xv[myrow]) : 0.f;
    float dt = dtsrc.load(b, h);
    if (a.dt_bias) dt = fminf(fmaxf(softplus_f32(dt + bias), a.dt_min), a.dt_max);
    const float da = expf(dt * ah), dtx = dt * xl;
    float v[NR];
#pragma unroll
    for (int j = 0; j < NR; ++j) {
        const float u = __shfl_sync(0xffffffffu, dtx, j * G);
        hv[j].x = fmaf(hv[j].x, da, u * bq.x);
        hv[j].y = fmaf(hv[j].y, da, u * bq.y);
        hv[j].z = fmaf(hv[j].z, da, u * bq.z);
        hv[j].w = fmaf(hv[j].w, da, u * bq.w);
        if (p0 + j < P) *reinterpret_cast<float4*>(st + j * R) = hv[j];
        v[j] = hv[j].x * cq.x + hv[j].y * cq.y + hv[j].z * cq.z + hv[j].w * cq.w;
    }
    transposed_sum<NR>(v, lane);
    if (lane % G == 0 && p0 + myrow < P) {
        float y = fmaf(dskip, xl, v[0]);
        const int64_t i = (int64_t)bh * P + p0 + myrow;
        if (a.z) y *= silu_f32(to_f32(static_cast<const T*>(a.z)[i]));
        static_cast<T*>(a.y)[i] = from_f32<T>(y);
    }
}

template <typename T, typename DT>
inline int32_t launch_step2_rows(const bm_step2_args& a, DT dt, bool chained, cudaStream_t st) {
    const int64_t bh = (int64_t)a.batch * a.nheads;
    const bool wave = bh > sm_count();
    const int nsplit = (int)cdiv(a.headdim, wave ? 64 : 16);
    const dim3 grid((unsigned)(bh * nsplit));
    if (wave) return launch_chained("step2", chained, grid, 256, 0, st, step2_rows_kernel<T, 8, DT>, a, dt, nsplit);
    return launch_chained("step2", chained, grid, 256, 0, st, step2_rows_kernel<T, 2, DT>, a, dt, nsplit);
}

}  // namespace bm
