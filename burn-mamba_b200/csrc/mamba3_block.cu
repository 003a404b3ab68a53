// Mamba-3 block around the SSD slot, float32 (csrc/host/mamba3.h): trapezoid coefficients and MIMO expansion, initial state,
// gate and down-projection of a prompt, and the whole step of one token between the two projections.
//
// Each replaces a run of elementwise passes over [b, s, m, h, p] or [b, h] tensors: 50 launches of a prompt became 4, 52 of a
// step became 1.  Measured: prompt b2 L389 d_model 1024 rank 4, the block 862 -> 566 us; step b64 at the same width 406 -> 119 us
// (52 us of it this step kernel: 134 MB of state in and out, bound by the latencies of its phases at two CTAs per SM).
#include "common.cuh"
#include "host/mamba3.h"
#include "step2.cuh"

#include <algorithm>

using namespace bm;

namespace {

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// A load that stays where it is written, ahead of the barriers, instead of at its use behind them.
__device__ __forceinline__ float ld_now(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

struct Columns {   // column offsets of the projection row
    int di, bc, x, b, c, dt, da, lam, rot, na;
    __device__ __forceinline__ explicit Columns(const bmx_m3_block& a) {
        di = a.nheads * a.headdim, bc = a.mimo_rank * a.ngroups * a.state_rank;
        x = di, b = 2 * di, c = b + bc, dt = c + bc, da = dt + a.nheads, lam = da + a.nheads, rot = lam + a.nheads;
        na = max(a.rope_dim / 2, 1);
    }
};
// Clamps that keep NaN, as the reference's do; fminf and fmaxf would drop it.
__device__ __forceinline__ float at_least(float x, float lo) { return x < lo ? lo : x; }
__device__ __forceinline__ float at_most(float x, float hi) { return x > hi ? hi : x; }

struct Trapezoid {   // src/mamba3/helpers.rs:42-73
    float dt, da, lam;
    __device__ __forceinline__ Trapezoid(const bmx_m3_block& a, float dd_dt, float dd_a, float lam_raw, float bias) {
        dt = at_most(at_least(softplus_f32(dd_dt + bias), a.dt_min), a.dt_max);
        da = -dt * at_least(softplus_f32(dd_a), a.a_floor);
        lam = 1.f / (1.f + expf(-lam_raw));
    }
};

// One CTA per token.  Waits on its loads (43 % of DRAM, b4 L1024 H32 rank 4).
__global__ void __launch_bounds__(256) m3_coefficients_kernel(bmx_m3_block a, float* dt, float* da, float* gamma, float* scale, float* v, float* rot) {
    const Columns col(a);
    const int64_t tok = blockIdx.x;
    const int s = tok % a.seqlen, H = a.nheads, P = a.headdim, M = a.mimo_rank;
    const float* row = a.proj + tok * a.ld;
    for (int h = threadIdx.x; h < H; h += blockDim.x) {
        const float bias = a.dt_bias[h];
        const Trapezoid t(a, row[col.dt + h], row[col.da + h], row[col.lam + h], bias);
        const float g = t.lam * t.dt;
        float sc = g;
        if (s + 1 < a.seqlen) {   // single_ssd/mod.rs:134-149
            const float* nx = row + a.ld;
            const Trapezoid u(a, nx[col.dt + h], nx[col.da + h], nx[col.lam + h], bias);
            sc += u.dt * (1.f - u.lam);
        }
        dt[tok * H + h] = t.dt, da[tok * H + h] = t.da, gamma[tok * H + h] = g, scale[tok * H + h] = sc;
    }
    for (int j = threadIdx.x; j < col.na; j += blockDim.x) rot[tok * col.na + j] = row[col.rot + j];
    for (int e = threadIdx.x * 4; e < col.di; e += blockDim.x * 4) {
        const float4 x = ld4(row + col.x + e);
        const int h = e / P, p = e - h * P;
        for (int m = 0; m < M; ++m) {
            float4 o = x;
            if (a.mimo_x) {
                const float4 w = ld4(a.mimo_x + ((int64_t)h * M + m) * P + p);
                o = make_float4(x.x * w.x, x.y * w.y, x.z * w.z, x.w * w.w);
            }
            *reinterpret_cast<float4*>(v + ((tok * M + m) * H + h) * P + p) = o;
        }
    }
}

// One CTA per (b, h).
__global__ void __launch_bounds__(256) m3_seed_kernel(bmx_m3_block a, const float* dt, const float* gamma, const float* ssm, const float* k, const float* v, float* h0) {
    const int bh = blockIdx.x, b = bh / a.nheads, h = bh % a.nheads, P = a.headdim, R = a.state_rank, M = a.mimo_rank;
    const int64_t t0 = (int64_t)b * a.seqlen * a.nheads + h;
    const float w = dt[t0] - gamma[t0];
    for (int e = threadIdx.x * 4; e < P * R; e += blockDim.x * 4) {
        const int p = e / R, r = e - p * R;
        float4 acc = ld4(ssm + (int64_t)bh * P * R + e);
        const float x = v[(int64_t)bh * P + p] * w;
        for (int m = 0; m < M; ++m) {
            const float c = a.mimo_x ? x * a.mimo_x[((int64_t)h * M + m) * P + p] : x;
            const float4 kq = ld4(k + (((int64_t)b * M + m) * a.nheads + h) * R + r);
            acc.x = fmaf(c, kq.x, acc.x), acc.y = fmaf(c, kq.y, acc.y), acc.z = fmaf(c, kq.z, acc.z), acc.w = fmaf(c, kq.w, acc.w);
        }
        *reinterpret_cast<float4*>(h0 + (int64_t)bh * P * R + e) = acc;
    }
}

__device__ __forceinline__ float gated(float y, float x, float d, float z, float mx, float mz, float mo) {
    return fmaf(d, x * mx, y) * silu_f32(z * mz) * mo;
}

// One CTA per token: src/mamba3/single_ssd/single_ssd/mod.rs:291-337.  The gates take 59 % of the issue
// slots (36 % of DRAM, b4 L1024 H32 rank 4).
__global__ void __launch_bounds__(256) m3_tail_kernel(bmx_m3_block a, const float* y, const float* b_rot, float* out, float* k_last, float* v_last) {
    const Columns col(a);
    const int64_t tok = blockIdx.x, b = tok / a.seqlen;
    const int H = a.nheads, P = a.headdim, M = a.mimo_rank;
    const bool last = tok % a.seqlen == a.seqlen - 1;
    const float* row = a.proj + tok * a.ld;
    const float4 one = make_float4(1.f, 1.f, 1.f, 1.f);
    for (int e = threadIdx.x * 4; e < col.di; e += blockDim.x * 4) {
        const int h = e / P, p = e - h * P;
        const float4 z = ld4(row + e), x = ld4(row + col.x + e);
        const float d = a.d[h];
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int m = 0; m < M; ++m) {
            const int64_t w = ((int64_t)h * M + m) * P + p;
            const float4 yq = ld4(y + ((tok * M + m) * H + h) * P + p), mx = a.mimo_x ? ld4(a.mimo_x + w) : one;
            const float4 mz = M > 1 ? ld4(a.mimo_z + w) : one, mo = M > 1 ? ld4(a.mimo_o + w) : one;
            o.x += gated(yq.x, x.x, d, z.x, mx.x, mz.x, mo.x);
            o.y += gated(yq.y, x.y, d, z.y, mx.y, mz.y, mo.y);
            o.z += gated(yq.z, x.z, d, z.z, mx.z, mz.z, mo.z);
            o.w += gated(yq.w, x.w, d, z.w, mx.w, mz.w, mo.w);
        }
        *reinterpret_cast<float4*>(out + tok * col.di + e) = o;
        if (last) *reinterpret_cast<float4*>(v_last + b * col.di + e) = x;
    }
    if (last) {
        const int64_t n = (int64_t)M * H * a.state_rank;
        for (int64_t e = threadIdx.x * 4; e < n; e += blockDim.x * 4) *reinterpret_cast<float4*>(k_last + b * n + e) = ld4(b_rot + tok * n + e);
    }
}

// ---------------------------------------------------------------------------------------------------------------
// The step between the projections (src/mamba3/double_ssd/double_ssd/mod.rs:635-760): coefficients, QK-norm and bias,
// rotation by the new angle, state update and readout, D skip, gate, MIMO down-projection, cache roll.  A lane owns four
// state columns, a warp holds NR rows (all requested first) and sums its NR M readouts with one transposing butterfly.
// NR = 8: one CTA per (b, h).  NR = 2, while the pairs are at most one per two SMs: a cluster of P / 16 CTAs, which all read the
// caches they share (k, angle) before the first rolls them.  Whole step, 2 / 8 rows, rank 4 N 128: 32 pairs 21.5 / 21.7 us, 64 53.1 /
// 53.8 (d_model 1024) and 22.5 / 23.5 (d_model 256); 80 30.8 / 27.5, 96 42.4 / 38.3, 128 44.5 / 40.4, 160 51.2 / 43.1, 256 62.5 /
// 48.4: from there on the clusters repeat the preparation of B and C for nothing.
// ---------------------------------------------------------------------------------------------------------------
template <int M, int NR>
__global__ void __launch_bounds__(256, 2) m3_step_kernel(bmx_m3_block a, float* state, float* k_state, float* v_state, float* angle, float* out, int nsplit) {
    extern __shared__ __align__(16) float sm[];
    const Columns col(a);
    const int R = a.state_rank, P = a.headdim, H = a.nheads, na = a.rope_dim / 2, nal = col.na;
    const int sp = blockIdx.x % nsplit, bh = blockIdx.x / nsplit, b = bh / H, h = bh % H, g = h / (H / a.ngroups);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r4 = lane * 4;
    float* cosv = sm;                                  // [nal]
    float* sinv = cosv + ((nal + 3) & ~3);             // [nal]
    float* braw = sinv + ((nal + 3) & ~3);             // [2][M][R] normed and biased B, then C
    float* rot = braw + 2 * M * R;                     // [2][M][R] rotated
    float* bp = rot + 2 * M * R;                       // [M][R] previous rotated B
    const float* row = a.proj + (int64_t)b * a.ld;
    const bool act = r4 < R;
    const int p0 = (sp * 8 + warp) * NR;
    float* st = state + ((int64_t)bh * P + p0) * R + r4;
    float4 hv[NR];
#pragma unroll
    for (int j = 0; j < NR; ++j) hv[j] = (p0 + j < P && act) ? ld4(st + (int64_t)j * R) : make_float4(0.f, 0.f, 0.f, 0.f);
    // per-row scalars: lane j holds those of row p0 + j
    const int prow = p0 + (lane & (NR - 1));
    const bool plive = prow < P;
    const float xl = plive ? ld_now(row + col.x + h * P + prow) : 0.f;
    const float xpl = plive ? v_state[(int64_t)bh * P + prow] : 0.f;
    float mxl[M];
#pragma unroll
    for (int m = 0; m < M; ++m) mxl[m] = plive && a.mimo_x ? a.mimo_x[((int64_t)h * M + m) * P + prow] : 1.f;
    // what the lane that ends up with (row, m) needs for the tail
    constexpr int NV = NR * M, GRP = 32 / NV;
    const int trow = lane / GRP / M, tm = lane / GRP % M, tp = p0 + trow;
    float tz = 0.f, tmx = 1.f, tmz = 1.f, tmo = 1.f;
    if (tp < P) {
        const int64_t w = ((int64_t)h * M + tm) * P + tp;
        tz = ld_now(row + h * P + tp);
        if (a.mimo_x) tmx = a.mimo_x[w];
        if (M > 1) tmz = a.mimo_z[w], tmo = a.mimo_o[w];
    }
    // step b64 H32 rank 4, in turns: these as plain loads 123.1 us, held here 119.0
    const Trapezoid t(a, ld_now(row + col.dt + h), ld_now(row + col.da + h), ld_now(row + col.lam + h), a.dt_bias[h]);
    const float alpha = expf(t.da), beta = (1.f - t.lam) * t.dt * alpha, gamma = t.lam * t.dt;
    // raw B / C rows of the head's group, one warp per row: RMS norm over r, + bias (src/mamba3/helpers.rs:82-95)
    for (int rw = warp; rw < 2 * M; rw += 8) {
        const int isc = rw / M, m = rw % M;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (act) v = ld4(row + (isc ? col.c : col.b) + (m * a.ngroups + g) * R + r4);
        float ss = v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        const float inv = 1.f / sqrtf(ss / (float)R + a.eps);
        if (act) {
            const float4 w = ld4((isc ? a.c_norm : a.b_norm) + r4), bi = ld4((isc ? a.c_bias : a.b_bias) + ((int64_t)h * M + m) * R + r4);
            *reinterpret_cast<float4*>(braw + rw * R + r4) = make_float4(fmaf(v.x * inv, w.x, bi.x), fmaf(v.y * inv, w.y, bi.y),
                                                                         fmaf(v.z * inv, w.z, bi.z), fmaf(v.w * inv, w.w, bi.w));
        }
    }
    for (int m = warp; m < M; m += 8)
        if (act) *reinterpret_cast<float4*>(bp + m * R + r4) = ld4(k_state + (((int64_t)b * M + m) * H + h) * R + r4);
    // angle := wrap(angle + dt range pi tanh(rot)) (src/mamba3/rotation/mod.rs:559-567, :744-747)
    float th = 0.f;
    const bool ang = tid < nal;   // nal <= 64
    if (ang) {
        th = wrap_angle(angle[(int64_t)bh * nal + tid] + t.dt * (tanhf(ld_now(row + col.rot + tid)) * (a.range * 3.14159265358979323846f)));
        sincosf(th, &sinv[tid], &cosv[tid]);
    }
    __syncthreads();
    // rotation of the leading rope_dim entries, pairs (2j, 2j + 1) for rank 1, halves otherwise (src/modules/misc/rope.rs:50-170)
    for (int e = tid; e < 2 * M * (R / 2); e += 256) {
        const int rw = e / (R / 2), j = e - rw * (R / 2);
        const int lo = M == 1 ? 2 * j : j, hi = M == 1 ? 2 * j + 1 : j + R / 2;
        const float* src = braw + rw * R;
        float x = src[lo], y = src[hi];
        if (j < na) {
            const float c = cosv[j], s = sinv[j], u = c * x - s * y;
            y = s * x + c * y;
            x = u;
        }
        rot[rw * R + lo] = x, rot[rw * R + hi] = y;
    }
    __syncthreads();
    float4 bq[M], cq[M], pq[M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
        bq[m] = act ? ld4(rot + m * R + r4) : z4;
        cq[m] = act ? ld4(rot + (M + m) * R + r4) : z4;
        pq[m] = act ? ld4(bp + m * R + r4) : z4;
    }
    float gl[M], btl[M];
#pragma unroll
    for (int m = 0; m < M; ++m) gl[m] = gamma * xl * mxl[m], btl[m] = beta * xpl * mxl[m];
    float v[NV];
#pragma unroll
    for (int j = 0; j < NR; ++j) {
        float4 q = make_float4(alpha * hv[j].x, alpha * hv[j].y, alpha * hv[j].z, alpha * hv[j].w);
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const float gg = __shfl_sync(0xffffffffu, gl[m], j), bt = __shfl_sync(0xffffffffu, btl[m], j);
            q.x = fmaf(gg, bq[m].x, fmaf(bt, pq[m].x, q.x));
            q.y = fmaf(gg, bq[m].y, fmaf(bt, pq[m].y, q.y));
            q.z = fmaf(gg, bq[m].z, fmaf(bt, pq[m].z, q.z));
            q.w = fmaf(gg, bq[m].w, fmaf(bt, pq[m].w, q.w));
        }
        if (p0 + j < P && act) *reinterpret_cast<float4*>(st + (int64_t)j * R) = q;
#pragma unroll
        for (int m = 0; m < M; ++m) v[j * M + m] = q.x * cq[m].x + q.y * cq[m].y + q.z * cq[m].z + q.w * cq[m].w;
    }
    transposed_sum<NV>(v, lane);   // lane: y[trow][tm]
    const float tx = __shfl_sync(0xffffffffu, xl, trow);
    float o = gated(v[0], tx, a.d[h], tz, tmx, tmz, tmo);
#pragma unroll
    for (int q = GRP; q < GRP * M; q <<= 1) o += __shfl_xor_sync(0xffffffffu, o, q);   // over m
    if (tm == 0 && lane % GRP == 0 && tp < P) out[(int64_t)bh * P + tp] = o;
    if (plive && lane < NR) v_state[(int64_t)bh * P + prow] = xl;
    // cache roll, after every CTA of the pair has read k and angle
    if (nsplit > 1) {
        asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
        if (sp) return;
    }
#pragma unroll
    for (int m = 0; m < M; ++m)
        if (warp == m && act) *reinterpret_cast<float4*>(k_state + (((int64_t)b * M + m) * H + h) * R + r4) = bq[m];
    if (ang) angle[(int64_t)bh * nal + tid] = th;
}

template <int M>
int32_t launch_step(const bmx_m3_block& a, float* state, float* k_state, float* v_state, float* angle, float* out, cudaStream_t st) {
    const int64_t bh = (int64_t)a.batch * a.nheads;
    const int nal = std::max(a.rope_dim / 2, 1);
    const size_t smem = sizeof(float) * (size_t)(2 * ((nal + 3) & ~3) + 5 * M * a.state_rank);
    const bool wave = bh > sm_count() / 2;
    const int nsplit = (int)cdiv(a.headdim, wave ? 64 : 16);
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = nsplit, at.val.clusterDim.y = 1, at.val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(bh * nsplit)), cfg.blockDim = 256, cfg.dynamicSmemBytes = smem, cfg.stream = st, cfg.attrs = &at, cfg.numAttrs = nsplit > 1;
    return check_cuda(wave ? cudaLaunchKernelEx(&cfg, m3_step_kernel<M, 8>, a, state, k_state, v_state, angle, out, nsplit)
                           : cudaLaunchKernelEx(&cfg, m3_step_kernel<M, 2>, a, state, k_state, v_state, angle, out, nsplit),
                      "m3_step");
}

unsigned tokens(const bmx_m3_block* a) { return (unsigned)((int64_t)a->batch * a->seqlen); }

// The block's own pointers; a kernel's other operands are checked where it is launched.
int32_t check_block(const bmx_m3_block* a) {
    BM_REQUIRE_PTR(a->proj);
    BM_REQUIRE_PTR(a->dt_bias);
    BM_REQUIRE_PTR(a->d);
    BM_REQUIRE_PTR(a->b_norm);
    BM_REQUIRE_PTR(a->c_norm);
    BM_REQUIRE_PTR(a->b_bias);
    BM_REQUIRE_PTR(a->c_bias);
    BM_OPTIONAL_PTR(a->mimo_x);
    if (a->mimo_rank > 1) {
        BM_REQUIRE_PTR(a->mimo_z);
        BM_REQUIRE_PTR(a->mimo_o);
    }
    return BM_OK;
}

}  // namespace

extern "C" int32_t bmx_m3_coefficients(const bmx_m3_block* a, float* dt, float* da, float* gamma, float* scale, float* v, float* rot, void* stream) {
    if (int32_t e = check_block(a)) return e;
    BM_REQUIRE_PTR(dt);
    BM_REQUIRE_PTR(da);
    BM_REQUIRE_PTR(gamma);
    BM_REQUIRE_PTR(scale);
    BM_REQUIRE_PTR(v);
    BM_REQUIRE_PTR(rot);
    m3_coefficients_kernel<<<tokens(a), 256, 0, static_cast<cudaStream_t>(stream)>>>(*a, dt, da, gamma, scale, v, rot);
    return check_launch("m3_coefficients");
}
extern "C" int32_t bmx_m3_seed(const bmx_m3_block* a, const float* dt, const float* gamma, const float* ssm, const float* k, const float* v, float* h0,
                               void* stream) {
    if (int32_t e = check_block(a)) return e;
    BM_REQUIRE_PTR(dt);
    BM_REQUIRE_PTR(gamma);
    BM_REQUIRE_PTR(ssm);
    BM_REQUIRE_PTR(k);
    BM_REQUIRE_PTR(v);
    BM_REQUIRE_PTR(h0);
    m3_seed_kernel<<<(unsigned)((int64_t)a->batch * a->nheads), 256, 0, static_cast<cudaStream_t>(stream)>>>(*a, dt, gamma, ssm, k, v, h0);
    return check_launch("m3_seed");
}
extern "C" int32_t bmx_m3_tail(const bmx_m3_block* a, const float* y, const float* b_rot, float* out, float* k_last, float* v_last, void* stream) {
    if (int32_t e = check_block(a)) return e;
    BM_REQUIRE_PTR(y);
    BM_REQUIRE_PTR(b_rot);
    BM_REQUIRE_PTR(out);
    BM_REQUIRE_PTR(k_last);
    BM_REQUIRE_PTR(v_last);
    m3_tail_kernel<<<tokens(a), 256, 0, static_cast<cudaStream_t>(stream)>>>(*a, y, b_rot, out, k_last, v_last);
    return check_launch("m3_tail");
}
// State rows of at most 128 columns in whole 16-byte vectors, at most 64 head columns (one CTA, or a portable cluster).
extern "C" int32_t bmx_m3_step_covers(const bmx_m3_block* a) {
    const int m = a->mimo_rank;
    return (m == 1 || m == 2 || m == 4) && a->state_rank % 4 == 0 && a->state_rank <= 128 && a->headdim <= 64 && a->rope_dim <= a->state_rank;
}
extern "C" int32_t bmx_m3_step(const bmx_m3_block* a, float* state, float* k_state, float* v_state, float* angle, float* out, void* stream) {
    if (int32_t e = check_block(a)) return e;
    BM_REQUIRE_PTR(state);
    BM_REQUIRE_PTR(k_state);
    BM_REQUIRE_PTR(v_state);
    BM_REQUIRE_PTR(angle);
    BM_REQUIRE_PTR(out);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    switch (a->mimo_rank) {
        case 1: return launch_step<1>(*a, state, k_state, v_state, angle, out, st);
        case 2: return launch_step<2>(*a, state, k_state, v_state, angle, out, st);
        default: return launch_step<4>(*a, state, k_state, v_state, angle, out, st);
    }
}
