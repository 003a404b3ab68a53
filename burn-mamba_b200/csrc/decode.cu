// Decode-step kernels of the Mamba-2 layer chain (csrc/host/decode.h): the streaming projection for small batches, and
// the norm, conv, state and gated-norm steps that read its partial sums.
//
// What bounds a step at batch 1 is the weights: 80 MB per layer at d_model 2560, 12.5 us of HBM time, against 43 us for
// library products that start cold after every small kernel.  The projection kernel's CTAs fetch their first weights, as
// many as an SM's shared memory holds, while the kernels before them still run.  Measured, 8 layers at d_model 2560 and
// batch 1: 536 us with library products and plain launches, 232 us as this chain (29 us per layer; what is left besides
// the 12.5 us of streaming is four dependent kernels' latencies).  Batch 256, 4 layers: 1187 -> 990 us (the state kernel's
// 8 rows in flight per warp 226 -> 195 us per layer, 6.9 TB/s; no dt cast, no residual copy, no launch gaps).
#include "common.cuh"
#include "host/decode.h"
#include "step2.cuh"
#include "tc_common.cuh"

#include <algorithm>
#include <mutex>

using namespace bm;

namespace {

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
                     tc::smem_u32(dst)),
                 "l"(m), "r"(tc::smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
                     tc::smem_u32(dst)),
                 "l"(m), "r"(tc::smem_u32(bar)), "r"(c0), "r"(c1)
                 : "memory");
}

// ---------------------------------------------------------------------------------------------------------------
// Streaming projection.  out^T = W^T x^T: a CTA takes 128 output columns and one slice of K, the weight tile is the
// MN-major A operand (128 columns x 64 k, straight from the row-major [k, n] weight by TMA), the batch rows are the
// K-major B operand (16 of them, those past the batch zero-filled by the copy), the accumulator sits in TMEM with one output
// column per lane.  Slices are summed by whoever reads the result, so no CTA waits on another.
// With two planes the batch rows come as bf16 pairs hi + lo (16 bits of the float32 value): the accumulator columns of both
// are summed on the way out.  The second plane is free: its rows would be padding.
// 2 bytes of weight per `batch` multiply-adds: HBM is its floor.  Alone and cold it reaches 3.5 TB/s (54 MB in 15.6 us), the rest
// is launch, descriptor fetch and first copies, which the chain puts under the kernels before it.  All of an SM's shared memory is weight stages of 16 KB: two
// CTAs with 6 of them, or one with 12 where one CTA per SM covers the weight with fewer slices to sum.
// ---------------------------------------------------------------------------------------------------------------
constexpr int kLinCols = 128, kLinK = 64, kLinThreads = 128;
constexpr int kLinWBytes = kLinCols * kLinK * 2;
constexpr int kLinRows = 16, kLinStageBytes = kLinWBytes + kLinRows * kLinK * 2;
__host__ __device__ constexpr int lin_stages(bool deep) { return deep ? 12 : 6; }

// false when the budget ran out
__device__ __forceinline__ bool wait_bounded(uint64_t* bar, uint32_t parity) {
    for (uint32_t n = 0; n < tc::kWaitBudget; ++n)
        if (tc::mbar_try_wait(bar, parity)) return true;
    return false;
}

template <bool DEEP, int PLANES>
__global__ void __launch_bounds__(kLinThreads) decode_linear_kernel(const __grid_constant__ CUtensorMap mw, const __grid_constant__ CUtensorMap mx,
                                                                    float* part, int batch, int n, int kblocks, int nslice, volatile int32_t* status,
                                                                    int stall) {
    constexpr int ST = lin_stages(DEEP), SB = kLinStageBytes, TCOLS = 32;   // the smallest TMEM allocation
    extern __shared__ __align__(1024) unsigned char raw[];
    unsigned char* base = raw + ((1024u - (tc::smem_u32(raw) & 1023u)) & 1023u);
    __shared__ uint64_t full[ST], empty[ST], done;
    __shared__ uint32_t tmem_slot;
    __shared__ int gave_up, loads;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int col0 = blockIdx.x * kLinCols, s = blockIdx.y;
    const int kb0 = (int)((int64_t)kblocks * s / nslice), nkb = (int)((int64_t)kblocks * (s + 1) / nslice) - kb0;
    pdl_launch_dependents();
    if (tid == 0) {
        for (int i = 0; i < ST; ++i) tc::mbar_init(&full[i], 1), tc::mbar_init(&empty[i], 1);
        tc::mbar_init(&done, 1);
        gave_up = 0;
        tc::fence_mbar_init();
        tc::tma_prefetch_desc(&mw);
        tc::tma_prefetch_desc(&mx);
    }
    if (warp == 1) {
        tc::tmem_alloc(&tmem_slot, TCOLS);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tmem_slot;
    if (tid == 0) {
        auto load_w = [&](int i) {
            unsigned char* st = base + (i % ST) * SB;
            tc::mbar_expect_tx(&full[i % ST], SB);
            tma_load_2d(st, &mw, &full[i % ST], col0, (kb0 + i) * kLinK);
            tma_load_2d(st + kLinWBytes / 2, &mw, &full[i % ST], col0 + 64, (kb0 + i) * kLinK);
        };
        auto load_x = [&](int i) { tma_load_3d(base + (i % ST) * SB + kLinWBytes, &mx, &full[i % ST], (kb0 + i) * kLinK, 0, 0); };
        const int pre = stall ? 0 : min(ST, nkb);
        for (int i = 0; i < pre; ++i) load_w(i);   // weights: nothing in the chain writes them
        pdl_wait();                                // x: the predecessor does
        asm volatile("fence.proxy.async;" ::: "memory");
        for (int i = 0; i < pre; ++i) load_x(i);
        bool ok = !stall;
        int issued = pre;
        for (int i = ST; ok && i < nkb; ++i) {
            ok = wait_bounded(&empty[i % ST], (i / ST - 1) & 1);
            if (ok) load_w(i), load_x(i), ++issued;
        }
        if (!ok) gave_up = 1;
        loads = issued;
    } else if (tid == 32) {
        const uint32_t idesc = tc::umma_idesc_bf16(kLinCols, kLinRows, true, false);
        bool ok = true;
        pdl_wait();   // before the bounded waits: the predecessor's time is not theirs
        for (int i = 0; ok && i < nkb; ++i) {
            ok = wait_bounded(&full[i % ST], (i / ST) & 1);
            if (!ok) break;
            tc::tc_fence_after();
            const uint32_t st = tc::smem_u32(base + (i % ST) * SB);
            const uint64_t da = tc::umma_desc_mnmajor(st, kLinWBytes / 2), db = tc::umma_desc_kmajor(st + kLinWBytes);
#pragma unroll
            for (int kk = 0; kk < kLinK / 16; ++kk)
                tc::umma_ss(tmem, tc::desc_advance(da, kk * 2048), tc::desc_advance(db, kk * 32), idesc, i > 0 || kk > 0);
            tc::umma_commit(&empty[i % ST]);
        }
        if (!ok) gave_up = 1;
        tc::umma_commit(&done);
    }
    __syncwarp();
    pdl_wait();
    const bool landed = __syncthreads_and(wait_bounded(&done, 0));   // one answer for the CTA
    if (landed && !gave_up) {
        tc::tc_fence_after();
        const int c = col0 + tid;
        uint32_t r[16];
        tc::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16), r);
        tc::tmem_wait_ld();
        if (c < n) {
            float* o = part + (int64_t)s * batch * n + c;
            constexpr int ROWS = kLinRows / PLANES;
#pragma unroll
            for (int j = 0; j < ROWS; ++j)
                if (j < batch) o[(int64_t)j * n] = __uint_as_float(r[j]) + (PLANES == 2 ? __uint_as_float(r[(ROWS + j) & 15]) : 0.f);
        }
    } else {
        // What this CTA owes is NaN, so that nothing downstream passes for a result, and the host's status word says why.
        const int c = col0 + tid;
        if (c < n)
            for (int j = 0; j < batch; ++j) part[((int64_t)s * batch + j) * n + c] = __int_as_float(0x7fffffff);
        if (tid == 0) {
            *status = BM_ERR_TIMEOUT;
            __threadfence_system();
            // copies in flight land in this CTA's shared memory: wait for the last one of every stage (bounded) before it is
            // given back
            for (int i = max(0, loads - ST); i < loads; ++i) wait_bounded(&full[i % ST], (i / ST) & 1);
        }
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 1) tc::tmem_dealloc(tmem, TCOLS);
}

// ---------------------------------------------------------------------------------------------------------------
// Row kernels.  One CTA per batch row, one 8-wide vector per thread (rows up to 8192 wide).
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void unpack8(const uint4& w, float (&v)[8]) {
    const uint32_t q[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&q[j]));
        v[2 * j] = f.x, v[2 * j + 1] = f.y;
    }
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
    return make_uint4(tc::pack_bf16x2(v[0], v[1]), tc::pack_bf16x2(v[2], v[3]), tc::pack_bf16x2(v[4], v[5]), tc::pack_bf16x2(v[6], v[7]));
}
// Eight columns of a row: the sum of the slices, or the dense values.
__device__ __forceinline__ void rows_load8(const bmx_rows& r, int64_t row, int c, float (&v)[8]) {
    if (r.part == nullptr) {
        unpack8(*reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(r.dense) + row * r.ld + c), v);
        return;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 0.f;
    const float* p = r.part + row * r.ld + c;
    for (int s0 = 0; s0 < r.nslice; s0 += 4) {   // four slices requested at a time
        float4 a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            a[i] = b[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (s0 + i < r.nslice) a[i] = step2_ld4(p + (s0 + i) * r.slice), b[i] = step2_ld4(p + (s0 + i) * r.slice + 4);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[0] += a[i].x, v[1] += a[i].y, v[2] += a[i].z, v[3] += a[i].w;
            v[4] += b[i].x, v[5] += b[i].y, v[6] += b[i].z, v[7] += b[i].w;
        }
    }
}
// Stores eight values as bf16 and, with a second plane (`lo`, elements further on; 0 = none), what the rounding left.
__device__ __forceinline__ void store_planes(__nv_bfloat16* dst, int64_t lo, float (&v)[8]) {
    const uint4 hi = pack8(v);
    *reinterpret_cast<uint4*>(dst) = hi;
    if (lo > 0) {
        float h[8];
        unpack8(hi, h);
#pragma unroll
        for (int j = 0; j < 8; ++j) h[j] = v[j] - h[j];
        *reinterpret_cast<uint4*>(dst + lo) = pack8(h);
    }
}
__device__ __forceinline__ float block_sum(float v) {
    __shared__ float red[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = 0.f;
    for (int i = 0; i < (int)((blockDim.x + 31) >> 5); ++i) v += red[i];
    return v;
}

// x' = residual + add; x_out = x'; out = x' / sqrt(mean(x'^2) + eps) * gamma  (src/modules/layer.rs:224-229 around
// src/modules/norm/rms_norm.rs:53-98).  `prev`, the mixer step whose out-projection `add` is: its gated norm's row scale
// is applied to the sums here, and its B / C conv windows slide here, after every reader of the old ones.  Between the
// layers of a chain the residual stream stays float32 (`x32`), so that a layer adds two bf16 roundings (the operands of its
// projections) to it and not six.
__global__ void __launch_bounds__(1024) decode_norm_kernel(const __nv_bfloat16* residual, const float* residual32, bmx_rows add, int has_add, bmx_mixer prev,
                                                           int has_prev, const __nv_bfloat16* gamma, float eps, float* x32, __nv_bfloat16* x_out,
                                                           __nv_bfloat16* out, int64_t out_lo, int width) {
    pdl_launch_dependents();
    const int64_t row = blockIdx.x;
    const int c = threadIdx.x * 8;
    const bool live = c < width;
    uint4 graw = make_uint4(0, 0, 0, 0);
    if (live && gamma) graw = *reinterpret_cast<const uint4*>(gamma + c);
    pdl_wait();
    float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, v[8];
    if (live) {
        if (residual) unpack8(*reinterpret_cast<const uint4*>(residual + row * width + c), x);
        if (residual32) {
            const float4 a = step2_ld4(residual32 + row * width + c), b = step2_ld4(residual32 + row * width + c + 4);
            x[0] = a.x, x[1] = a.y, x[2] = a.z, x[3] = a.w, x[4] = b.x, x[5] = b.y, x[6] = b.z, x[7] = b.w;
        }
        if (has_add) rows_load8(add, row, c, v);
    }
    float scale = 1.f;
    const int di = prev.nheads * prev.headdim, gr = 2 * prev.ngroups * 128;
    if (has_prev) {
        float ss = 0.f;
        for (int i = threadIdx.x; i < prev.nss; i += blockDim.x) ss += prev.ss[row * prev.nss + i];
        scale = rsqrtf(block_sum(ss) / (float)di + eps);
        __syncthreads();   // block_sum's scratch is used again below
    }
    if (live) {
        if (has_add) {
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = fmaf(v[j], scale, x[j]);
        }
        if (x_out) *reinterpret_cast<uint4*>(x_out + row * width + c) = pack8(x);
        if (x32) {
            *reinterpret_cast<float4*>(x32 + row * width + c) = make_float4(x[0], x[1], x[2], x[3]);
            *reinterpret_cast<float4*>(x32 + row * width + c + 4) = make_float4(x[4], x[5], x[6], x[7]);
        }
    }
    if (out != nullptr) {
        float ss = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) ss = fmaf(x[j], x[j], ss);
        const float inv = rsqrtf(block_sum(ss) / (float)width + eps);
        if (live) {
            float g[8];
            unpack8(graw, g);
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = x[j] * inv * g[j];
            store_planes(out + row * width + c, out_lo, x);
        }
    }
    if (has_prev)
        for (int i = threadIdx.x; i < gr; i += blockDim.x) {
            float4* win = reinterpret_cast<float4*>(prev.window + (row * (di + gr) + di + i) * 4);
            const float4 w = *win;
            *win = make_float4(w.y, w.z, w.w, rows_value(prev.proj, row, 2 * di + i));
        }
}

// The mixer's step between its two streaming projections: causal conv of this token, state update and readout, gate, and
// the gated norm up to its row scale, which is a factor of every output column and is applied to the out-projection's sums
// (decode_norm_kernel).  CTA = 16 rows of one (batch, head).  The x channels' windows slide here; those of B / C have a
// reader in every head and slide later.  State, windows and taps are fetched before the wait.
// Taken while the (batch, head) pairs are fewer than two per SM.  It leaves the conv outputs and y in float32, where the kernels
// apart round them to bf16 (error of a step against float64 1.7e-3 against 3.0e-3, of which the bf16 output is 1.6e-3), and it is
// three launches in one.  That is faster only with very few pairs, since every head redoes the conv of B / C: per layer, this
// / apart: 80 pairs 29.6 / 31.5 us (d_model 2560, b1); 128 22.9 / 21.7, 144 26.6 / 25.3, 192 24.7 / 22.4, 240 38.2 / 35.8, 288
// 31.2 / 28.5; 320 39.3 / 36.3, 640 53.6 / 39.9.  So from about 100 pairs on the precision is paid for with 5 to 16 % of a layer's
// time up to the line, and would be with up to a third above it.
constexpr int kMixRows = 16;
__global__ void __launch_bounds__(256) decode_mixer_kernel(bmx_mixer a, int nsplit) {
    constexpr int R = 128, NR = kMixRows / 8, G = 32 / NR;
    __shared__ float bc[2 * R], red[8];
    pdl_launch_dependents();
    const int sp = blockIdx.x % nsplit, bh = blockIdx.x / nsplit, b = bh / a.nheads, h = bh % a.nheads, P = a.headdim;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, myrow = lane / G;
    const int p0 = (sp * 8 + warp) * NR, di = a.nheads * P, V = di + 2 * a.ngroups * R;
    const bool mine = p0 + myrow < P;
    float* st = a.state + ((int64_t)bh * P + p0) * R + lane * 4;
    float4 hv[NR];
#pragma unroll
    for (int j = 0; j < NR; ++j)
        if (p0 + j < P) hv[j] = step2_ld4(st + j * R);
    const int ch = h * P + (mine ? p0 + myrow : 0);                                                  // the lane's x channel
    const int cb = di + ((tid >> 7) * a.ngroups + h / (a.nheads / a.ngroups)) * R + (tid & 127);     // the thread's B or C channel
    float* xwin = a.window + ((int64_t)b * V + ch) * 4;
    const float4 xw = step2_ld4(xwin), bw = step2_ld4(a.window + ((int64_t)b * V + cb) * 4);
    const float4 xt = step2_ld4(a.conv_w + (int64_t)ch * 4), bt = step2_ld4(a.conv_w + (int64_t)cb * 4);
    const float xb = a.conv_b[ch], bb = a.conv_b[cb], ah = a.a[h], dskip = a.d[h], dtb = a.dt_bias[h];
    const float gamma = __bfloat162float(static_cast<const __nv_bfloat16*>(a.gamma)[ch]);
    pdl_wait();
    const float bn = rows_value(a.proj, b, di + cb), xn = rows_value(a.proj, b, di + ch), z = rows_value(a.proj, b, ch);
    float dt = rows_value(a.proj, b, di + V + h);
    auto conv = [](const float4& w, float nw, const float4& t, float bias) {
        return silu_f32(bias + (w.y * t.x + w.z * t.y + w.w * t.z + nw * t.w));
    };
    bc[tid] = conv(bw, bn, bt, bb);
    const float xl = mine ? conv(xw, xn, xt, xb) : 0.f;
    if (mine && lane % G == 0) *reinterpret_cast<float4*>(xwin) = make_float4(xw.y, xw.z, xw.w, xn);
    dt = fminf(fmaxf(softplus_f32(dt + dtb), a.dt_min), a.dt_max);
    const float da = expf(dt * ah), dtx = dt * xl;
    __syncthreads();
    const float4 bq = step2_ld4(bc + lane * 4), cq = step2_ld4(bc + R + lane * 4);
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
    float ss = 0.f;
    if (mine && lane % G == 0) {
        const float y = fmaf(dskip, xl, v[0]), gate = silu_fast(z);
        const float u = a.norm_before_gate ? y : y * gate;
        ss = u * u;
        const float g = u * gamma * (a.norm_before_gate ? gate : 1.f);
        const __nv_bfloat16 hi = __float2bfloat16_rn(g);
        __nv_bfloat16* o = static_cast<__nv_bfloat16*>(a.out) + (int64_t)b * di + ch;
        o[0] = hi;
        if (a.planes == 2) o[(int64_t)a.batch * di] = __float2bfloat16_rn(g - __bfloat162float(hi));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    if (tid == 0) {
        float t = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) t += red[i];
        a.ss[(int64_t)b * a.nss + h * nsplit + sp] = t;
    }
}

// RmsNormGated (src/modules/norm/rms_norm_gated.rs:70-135), the gate read from the projection's partial sums.
__global__ void __launch_bounds__(1024) decode_gated_norm_kernel(bm_rmsnorm_gated_args a, bmx_rows z, int64_t out_lo) {
    pdl_launch_dependents();
    const int64_t row = blockIdx.x;
    const int c = threadIdx.x * 8;
    const bool live = c < a.width;
    uint4 graw = make_uint4(0, 0, 0, 0);
    if (live) graw = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(a.gamma) + c);
    pdl_wait();
    float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, gate[8];
    if (live) {
        unpack8(*reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(a.x) + row * a.x_stride + c), x);
        rows_load8(z, row, c, gate);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            gate[j] = silu_fast(gate[j]);
            if (!a.norm_before_gate) x[j] *= gate[j];
        }
    }
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) ss = fmaf(x[j], x[j], ss);
    const float inv = rsqrtf(block_sum(ss) / (float)a.width + a.eps);
    if (live) {
        float g[8];
        unpack8(graw, g);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            x[j] = x[j] * inv * g[j];
            if (a.norm_before_gate) x[j] *= gate[j];
        }
        store_planes(static_cast<__nv_bfloat16*>(a.out) + row * a.width + c, out_lo, x);
    }
}

// bm_conv_step for 4 taps with the new column read from `in` (src/mamba2/mamba2.rs:865-902).  A thread keeps two batch
// rows of one channel, so that two windows are in flight and the taps are fetched once.
__global__ void __launch_bounds__(128) decode_conv_kernel(bm_conv_step_args a, bmx_rows in, int col) {
    pdl_launch_dependents();
    const int v = blockIdx.x * 128 + threadIdx.x, b0 = blockIdx.y * 2;
    const bool live = v < a.channels;
    float4 w = make_float4(0.f, 0.f, 0.f, 0.f), win[2];
    float bias = 0.f;
    if (live) {
        w = *reinterpret_cast<const float4*>(a.weight + (int64_t)v * 4);
        bias = a.bias ? a.bias[v] : 0.f;
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if (b0 + i < a.batch) win[i] = *reinterpret_cast<const float4*>(a.window + ((int64_t)(b0 + i) * a.channels + v) * 4);
    }
    pdl_wait();
    if (!live) return;
    __nv_bfloat16 *dst, *ox = static_cast<__nv_bfloat16*>(a.out);
    int64_t ds;
    if (v < a.split_x) dst = ox + v, ds = a.split_x;
    else if (v < a.split_x + a.split_bc) dst = static_cast<__nv_bfloat16*>(a.out_b) + (v - a.split_x), ds = a.split_bc;
    else dst = static_cast<__nv_bfloat16*>(a.out_c) + (v - a.split_x - a.split_bc), ds = a.split_bc;
    float xn[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) xn[i] = b0 + i < a.batch ? rows_value(in, b0 + i, col + v) : 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int b = b0 + i;
        if (b >= a.batch) break;
        const float4 nw = make_float4(win[i].y, win[i].z, win[i].w, xn[i]);
        *reinterpret_cast<float4*>(a.window + ((int64_t)b * a.channels + v) * 4) = nw;
        dst[b * ds] = __float2bfloat16_rn(silu_f32(bias + (nw.x * w.x + nw.y * w.y + nw.z * w.z + nw.w * w.w)));
    }
}

template <bool DEEP, int PLANES>
int32_t launch_linear(const CUtensorMap& mw, const CUtensorMap& mx, float* part, int batch, int k, int n, int nslice, int32_t* status, bool first,
                      int stall, cudaStream_t st) {
    constexpr size_t smem = (size_t)lin_stages(DEEP) * kLinStageBytes + 1024;
    static uint64_t allowed = 0;   // devices whose shared-memory limit for this kernel is raised
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev > 63 || !(__atomic_load_n(&allowed, __ATOMIC_RELAXED) >> dev & 1)) {
        if (int32_t e = check_cuda(cudaFuncSetAttribute(decode_linear_kernel<DEEP, PLANES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                                   "cudaFuncSetAttribute(decode_linear)"))
            return e;
        if (dev <= 63) __atomic_fetch_or(&allowed, (uint64_t)1 << dev, __ATOMIC_RELAXED);
    }
    return launch_chained("decode_linear", !first, dim3((unsigned)cdiv(n, kLinCols), nslice), kLinThreads, smem, st, decode_linear_kernel<DEEP, PLANES>, mw, mx,
                          part, batch, n, (int)cdiv(k, kLinK), nslice, status, stall);
}

}  // namespace

// One word per device, in pinned host memory that lives as long as the process: a graph may replay a step at any time, and
// the host looks at the word without a copy or a synchronisation.
constexpr int kStatusDevices = 64;
extern "C" int32_t* bmx_chain_status(int32_t device) {
    static std::mutex mu;
    static int32_t* words = nullptr;
    if (device < 0 || device >= kStatusDevices) {
        fail(BM_ERR_UNSUPPORTED, "device ordinal %d out of range", device);
        return nullptr;
    }
    std::lock_guard<std::mutex> lock(mu);
    if (words == nullptr) {
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;   // the first step of a process may be one that is captured
        cudaThreadExchangeStreamCaptureMode(&mode);
        void* p = nullptr;
        const int32_t e = check_cuda(cudaHostAlloc(&p, kStatusDevices * sizeof(int32_t), cudaHostAllocPortable | cudaHostAllocMapped), "cudaHostAlloc(status)");
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (e) return nullptr;
        std::fill_n(static_cast<int32_t*>(p), kStatusDevices, 0);
        words = static_cast<int32_t*>(p);
    }
    return words + device;
}
extern "C" int32_t bmx_chain_take_status(int32_t* word) {
    if (__atomic_exchange_n(word, 0, __ATOMIC_RELAXED) == 0) return BM_OK;
    return fail(BM_ERR_TIMEOUT, "a bounded wait of a decode step on this device ran out: that step's output and the caches it updated are not valid");
}

// A CTA takes 128 columns x one slice of K, at least two 64-wide k blocks.  Few column tiles: one CTA per SM with twice the
// stages, so that the reader sums half the slices with the same bytes in flight.  More than a third of the SMs: that would be
// two slices or one, which leave SMs without a CTA, so two CTAs share an SM and the slices fill those slots.  Per layer at
// batch 1, one CTA / two CTAs per SM (in-projection's tiles): 27 tiles 18.4 / 19.2 us, 35 18.6 / 20.0, 43 20.0 / 20.7;
// 51 22.1 / 22.1, 59 24.1 / 23.7, 67 26.1 / 24.8 (batch 8: 24.5 / 24.9, 27.7 / 30.6, 25.8 / 27.2; 28.8 / 28.5, 31.6 / 31.5,
// 33.8 / 32.0).  For an out-projection's 6 to 20 tiles the two differ by 3 % or less.
// Batches above 8 are left to the library product: 8 rows in two planes are what the 16-row operand holds.  Up to there the
// library takes, library / streaming per layer: d_model 768 27.4 / 18.8 us at batch 1, 26.4 / 24.7 at 8; 1536 24.9 / 21.6, 28.7 /
// 28.1; 2560 35.3 / 29.2, 43.5 / 39.7.
constexpr int kLinBatch = kLinRows / 2;
static bool linear_deep(int tiles) { return tiles <= sm_count() / 3; }
extern "C" int32_t bmx_decode_slices(int32_t batch, int32_t k, int32_t n) {
    if (batch < 1 || batch > kLinBatch || k % 8 || n % 8 || k < kLinK || n < kLinCols) return 0;
    const int tiles = (int)cdiv(n, kLinCols), kb = (int)cdiv(k, kLinK);
    return std::max(1, std::min({(linear_deep(tiles) ? 1 : 2) * sm_count() / tiles, kb / 2, 16}));
}

extern "C" int32_t bmx_decode_linear(const void* x, int32_t planes, const void* w, float* part, int32_t batch, int32_t k, int32_t n, int32_t nslice,
                                     int32_t* status, int32_t first, int32_t stall, void* stream) {
    CUtensorMap mw, mx;
    const char* err = nullptr;
    BM_REQUIRE_PTR(x);
    BM_REQUIRE_PTR(w);
    BM_REQUIRE_PTR(part);
    BM_REQUIRE_PTR(status);
    const uint64_t dw[2] = {(uint64_t)n, (uint64_t)k}, sw[1] = {(uint64_t)n * 2};
    const uint64_t dx[3] = {(uint64_t)k, (uint64_t)batch, (uint64_t)planes}, sx[2] = {(uint64_t)k * 2, (uint64_t)batch * k * 2};
    const uint32_t bw[2] = {64, kLinK}, bx[3] = {kLinK, (uint32_t)(kLinRows / planes), (uint32_t)planes};
    if (!tc::make_tensor_map_bf16(&mw, w, 2, dw, sw, bw, 128, &err) || !tc::make_tensor_map_bf16(&mx, x, 3, dx, sx, bx, 128, &err))
        return fail(BM_ERR_CUDA, "%s", err);
    auto go = [&](auto f) { return f(mw, mx, part, batch, k, n, nslice, status, first != 0, stall, static_cast<cudaStream_t>(stream)); };
    if (linear_deep((int)cdiv(n, kLinCols))) return planes == 2 ? go(launch_linear<true, 2>) : go(launch_linear<true, 1>);
    return planes == 2 ? go(launch_linear<false, 2>) : go(launch_linear<false, 1>);
}

static int32_t check_rows(const bmx_rows* r) {
    BM_REQUIRE(r != nullptr, BM_ERR_NULL_POINTER, "rows are NULL");
    if (r->part) BM_REQUIRE_PTR(r->part);
    else BM_REQUIRE_PTR(r->dense);
    return BM_OK;
}
static int32_t check_mixer(const bmx_mixer* a) {
    if (int32_t e = check_rows(&a->proj)) return e;
    BM_REQUIRE_PTR(a->state);
    BM_REQUIRE_PTR(a->window);
    BM_REQUIRE_PTR(a->conv_w);
    BM_REQUIRE_PTR(a->conv_b);
    BM_REQUIRE_PTR(a->a);
    BM_REQUIRE_PTR(a->d);
    BM_REQUIRE_PTR(a->dt_bias);
    BM_REQUIRE_PTR(a->gamma);
    BM_REQUIRE_PTR(a->out);
    BM_REQUIRE_PTR(a->ss);
    return BM_OK;
}
static unsigned row_threads(int width) { return (unsigned)(cdiv(width, 8 * 32) * 32); }

extern "C" int32_t bmx_decode_norm(const void* residual, const float* residual32, const bmx_rows* add, const bmx_mixer* prev, const void* gamma, float eps,
                                   float* x32, void* x_out, void* out, int32_t planes, int32_t batch, int32_t width, int32_t first, void* stream) {
    using T = __nv_bfloat16;
    if (add)
        if (int32_t e = check_rows(add)) return e;
    if (prev)
        if (int32_t e = check_mixer(prev)) return e;
    BM_OPTIONAL_PTR(residual);
    BM_OPTIONAL_PTR(residual32);
    BM_OPTIONAL_PTR(x32);
    BM_OPTIONAL_PTR(x_out);
    BM_OPTIONAL_PTR(out);
    if (out) BM_REQUIRE_PTR(gamma);
    const bmx_rows none{};
    const bmx_mixer nomix{};
    return launch_chained("decode_norm", !first, batch, row_threads(width), 0, static_cast<cudaStream_t>(stream), decode_norm_kernel,
                          static_cast<const T*>(residual), residual32, add ? *add : none, add != nullptr, prev ? *prev : nomix, prev != nullptr,
                          static_cast<const T*>(gamma), eps, x32, static_cast<T*>(x_out), static_cast<T*>(out),
                          planes == 2 ? (int64_t)batch * width : 0, width);
}

extern "C" int32_t bmx_decode_mixer_sums(int32_t batch, int32_t nheads, int32_t headdim) {
    return (int64_t)batch * nheads < 2 * sm_count() ? nheads * (int32_t)cdiv(headdim, kMixRows) : 0;
}
extern "C" int32_t bmx_decode_mixer(const bmx_mixer* a, void* stream) {
    if (int32_t e = check_mixer(a)) return e;
    const int nsplit = (int)cdiv(a->headdim, kMixRows);
    return launch_chained("decode_mixer", true, a->batch * a->nheads * nsplit, 256, 0, static_cast<cudaStream_t>(stream), decode_mixer_kernel, *a, nsplit);
}

extern "C" int32_t bmx_decode_conv(const bm_conv_step_args* a, const bmx_rows* in, int32_t col, void* stream) {
    if (int32_t e = check_rows(in)) return e;
    BM_REQUIRE_PTR(a->window);
    BM_REQUIRE_PTR(a->weight);
    BM_OPTIONAL_PTR(a->bias);
    BM_REQUIRE_PTR(a->out);
    BM_REQUIRE_PTR(a->out_b);
    BM_REQUIRE_PTR(a->out_c);
    return launch_chained("decode_conv", true, dim3((unsigned)cdiv(a->channels, 128), (unsigned)cdiv(a->batch, 2)), 128, 0,
                          static_cast<cudaStream_t>(stream), decode_conv_kernel, *a, *in, col);
}

extern "C" int32_t bmx_decode_state(const bm_step2_args* a, const bmx_rows* in, int32_t col, void* stream) {
    if (int32_t e = check_rows(in)) return e;
    BM_REQUIRE_PTR(a->state);
    BM_REQUIRE_PTR(a->x);
    BM_REQUIRE_PTR(a->a);
    BM_REQUIRE_PTR(a->b);
    BM_REQUIRE_PTR(a->c);
    BM_OPTIONAL_PTR(a->d);
    BM_REQUIRE_PTR(a->dt_bias);
    BM_REQUIRE_PTR(a->y);
    return launch_step2_rows<__nv_bfloat16>(*a, DtRows{*in, col}, true, static_cast<cudaStream_t>(stream));
}

extern "C" int32_t bmx_decode_gated_norm(const bm_rmsnorm_gated_args* a, const bmx_rows* z, int32_t planes, void* stream) {
    if (int32_t e = check_rows(z)) return e;
    BM_REQUIRE_PTR(a->x);
    BM_REQUIRE_PTR(a->gamma);
    BM_REQUIRE_PTR(a->out);
    return launch_chained("decode_gated_norm", true, a->rows, row_threads(a->width), 0, static_cast<cudaStream_t>(stream), decode_gated_norm_kernel, *a, *z,
                          planes == 2 ? (int64_t)a->rows * a->width : 0);
}
