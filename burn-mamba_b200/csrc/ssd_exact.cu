// Exact chunked SSD forward: K1 + K3 chunk scan and chunk state, K4 state passing, K5 chunk output, in float32 on CUDA
// cores.  Serves float32 inputs (rel-L2 1e-4 parity), shapes the tensor-core path does not cover, and is the on-device
// cross-check for the tensor-core kernels.
//
// Reference decomposition: src/mamba2/ssd/serial.rs:138-506 (Mamba-2),
// src/mamba3/double_ssd/ssd/serial.rs:118-409 and src/mamba3/single_ssd/ssd/serial.rs:56-268 (Mamba-3).
//
// Split.  The result does not depend on the chunk length (only `chunk_states` does), so the kernels use chunks of 64
// fused rows whatever the caller's Q: the work of a row inside its chunk grows with the chunk, and a short sequence
// gives too few CTAs at Q = 256 (2 x 8 x 2 of them for b2 L500 H8).  A chunk is one tile: K3 is one 64-row outer product
// per (chunk, head), K5 one tile of C B^T, C h^T and W V, each operand staged in shared memory once and multiplied from
// registers (ssd_exact_tiles.cuh).
// Measured against chunks of the caller's length and 32 x 32 tiles read element by element from shared memory:
//   b2 L512 H8 P64 N64 (Q 256):             K1 + K3 72 -> 7 us, K4 9 -> 4, K5 44 -> 12
//   b2 L389 H32 P64 N128, MIMO rank 4:      K1 + K3 969 -> 61 us, K4 41 -> 20, K5 1239 -> 142 (5.7 GFLOP at 25 TFLOP/s)
#include "ssd_exact_tiles.cuh"

#include <mutex>

namespace bm {
namespace exact {

int inner_chunk(int Q, int M, bool want_states) {
    int q = TR / M > 1 ? TR / M : 1;
    if (q >= Q) return Q;
    if (want_states) {   // the caller's chunk boundaries have to be boundaries here
        while (Q % q) --q;
        // Chunks that leave more than half of their tile empty cost more than the caller's own, walked tile by tile with their
        // states in place: a prime Q would keep a state per token (b1 L4096 H8 P64 N128 at Q = 127: 1.1 GB for 9 MB of results).
        if (2 * q * M < TR) return Q;
    }
    return q;
}

int longer_chunk(int q, int Q, bool want_states) {
    q = q * 2 < Q ? q * 2 : Q;
    while (want_states && Q % q) ++q;
    return q;
}

namespace {

// K1 + K3: cum_l = inclusive cumsum of da over the chunk (positions past seqlen behave as dt = 0 padding,
// src/mamba2/mamba2.rs:703-722), cs_l = source-column scale, and
//   S_n[p, r] = sum_j v_j[p] B_j[r] cs_t(j) exp(Aend - cum_t(j))        (state: v, B)
//   G_n[p, r] = sum_i dy_i[p] C_i[r] exp(cum_t(i))                      (readout gradient, the second half of the grid)
// for one 64 x W block of one chunk.  Of issue slots 71 % are used, the shared-memory pipe stands at
// 59 % and the float32 pipe at 53 % (b8 L2048 H16 P64 N128): 64 W multiply-adds per row against 64 + W staged values.
template <typename T, bool VEC, int W>
__global__ void __launch_bounds__(kThreads, W == 128 ? 3 : 4)
chunk_state_kernel(Params p, const void* dy, float* dstates, float* zero_a, float* zero_b, int64_t zero_n, float* zero_h1, float* zero_h2) {
    extern __shared__ __align__(16) float smem[];
    float* vs = smem;            // [TR][TP]
    float* bs = smem + TR * TP;  // [TR][W]
    __shared__ TileRows tr;
    __shared__ float scum[TR], scs[TR], wgt[TR], s_aend;
    const int h = blockIdx.y, b = blockIdx.z, tid = threadIdx.x;
    const int nrb = (p.R + W - 1) / W, modes = dy ? 2 : 1;
    int x = blockIdx.x;
    const int n = x % p.NC; x /= p.NC;
    const int mode = x % modes; x /= modes;
    const int rb = x % nrb, pb = x / nrb;
    const int g = h / (p.H / p.G), QM = p.Q * p.M;
    if (zero_n > 0) {   // this CTA's share of the accumulators that a later kernel adds into
        const int64_t nblk = (int64_t)gridDim.x * gridDim.y * gridDim.z, me = ((int64_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
        for (int64_t i = me * kThreads + tid; i < zero_n; i += nblk * kThreads) zero_a[i] = 0.f, zero_b[i] = 0.f;
    }
    if (blockIdx.x == 0 && b == 0 && tid == 0) {
        if (zero_h1) zero_h1[h] = 0.f;
        if (zero_h2) zero_h2[h] = 0.f;
    }
    const void* src_v = mode ? dy : p.v;
    const void* src_b = mode ? p.cmat : p.bmat;
    auto stage_tile = [&](int i0) {
        fill_rows(tr, p, b, n, i0, tid);
        __syncthreads();
        stage<T, VEC, TP>(vs, TP, static_cast<const T*>(src_v), tr, p.H, h, p.P, pb * TP, tid);
        stage_bc<T, VEC, W>(bs, W, src_b, tr, p, g, h, rb * W, tid);
        cp_async_commit();
    };
    stage_tile(0);
    const bool small = p.Q <= TR;
    const int64_t cbase = (((int64_t)b * p.H + h) * p.NC + n) * p.Q;
    if (tid < 32) {
        const float ah = p.a ? p.a[h] : 1.f, bias = p.dt_bias ? p.dt_bias[h] : 0.f;
        const bool publish = !small || (mode == 0 && rb == 0 && pb == 0);
        float run = 0.f;
        for (int l0 = 0; l0 < p.Q; l0 += 32) {
            const int l = l0 + tid, s = n * p.Q + l;
            float da = 0.f, c = 0.f;
            if (l < p.Q && s < p.S) {
                const int64_t gi = ((int64_t)b * p.S + s) * p.H + h;
                float raw = p.dsrc[gi];
                if (p.dt_bias) raw = fminf(fmaxf(softplus_f32(raw + bias), p.dt_min), p.dt_max);
                da = raw * ah;
                c = p.cs_mode == 1 ? raw : (p.cs_mode == 2 ? p.colscale[gi] : 1.f);
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float up = __shfl_up_sync(0xffffffffu, da, o);
                if (tid >= o) da += up;
            }
            da += run;
            run = __shfl_sync(0xffffffffu, da, 31);
            if (l < p.Q) {
                if (small) scum[l] = da, scs[l] = c;
                if (publish) {
                    p.cum[cbase + l] = da, p.cs[cbase + l] = c;
                    // same-time weight: column scale (non-strict cores) or gamma (strict core)
                    if (p.gs) p.gs[cbase + l] = !p.strict ? c : (p.gamma && s < p.S) ? p.gamma[((int64_t)b * p.S + s) * p.H + h] : 0.f;
                }
            }
        }
        if (tid == 0) s_aend = run;
    }
    constexpr int NP = W == 128 ? 8 : 4;   // rows p of the thread: 8 x 4 outputs at W = 128, 4 x 4 at 64
    const int tx = W == 128 ? tid & 31 : tid & 15, ty = W == 128 ? tid >> 5 : tid >> 4;
    float acc[NP][4];
#pragma unroll
    for (int i = 0; i < NP; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    for (int i0 = 0; i0 < QM; i0 += TR) {
        if (i0 > 0) {
            __syncthreads();
            stage_tile(i0);
        }
        cp_async_wait<0>();
        __syncthreads();
        if (tid < TR) {
            const int t = tr.t[tid];
            const float c = small ? scum[t] : p.cum[cbase + t], k = small ? scs[t] : p.cs[cbase + t];
            wgt[tid] = tr.idx[tid] < 0 ? 0.f : mode ? expf(c) : k * expf(s_aend - c);
        }
        __syncthreads();
        for (int e = tid; e < TR * TP / 4; e += kThreads) {
            float4* q = reinterpret_cast<float4*>(vs) + e;
            const float w = wgt[e / (TP / 4)];
            const float4 v = *q;
            *q = make_float4(v.x * w, v.y * w, v.z * w, v.w * w);
        }
        __syncthreads();
        const int rows = min(TR, QM - i0);
#pragma unroll 4
        for (int k = 0; k < rows; ++k) {
            const float4 bq = load4(bs + k * W + tx * 4);
#pragma unroll
            for (int i = 0; i < NP; i += 4) {
                const float4 vq = load4(vs + k * TP + ty * NP + i);
#pragma unroll
                for (int ii = 0; ii < 4; ++ii) {
                    const float v = f4(vq, ii);
                    acc[i + ii][0] = fmaf(v, bq.x, acc[i + ii][0]);
                    acc[i + ii][1] = fmaf(v, bq.y, acc[i + ii][1]);
                    acc[i + ii][2] = fmaf(v, bq.z, acc[i + ii][2]);
                    acc[i + ii][3] = fmaf(v, bq.w, acc[i + ii][3]);
                }
            }
        }
    }
    float* out = (mode ? dstates : p.states) + (((int64_t)b * p.NC + n) * p.H + h) * (int64_t)p.P * p.R;
    const int r = rb * W + tx * 4;
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        const int pp = pb * TP + ty * NP + i;
        if (pp >= p.P || r >= p.R) continue;
        float* o = out + (int64_t)pp * p.R + r;
        if (VEC) {
            *reinterpret_cast<float4*>(o) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (r + j < p.R) o[j] = acc[i][j];
        }
    }
}

// K4: h_{n+1} = exp(Aend_n) h_n + S_n; the buffer of S_n is overwritten with the state entering chunk n
// (src/mamba2/ssd/serial.rs:275-343), copied to `states_out` where n is a boundary of the caller's chunks.  With
// `dstates` a second half of the grid runs the reverse recurrence dS_n = dh_{n+1}, dh_n = exp(Aend_n) dh_{n+1} + G_n.
// A stream over the chunk states: the maps do not depend on the state, so eight chunks are fetched ahead.
constexpr int kAhead = 8;
template <int V>   // values per thread
__global__ void __launch_bounds__(128) state_passing_kernel(Params p, float* dstates, const float* dh_final, float* dh0) {
    const int PR = p.P * p.R;
    const int o = ((blockIdx.x >> (dstates ? 1 : 0)) * blockDim.x + threadIdx.x) * V;
    const int h = blockIdx.y, b = blockIdx.z;
    const bool reverse = dstates && (blockIdx.x & 1);
    if (o >= PR) return;
    const int64_t bh = (int64_t)b * p.H + h;
    auto ld = [](const float* q, float (&v)[V]) {
        if constexpr (V == 4) {
            const float4 t = load4(q);
            v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
        } else {
            v[0] = *q;
        }
    };
    auto st = [](float* q, const float (&v)[V]) {
        if constexpr (V == 4) *reinterpret_cast<float4*>(q) = make_float4(v[0], v[1], v[2], v[3]);
        else *q = v[0];
    };
    const float* seed = reverse ? dh_final : p.h0;
    float run[V];
#pragma unroll
    for (int k = 0; k < V; ++k) run[k] = 0.f;
    if (seed) ld(seed + bh * PR + o, run);
    float* buf = (reverse ? dstates : p.states) + ((int64_t)b * p.NC * p.H + h) * PR + o;
    const int64_t step = (int64_t)p.H * PR;
    const float* aend = p.cum + bh * p.NC * p.Q + p.Q - 1;
    for (int n0 = 0; n0 < p.NC; n0 += kAhead) {
        float s[kAhead][V], e[kAhead];
        const int m = min(kAhead, p.NC - n0);
#pragma unroll
        for (int k = 0; k < kAhead; ++k)
            if (k < m) {
                const int n = reverse ? p.NC - 1 - (n0 + k) : n0 + k;
                ld(buf + n * step, s[k]);
                e[k] = expf(aend[(int64_t)n * p.Q]);
            }
#pragma unroll
        for (int k = 0; k < kAhead; ++k)
            if (k < m) {
                const int n = reverse ? p.NC - 1 - (n0 + k) : n0 + k;
                st(buf + n * step, run);
                if (!reverse && p.states_out && (int64_t)n * p.Q % p.Qout == 0)
                    st(p.states_out + (((int64_t)b * ((p.S + p.Qout - 1) / p.Qout) + (int64_t)n * p.Q / p.Qout) * p.H + h) * PR + o, run);
#pragma unroll
                for (int v = 0; v < V; ++v) run[v] = fmaf(e[k], run[v], s[k][v]);
            }
    }
    float* last = reverse ? dh0 : p.h_final;
    if (last) st(last + bh * PR + o, run);
}

}  // namespace

namespace {

// K5: y_i = exp(cum_t(i)) C_i . h_n + sum_j (C_i . B_j) kern(i, j) v_j (+ D v_i) (* silu(z_i)), with
//   kern(i, j) = exp(cum_t(i) - cum_t(j)) cs_t(j)   for t(j) <  t(i)
//              = cs_t (non-strict) | gamma_t (strict) for t(j) == t(i)
//              = 0                                     for t(j) >  t(i)
// (src/mamba2/ssd/serial.rs:349-506; src/mamba3/single_ssd/ssd/serial.rs:156-268 with the same-step
// term of src/mamba3/single_ssd/ssd/diag.rs:50-100 folded into the same-time block).
// One CTA per (64-row tile, head, 64-wide block of P).  Column groups above the diagonal are skipped in both products.
// Shared memory at W = 128: C 33 KB, B (its space then holds the 64 x 64 weights and V) 33 KB, h 33 KB: two CTAs per SM.
template <typename T, bool VEC, int W>
__global__ void __launch_bounds__(kThreads, 2) chunk_scan_kernel(Params p) {
    constexpr int LD = W + 4;
    extern __shared__ __align__(16) float smem[];
    float* Cs = smem;
    float* Hs = Cs + TR * LD;
    float* Bs = Hs + TP * LD;      // union: Bs | Ws, Vs
    float* Ws = Bs;                // [TR][LDX]
    float* Vs = Bs + TR * LDX;     // [TR][TP]
    __shared__ TileRows ti, tj;
    __shared__ float ci[TR], gi[TR], cj[TR], kj[TR];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int QM = p.Q * p.M, ntile = (QM + TR - 1) / TR;
    const int npb = (p.P + TP - 1) / TP, nrb = (p.R + W - 1) / W;
    int64_t bx = blockIdx.x;
    const int pb = bx % npb; bx /= npb;
    const int it = bx % ntile; bx /= ntile;
    const int h = bx % p.H, n = bx / p.H, b = blockIdx.y;
    const int g = h / (p.H / p.G), i0 = it * TR;
    if ((int64_t)n * p.Q + i0 / p.M >= p.S) return;   // a tile past the end of the sequence
    const int64_t cbase = (((int64_t)b * p.H + h) * p.NC + n) * p.Q;
    const float* hin = p.states + (((int64_t)b * p.NC + n) * p.H + h) * (int64_t)p.P * p.R;
    const int i_last = min(i0 + TR, QM) - 1;
    const int j_end = min(QM, (i_last / p.M + 1) * p.M);   // columns with t(j) <= t(i_last)
    const int njt = (j_end + TR - 1) / TR;
    fill_rows(ti, p, b, n, i0, tid);
    __syncthreads();
    float acc[4][4];   // rows 4 ty + i, columns 4 tx + j of the P block
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    for (int jt = 0; jt < njt; ++jt) {
        const int j0 = jt * TR;
        float w[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) w[i][j] = 0.f;
        if (jt > 0) __syncthreads();   // the last round's weights and V are read
        fill_rows(tj, p, b, n, j0, tid);
        if (tid < TR) {
            const int t = min((j0 + tid) / p.M, p.Q - 1);
            cj[tid] = p.cum[cbase + t], kj[tid] = p.cs[cbase + t];
            const int u = min((i0 + tid) / p.M, p.Q - 1), s = n * p.Q + u;
            ci[tid] = p.cum[cbase + u];
            gi[tid] = !p.strict ? p.cs[cbase + u] : (p.gamma && s < p.S) ? p.gamma[((int64_t)b * p.S + s) * p.H + h] : 0.f;
        }
        __syncthreads();
        // column groups (16 wide) this warp's rows reach
        const int wrow_last = min(i0 + (tid >> 5) * 8 + 7, QM - 1);
        const int jmax = min(TR, (wrow_last / p.M + 1) * p.M - j0);
        const int nj = max(1, min(4, (jmax + 15) >> 4));
        for (int rb = 0; rb < nrb; ++rb) {
            if (rb > 0) __syncthreads();
            stage_bc<T, VEC, W>(Cs, LD, p.cmat, ti, p, g, h, rb * W, tid);
            stage_bc<T, VEC, W>(Bs, LD, p.bmat, tj, p, g, h, rb * W, tid);
            cp_async_commit();
            if (jt == 0) stage_state<VEC, W>(Hs, LD, hin, p.P, p.R, pb * TP, rb * W, tid);
            cp_async_commit();
            cp_async_wait<1>();
            __syncthreads();
            mul_kk_upto(nj, Cs + ty * 4 * LD, LD, Bs + tx * LD, LD, W, w);
            if (rb == nrb - 1) {
                __syncthreads();   // B is read: its space takes V and the weights
                stage<T, VEC, TP>(Vs, TP, static_cast<const T*>(p.v), tj, p.H, h, p.P, pb * TP, tid);
                cp_async_commit();
            }
            if (jt == 0) {
                if (rb == nrb - 1) cp_async_wait<1>(); else cp_async_wait<0>();
                __syncthreads();
                mul_kk<4>(Cs + ty * 4 * LD, LD, Hs + tx * LD, LD, W, acc);
            }
        }
        if (jt == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float e = expf(ci[ty * 4 + i]);
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] *= e;
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int ii = ty * 4 + i, jj = tx + 16 * j;
                float kern = 0.f;
                if (i0 + ii < QM && j0 + jj < QM) {
                    const int a = ti.t[ii], c = tj.t[jj];
                    if (c < a) kern = expf(ci[ii] - cj[jj]) * kj[jj];
                    else if (c == a) kern = gi[ii];
                }
                Ws[ii * LDX + jj] = w[i][j] * kern;
            }
        cp_async_wait<0>();
        __syncthreads();
        mul_km<1, false>(Ws + ty * 4 * LDX, LDX, Vs + tx * 4, TP, max(4, min(TR, (jmax + 3) & ~3)), acc);
    }
    // ---- epilogue: D skip, optional gate, store ----
    const int p0 = pb * TP + tx * 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int64_t ri = ti.idx[ty * 4 + i];
        if (ri < 0 || p0 >= p.P) continue;
        const int64_t gidx = (ri * p.H + h) * p.P + p0;
        const float dskip = p.d ? p.d[h] : 0.f;
        const T* v = static_cast<const T*>(p.v) + gidx;
        const T* z = p.z ? static_cast<const T*>(p.z) + gidx : nullptr;
        T* y = static_cast<T*>(p.y) + gidx;
        if (VEC) {
            const float4 vq = load4(v), zq = z ? load4(z) : make_float4(0.f, 0.f, 0.f, 0.f);
            float o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                o[j] = p.d ? fmaf(dskip, f4(vq, j), acc[i][j]) : acc[i][j];
                if (z) o[j] *= silu_f32(f4(zq, j));
            }
            if constexpr (sizeof(T) == 4) {
                *reinterpret_cast<float4*>(y) = make_float4(o[0], o[1], o[2], o[3]);
            } else {
                __nv_bfloat162 lo = __floats2bfloat162_rn(o[0], o[1]), hi = __floats2bfloat162_rn(o[2], o[3]);
                *reinterpret_cast<uint2*>(y) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
            }
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (p0 + j < p.P) {
                    float o = p.d ? fmaf(dskip, to_f32(v[j]), acc[i][j]) : acc[i][j];
                    if (z) o *= silu_f32(to_f32(z[j]));
                    y[j] = from_f32<T>(o);
                }
        }
    }
}

// Vector loads need rows that are multiples of four entries (and no rotation while loading B / C).
bool vec_ok(const Params& p) { return p.P % 4 == 0 && p.R % 4 == 0 && p.angles == nullptr; }

// Calls f(T{}, bool constant, int constant) for the runtime dtype, vector flag and block width.
template <typename F>
int32_t dispatch(const Params& p, F f) {
    const bool vec = vec_ok(p), wide = p.R > 64;
    auto go = [&](auto t) {
        if (vec) return wide ? f(t, std::true_type{}, std::integral_constant<int, 128>{}) : f(t, std::true_type{}, std::integral_constant<int, 64>{});
        return wide ? f(t, std::false_type{}, std::integral_constant<int, 128>{}) : f(t, std::false_type{}, std::integral_constant<int, 64>{});
    };
    return p.dtype == BM_DTYPE_F32 ? go(float{}) : go(__nv_bfloat16{});
}

template <typename K>
int32_t allow_smem(K kernel, size_t bytes, const char* what) {
    if (bytes <= 32 * 1024) return BM_OK;   // the 48 KB default also holds the static arrays
    return check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes), what);
}

}  // namespace

int32_t launch_chunk_state(const Params& p, const void* dy, float* dstates, float* zero_a, float* zero_b, int64_t zero_n, float* zero_h1,
                           float* zero_h2, cudaStream_t stream) {
    return dispatch(p, [&](auto t, auto vec, auto w) -> int32_t {
        using T = decltype(t);
        constexpr int W = decltype(w)::value;
        auto kernel = chunk_state_kernel<T, decltype(vec)::value, W>;
        const size_t smem = (size_t)TR * (TP + W) * sizeof(float);
        if (int32_t e = allow_smem(kernel, smem, "cudaFuncSetAttribute(chunk_state)")) return e;
        const int64_t x = (int64_t)p.NC * cdiv(p.P, TP) * cdiv(p.R, W) * (dy ? 2 : 1);
        kernel<<<dim3((unsigned)x, p.H, p.B), kThreads, smem, stream>>>(p, dy, dstates, zero_a, zero_b, zero_n, zero_h1, zero_h2);
        return check_launch("chunk_state");
    });
}

int32_t launch_state_passing(const Params& p, float* dstates, const float* dh_final, float* dh0, cudaStream_t stream) {
    const int PR = p.P * p.R, v = PR % 4 == 0 ? 4 : 1;
    const dim3 grid((unsigned)cdiv(PR, 128 * v) * (dstates ? 2 : 1), p.H, p.B);
    if (v == 4) state_passing_kernel<4><<<grid, 128, 0, stream>>>(p, dstates, dh_final, dh0);
    else state_passing_kernel<1><<<grid, 128, 0, stream>>>(p, dstates, dh_final, dh0);
    return check_launch("state_passing");
}

static size_t scan_bytes(int B, int S, int H, int q) { return align_up((size_t)B * H * cdiv(S, q) * q * sizeof(float), 256); }
static size_t state_bytes(int B, int S, int H, int P, int R, int q) { return align_up((size_t)B * cdiv(S, q) * H * P * R * sizeof(float), 256); }

// Workspace at inner chunk length q: cum and column scale, and the chunk states unless they live in the caller's buffer.
static size_t need_bytes(const Params& p, int q) {
    const bool in_place = p.states_out != nullptr && q == p.Qout;
    return 2 * scan_bytes(p.B, p.S, p.H, q) + (in_place ? 0 : state_bytes(p.B, p.S, p.H, p.P, p.R, q));
}

static size_t bytes_at(int B, int S, int H, int P, int R, int Q, bool want_states, int q) {
    Params p{};
    p.B = B, p.S = S, p.H = H, p.P = P, p.R = R, p.Qout = Q;
    float dummy;
    p.states_out = want_states ? &dummy : nullptr;
    return need_bytes(p, q);
}
size_t workspace_bytes(int B, int S, int H, int P, int R, int M, int Q, bool want_states) {
    return bytes_at(B, S, H, P, R, Q, want_states, inner_chunk(Q, M, want_states));
}
size_t least_bytes(int B, int S, int H, int P, int R, int Q, bool want_states) { return bytes_at(B, S, H, P, R, Q, want_states, Q); }

// Shorter chunks are faster but keep more states: the chunk grows towards the caller's length until the scratch holds them.
static int fitting_chunk(const Params& p, size_t bytes) {
    const bool want_states = p.states_out != nullptr;
    int q = inner_chunk(p.Q, p.M, want_states);
    while (need_bytes(p, q) > bytes && q < p.Q) q = longer_chunk(q, p.Q, want_states);
    return q;
}

static int32_t run_at(Params p, int q, void* workspace, size_t ws_bytes, cudaStream_t stream) {
    const size_t need = need_bytes(p, q);
    if (workspace == nullptr || ws_bytes < need)
        return fail(BM_ERR_WORKSPACE_TOO_SMALL, "workspace of %zu bytes given, %zu needed", ws_bytes, need);
    if (!aligned16(workspace)) return fail(BM_ERR_BAD_ALIGNMENT, "workspace is not 16-byte aligned");
    if ((int64_t)p.P * p.R > 256 * 256 || p.P > 1024 || p.R > 1024)
        return fail(BM_ERR_UNSUPPORTED, "headdim %d x state_rank %d is beyond the exact path's tile limits", p.P, p.R);
    if (p.B > 65535 || p.H > 65535) return fail(BM_ERR_UNSUPPORTED, "batch / nheads above 65535");
    if ((size_t)16 * (p.P + p.R) * sizeof(float) > 48 * 1024)
        return fail(BM_ERR_UNSUPPORTED, "headdim + state_rank too large for the exact path");
    p.Q = q;
    p.NC = (int)cdiv(p.S, q);
    char* w = static_cast<char*>(workspace);
    const size_t scan = scan_bytes(p.B, p.S, p.H, q);
    p.cum = reinterpret_cast<float*>(w);
    p.cs = reinterpret_cast<float*>(w + scan);
    p.states = reinterpret_cast<float*>(w + 2 * scan);
    if (p.states_out && q == p.Qout) {   // the caller's buffer has exactly the states the kernels need
        p.states = p.states_out;
        p.states_out = nullptr;
    }
    if (int32_t e = launch_chunk_state(p, nullptr, nullptr, nullptr, nullptr, 0, nullptr, nullptr, stream)) return e;
    if (int32_t e = launch_state_passing(p, nullptr, nullptr, nullptr, stream)) return e;
    return dispatch(p, [&](auto t, auto vec, auto wc) -> int32_t {
        using T = decltype(t);
        constexpr int W = decltype(wc)::value, LD = W + 4;
        auto kernel = chunk_scan_kernel<T, decltype(vec)::value, W>;
        const int bv = TR * LD > TR * (LDX + TP) ? TR * LD : TR * (LDX + TP);
        const size_t smem = (size_t)(2 * TR * LD + bv) * sizeof(float);
        if (int32_t e = allow_smem(kernel, smem, "cudaFuncSetAttribute(chunk_scan)")) return e;
        const int64_t tiles = cdiv((int64_t)q * p.M, TR) * cdiv(p.P, TP) * p.H * p.NC;
        kernel<<<dim3((unsigned)tiles, p.B), kThreads, smem, stream>>>(p);
        return check_launch("chunk_scan");
    });
}

int32_t run(Params p, void* workspace, size_t ws_bytes, cudaStream_t stream) {
    p.Qout = p.Q;
    p.states_out = p.states;
    return run_at(p, fitting_chunk(p, ws_bytes), workspace, ws_bytes, stream);
}

}  // namespace exact
}  // namespace bm

// ---------------------------------------------------------------------------------------------
// Allocation-free variant of the exact Mamba-2 SSD forward.
//
// Some hosts of this library may never allocate device memory once they are running: a serving
// process whose memory budget is fixed and handed out at start-up, a plugin that is given raw tensor
// pointers by its framework but has no handle on that framework's allocator (so it cannot size and
// obtain the workspace bm_ssd2_fwd asks for), or code that runs where cudaMalloc would serialise
// the whole device.  For them the scratch of the exact path lives inside the library image: a
// file-scope device array that every GPU loading the library holds until the process exits.
// ---------------------------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_noalloc_scratch[BM_SSD2_NOALLOC_SCRATCH_BYTES];

namespace bm {
namespace exact {

// In host code `g_noalloc_scratch` is only a stand-in for the symbol; the address the kernels can
// use comes from cudaGetSymbolAddress, asked once per device with that device current.
static int32_t noalloc_scratch_ptr(void** out) {
    constexpr int kMaxDevices = 64;
    static void* ptrs[kMaxDevices] = {nullptr};
    static std::mutex mu;
    int dev = -1;
    if (int32_t e = check_cuda(cudaGetDevice(&dev), "cudaGetDevice")) return e;
    if (dev < 0 || dev >= kMaxDevices) return fail(BM_ERR_UNSUPPORTED, "device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> lock(mu);
    if (ptrs[dev] == nullptr) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return check_cuda(e, "cudaGetSymbolAddress(scratch)");
        if (p == nullptr) return fail(BM_ERR_CUDA, "cudaGetSymbolAddress returned a null address");
        ptrs[dev] = p;
    }
    *out = ptrs[dev];
    return BM_OK;
}

int32_t run_noalloc(Params p, cudaStream_t stream) {
    p.Qout = p.Q;
    p.states_out = p.states;
    const int q = fitting_chunk(p, (size_t)BM_SSD2_NOALLOC_SCRATCH_BYTES);
    const size_t need = need_bytes(p, q);
    if (need > (size_t)BM_SSD2_NOALLOC_SCRATCH_BYTES)
        return fail(BM_ERR_WORKSPACE_TOO_SMALL,
                    "this problem needs %zu bytes of scratch, the built-in scratch holds %zu: use bm_ssd2_fwd with a "
                    "caller-provided workspace",
                    need, (size_t)BM_SSD2_NOALLOC_SCRATCH_BYTES);
    void* scratch = nullptr;
    if (int32_t e = noalloc_scratch_ptr(&scratch)) return e;
    // Nothing in the scratch has to start at zero: K1 writes every cumsum / column-scale entry and K3
    // writes every chunk state before anything reads them, so the previous call's contents are dead.
    // The launches of a call go out together: two threads on one stream would otherwise use the array in turns.
    static std::mutex launches;
    std::lock_guard<std::mutex> lock(launches);
    return run_at(p, q, scratch, (size_t)BM_SSD2_NOALLOC_SCRATCH_BYTES, stream);
}

}  // namespace exact
}  // namespace bm
