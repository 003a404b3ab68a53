// Exact backward of the general chunked SSD (float32, CUDA cores).
//
// Follows the structure of the reference's recompute backward
// (src/mamba2/ssd/serial_recalculated/combined_backward.rs:126-590,
//  src/mamba3/single_ssd/ssd/serial_recalculated/combined_backward.rs:74-536): K1-K4 are recomputed
// from the saved inputs; the chunk-scan gradient splits into the state-readout term ("BLUE"), the
// intra-chunk term ("ORANGE" / lower + same-step), the state-passing recurrence run in reverse, and the
// chunk-state term; the cumulative-decay gradient is a suffix sum inside each chunk.
// With W = CB * kern, kern(i, j) = exp(cum_ti - cum_tj) cs_tj (t_j < t_i) | gs_t (t_j == t_i):
//   dW = dy v^T        dCB = dW * kern       dkern = dW * CB
//   dv_j = sum_i W_ij dy_i + w_j dS B_j (+ D dy_j)          w_j = cs_tj exp(Aend - cum_tj)
//   dB_j = sum_i dCB_ij C_i + w_j dS^T v_j
//   dC_i = sum_j dCB_ij B_j + e_i h_n^T dy_i                e_i = exp(cum_ti)
//   dh_n = exp(Aend_n) dh_{n+1} + sum_i e_i dy_i (x) C_i ,  dS_n = dh_{n+1}
//   dcum, dcs, dgs, dAend collect the scalar terms; d_da = suffix sum of dcum within the chunk.
#include "ssd_exact_tiles.cuh"

#include <algorithm>

namespace bm {
namespace exact {
namespace {

// Sum over the 16 threads of a row group (tx), result in all of them.
__device__ __forceinline__ float sum16(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float sum32(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One output row segment of 4 floats at column c of a row of `width`; added to memory when `add`.
template <bool VEC>
__device__ __forceinline__ void put4(float* row, int c, int width, float a, float b, float d, float e, bool add) {
    if (c >= width) return;
    if (VEC) {
        float4* q = reinterpret_cast<float4*>(row + c);
        if (add) atomicAdd(q, make_float4(a, b, d, e));
        else *q = make_float4(a, b, d, e);
    } else {
        const float v[4] = {a, b, d, e};
        for (int k = 0; k < 4; ++k)
            if (c + k < width) {
                if (add) atomicAdd(row + c + k, v[k]);
                else row[c + k] = v[k];
            }
    }
}

// The whole backward of one chunk that is one tile (Q M <= 64 rows, P <= 64, R <= W): the eight products of the header
// comment, each operand staged once, and the scalar gradients up to the finished suffix sum: 1.6 M multiply-adds per tile at
// P = R = 64, 2.7 M at R = 128, fed from shared memory (that pipe 56 % busy, the float32 pipe 38 %) by the eight warps of the
// one CTA that fits an SM (122 / 171 KB of shared memory).
// Measured at b2 L500 H8 P64 N64: 23 us, against 730 us for the column, row and finalise kernels below; the whole
// backward 1290 -> 45 us.
template <typename T, bool VEC, int W>
__global__ void __launch_bounds__(kThreads, 1) bwd_tile_kernel(BwdParams bp, const float* dstates) {
    constexpr int LD = W + 4, NQ = W / 64;
    const Params& p = bp.fwd;
    extern __shared__ __align__(16) float smem[];
    float* Cs = smem;
    float* Bs = Cs + TR * LD;
    float* Hs = Bs + TR * LD;      // dS_n, then h_n
    float* Ys = Hs + TP * LD;      // dy
    float* Xs = Ys + TR * LDX;     // v
    float* Ms = Xs + TR * LDX;     // CB * kern
    float* Ds = Ms + TR * LDX;     // dW * kern
    __shared__ TileRows tr;
    __shared__ float cum[TR], kol[TR], gam[TR], ew[TR], ww[TR];
    __shared__ float rowacc[TR], rowdc[TR], dws[TR], part[8][3][TR], dots[8], dds[8], dcum[TR], dcs[TR], dgs[TR];
    __shared__ float s_end[2];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, lane = tid & 31, warp = tid >> 5;
    const int h = blockIdx.x % p.H, n = blockIdx.x / p.H, b = blockIdx.y;
    const int hpg = p.H / p.G, g = h / hpg, QM = p.Q * p.M;
    const int64_t cbase = (((int64_t)b * p.H + h) * p.NC + n) * p.Q;
    const int64_t sbase = (((int64_t)b * p.NC + n) * p.H + h) * (int64_t)p.P * p.R;
    fill_rows(tr, p, b, n, 0, tid);
    __syncthreads();
    stage<T, VEC, W>(Cs, LD, static_cast<const T*>(p.cmat), tr, p.G, g, p.R, 0, tid);
    stage<T, VEC, W>(Bs, LD, static_cast<const T*>(p.bmat), tr, p.G, g, p.R, 0, tid);
    stage<T, VEC, TP>(Ys, LDX, static_cast<const T*>(bp.dy), tr, p.H, h, p.P, 0, tid);
    stage<T, VEC, TP>(Xs, LDX, static_cast<const T*>(p.v), tr, p.H, h, p.P, 0, tid);
    cp_async_commit();
    stage_state<VEC, W>(Hs, LD, dstates + sbase, p.P, p.R, 0, 0, tid);
    cp_async_commit();
    if (tid < TR) {
        const int t = tr.t[tid], s = n * p.Q + t;
        const float c = p.cum[cbase + t], k = p.cs[cbase + t], aend = p.cum[cbase + p.Q - 1];
        cum[tid] = c, kol[tid] = k;
        gam[tid] = !p.strict ? k : (p.gamma && s < p.S) ? p.gamma[((int64_t)b * p.S + s) * p.H + h] : 0.f;
        ew[tid] = expf(c), ww[tid] = tid < QM ? expf(aend - c) : 0.f;   // the column weight is kol * ww
        if (tid == 0) s_end[0] = expf(aend);
    }
    cp_async_wait<1>();
    __syncthreads();
    const int wrow = warp * 8, wlast = min(wrow + 7, QM - 1);
    const int jmax = min(TR, (wlast / p.M + 1) * p.M), nj = max(1, (jmax + 15) >> 4);   // columns the warp's rows reach
    const int k0 = min(wrow / p.M * p.M, TR);                                           // first row that reaches the warp's columns
    {
        float cb[4][4], dm[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) cb[i][j] = 0.f, dm[i][j] = 0.f;
        mul_kk_upto(nj, Cs + ty * 4 * LD, LD, Bs + tx * LD, LD, W, cb);
        mul_kk_upto(nj, Ys + ty * 4 * LDX, LDX, Xs + tx * LDX, LDX, TP, dm);
        float pc[4] = {0.f, 0.f, 0.f, 0.f}, pk[4] = {0.f, 0.f, 0.f, 0.f}, pg[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int ii = ty * 4 + i, ti = tr.t[ii];
            float row = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int jj = tx + 16 * j, tj = tr.t[jj];
                float kern = 0.f;
                if (ii < QM && jj < QM) {
                    const float dk = dm[i][j] * cb[i][j];
                    if (tj < ti) {
                        const float e = expf(cum[ii] - cum[jj]);
                        kern = e * kol[jj];
                        pc[j] = fmaf(dk, e, pc[j]);
                        pk[j] = fmaf(dk, kern, pk[j]);
                        row = fmaf(dk, kern, row);
                    } else if (tj == ti) {
                        kern = gam[ii];
                        pg[j] += dk;
                    }
                }
                Ms[ii * LDX + jj] = cb[i][j] * kern;
                Ds[ii * LDX + jj] = dm[i][j] * kern;
            }
            row = sum16(row);
            if (tx == 0) rowacc[ii] = row;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {   // the warp's two row groups, then the eight warps below
            pc[j] += __shfl_xor_sync(0xffffffffu, pc[j], 16);
            pk[j] += __shfl_xor_sync(0xffffffffu, pk[j], 16);
            pg[j] += __shfl_xor_sync(0xffffffffu, pg[j], 16);
            if (lane < 16) part[warp][0][tx + 16 * j] = pc[j], part[warp][1][tx + 16 * j] = pk[j], part[warp][2][tx + 16 * j] = pg[j];
        }
    }
    cp_async_wait<0>();
    __syncthreads();
    {   // dv
        float t1[4][4], dv[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) t1[i][j] = 0.f;
        mul_kk<4>(Bs + ty * 4 * LD, LD, Hs + tx * LD, LD, W, t1);
        const float dskip = p.d ? p.d[h] : 0.f;
        float ddp = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int ii = ty * 4 + i;
            const float4 x = load4(Xs + ii * LDX + tx * 4), y = load4(Ys + ii * LDX + tx * 4);
            const float w = kol[ii] * ww[ii];
            float dw = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                dw = fmaf(f4(x, j), t1[i][j], dw);   // dw_j = v_j^T dS B_j
                ddp = fmaf(f4(y, j), f4(x, j), ddp);
                dv[i][j] = fmaf(w, t1[i][j], dskip * f4(y, j));
            }
            dw = sum16(dw);
            if (tx == 0) dws[ii] = dw;
        }
        ddp = sum32(ddp);
        if (lane == 0) dds[warp] = ddp;
        mul_mm<1>(Ms + ty * 4, LDX, Ys + tx * 4, LDX, k0, TR, dv);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t ri = tr.idx[ty * 4 + i];
            if (ri >= 0) put4<VEC>(bp.dv + (ri * p.H + h) * p.P, tx * 4, p.P, dv[i][0], dv[i][1], dv[i][2], dv[i][3], false);
        }
    }
    {   // dB
        float acc[4][4 * NQ];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4 * NQ; ++j) acc[i][j] = 0.f;
        mul_km<NQ, true>(Xs + ty * 4 * LDX, LDX, Hs + tx * 4, LD, TP, acc);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float w = kol[ty * 4 + i] * ww[ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4 * NQ; ++j) acc[i][j] *= w;
        }
        mul_mm<NQ>(Ds + ty * 4, LDX, Cs + tx * 4, LD, k0, TR, acc);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t ri = tr.idx[ty * 4 + i];
            if (ri < 0) continue;
            float* row = bp.db + (ri * p.G + g) * p.R;
#pragma unroll
            for (int q = 0; q < NQ; ++q)
                put4<VEC>(row, q * 64 + tx * 4, p.R, acc[i][4 * q], acc[i][4 * q + 1], acc[i][4 * q + 2], acc[i][4 * q + 3], hpg > 1);
        }
    }
    __syncthreads();   // dS is read; its space takes h_n, entry by entry, with <dS, h> on the way
    {
        float dot = 0.f;
        const float* hin = p.states + sbase;
#pragma unroll 4
        for (int e = tid; e < TP * (W / 4); e += kThreads) {
            const int pp = e / (W / 4), c = (e % (W / 4)) * 4;
            if (pp >= p.P || c >= p.R) continue;   // zero in dS, stays zero
            float4* q = reinterpret_cast<float4*>(Hs + ((pp & 3) * 16 + (pp >> 2)) * LD + c);
            const float4 d = *q;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            const float* s = hin + (int64_t)pp * p.R + c;
            if (VEC) {
                v = load4(s);
            } else {
                v.x = s[0];
                if (c + 1 < p.R) v.y = s[1];
                if (c + 2 < p.R) v.z = s[2];
                if (c + 3 < p.R) v.w = s[3];
            }
            dot = fmaf(d.x, v.x, fmaf(d.y, v.y, fmaf(d.z, v.z, fmaf(d.w, v.w, dot))));
            *q = v;
        }
        dot = sum32(dot);
        if (lane == 0) dots[warp] = dot;
    }
    __syncthreads();
    {   // dC
        float acc[4][4 * NQ];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4 * NQ; ++j) acc[i][j] = 0.f;
        mul_km<NQ, true>(Ys + ty * 4 * LDX, LDX, Hs + tx * 4, LD, TP, acc);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int ii = ty * 4 + i;
            const float e = ew[ii];
            float row = 0.f;
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const float4 c = load4(Cs + ii * LD + q * 64 + tx * 4);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][4 * q + j] *= e;
                    row = fmaf(f4(c, j), acc[i][4 * q + j], row);
                }
            }
            row = sum16(row);
            if (tx == 0) rowdc[ii] = row;
        }
        mul_km<NQ, false>(Ds + ty * 4 * LDX, LDX, Bs + tx * 4, LD, min(TR, (jmax + 3) & ~3), acc);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t ri = tr.idx[ty * 4 + i];
            if (ri < 0) continue;
            float* row = bp.dc + (ri * p.G + g) * p.R;
#pragma unroll
            for (int q = 0; q < NQ; ++q)
                put4<VEC>(row, q * 64 + tx * 4, p.R, acc[i][4 * q], acc[i][4 * q + 1], acc[i][4 * q + 2], acc[i][4 * q + 3], hpg > 1);
        }
    }
    __syncthreads();
    // ---- scalars: per time step, then the suffix sum of dcum over the chunk (one warp, two steps per lane)
    if (tid < p.Q) {
        float u = 0.f, c = 0.f, gsum = 0.f;
        for (int m = 0; m < p.M; ++m) {
            const int i = tid * p.M + m;
            float a0 = 0.f, a1 = 0.f, a2 = 0.f;
#pragma unroll
            for (int w = 0; w < 8; ++w) a0 += part[w][0][i], a1 += part[w][1][i], a2 += part[w][2][i];
            u += rowacc[i] + rowdc[i] - (a1 + dws[i] * kol[i] * ww[i]);
            c += a0 + dws[i] * ww[i];
            gsum += a2;
        }
        dcum[tid] = u, dcs[tid] = c, dgs[tid] = gsum;
    } else if (tid < TR) {
        dcum[tid] = 0.f;
    }
    if (tid >= 64 && tid < 96) {   // dAend
        float a = 0.f;
        for (int i = tid - 64; i < QM; i += 32) a = fmaf(dws[i], kol[i] * ww[i], a);
        if (tid - 64 < 8) a = fmaf(s_end[0], dots[tid - 64], a);
        a = sum32(a);
        if (tid == 64) s_end[1] = a;
    }
    __syncthreads();
    if (warp == 0) {
        const float d0 = dcum[2 * lane], d1 = dcum[2 * lane + 1];
        float suf = d0 + d1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float up = __shfl_down_sync(0xffffffffu, suf, o);
            if (lane + o < 32) suf += up;
        }
        float later = __shfl_down_sync(0xffffffffu, suf, 1);
        if (lane == 31) later = 0.f;
        float run[2];
        run[1] = later + s_end[1] + d1;
        run[0] = run[1] + d0;
        float da_acc = 0.f;
        for (int k = 0; k < 2; ++k) {
            const int l = 2 * lane + k, s = n * p.Q + l;
            if (l < p.Q && s < p.S) {
                const int64_t gi = ((int64_t)b * p.S + s) * p.H + h;
                if (bp.d_da) bp.d_da[gi] = run[k];
                if (bp.d_cs) bp.d_cs[gi] = dcs[l];
                if (bp.d_gs) bp.d_gs[gi] = dgs[l];
                if (bp.d_dt) {   // Mamba-2: da = dt * A_h, cs = gs = dt
                    bp.d_dt[gi] = run[k] * p.a[h] + dcs[l] + dgs[l];
                    da_acc = fmaf(run[k], p.dsrc[gi], da_acc);
                }
            }
        }
        if (bp.d_a) {
            da_acc = sum32(da_acc);
            if (lane == 0) atomicAdd(&bp.d_a[h], da_acc);
        }
        if (p.d && bp.dd) {
            const float v = sum32(lane < 8 ? dds[lane] : 0.f);
            if (lane == 0) atomicAdd(&bp.dd[h], v);
        }
    }
}

}  // namespace

// =============================================================================================
// Wider heads or states (P up to 128, R up to 256, and MIMO ranks above 64): two kernels on 32 x 32 blocks that walk the
// tiles of a chunk, columns and rows apart, with the scalar gradients accumulated in memory.
// =============================================================================================
constexpr int BT = 32;  // fused rows / columns per backward tile

struct BwdWork {
    float* gs;        // [b, h, nc, Q] same-time weights
    float* dstates;   // [b, nc, h, p, r]: readout gradient G_n, overwritten with dS_n by the reverse pass
    float* dcum;      // [b, h, nc, Q] accumulators (zeroed)
    float* dcs;       // [b, h, nc, Q]
    float* dgs;       // [b, h, nc, Q]
    float* daend;     // [b, h, nc]
};

// Reverse state passing of these kernels: dS_n = dh_{n+1}; dh_n = exp(Aend_n) dh_{n+1} + G_n; dAend_n += <dh_{n+1}, exp(Aend_n) h_n>.
__global__ void bwd_state_passing_kernel(Params p, BwdWork w, const float* dh_final, float* dh0) {
    const int PR = p.P * p.R;
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    const int h = blockIdx.y, b = blockIdx.z;
    __shared__ float red[32];
    float dh = (o < PR && dh_final) ? dh_final[((int64_t)b * p.H + h) * PR + o] : 0.f;
    for (int n = p.NC - 1; n >= 0; --n) {
        const int64_t idx = (((int64_t)b * p.NC + n) * p.H + h) * PR + o;
        const float e = expf(p.cum[(((int64_t)b * p.H + h) * p.NC + n) * p.Q + p.Q - 1]);
        float g = 0.f, part = 0.f;
        if (o < PR) {
            g = w.dstates[idx];
            w.dstates[idx] = dh;
            part = dh * e * p.states[idx];
        }
        // block reduction of the dAend contribution
        for (int off = 16; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = part;
        __syncthreads();
        if (threadIdx.x < 32) {
            float v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
            for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
            if (threadIdx.x == 0) atomicAdd(&w.daend[((int64_t)b * p.H + h) * p.NC + n], v);
        }
        __syncthreads();
        dh = fmaf(e, dh, g);
    }
    if (o < PR) dh0[((int64_t)b * p.H + h) * PR + o] = dh;
}

// Shared-memory view used by the two tile kernels.
struct BwdTiles {
    float *dyI, *vJ, *cI, *bJ;   // [BT][P+1], [BT][P+1], [BT][R+1], [BT][R+1]
    float *Ws, *dCBs, *dKs, *Ks; // [BT][BT+1] each
    float* big;                  // [P][R] (dS_n or h_n)
    float* sc;                   // 4 x BT scalars
};
__device__ __forceinline__ BwdTiles carve_tiles(float* sm, int P, int R) {
    BwdTiles t;
    t.dyI = sm; sm += BT * (P + 1);
    t.vJ = sm; sm += BT * (P + 1);
    t.cI = sm; sm += BT * (R + 1);
    t.bJ = sm; sm += BT * (R + 1);
    t.Ws = sm; sm += BT * (BT + 1);
    t.dCBs = sm; sm += BT * (BT + 1);
    t.dKs = sm; sm += BT * (BT + 1);
    t.Ks = sm; sm += BT * (BT + 1);
    t.sc = sm; sm += 4 * BT;
    t.big = sm;
    return t;
}
static size_t bwd_smem_bytes(int P, int R) {
    return sizeof(float) * (size_t)(2 * BT * (P + 1) + 2 * BT * (R + 1) + 4 * BT * (BT + 1) + 4 * BT + P * R);
}

template <typename T>
__device__ __forceinline__ void stage_rows(float* dst, int ld, const T* src, const Params& p, int b, int n, int h_or_g, int HG,
                                           int width, int row0, int tid) {
    // rows = fused indices row0 .. row0 + BT of chunk n; src layout [b, s, m, HG, width]
    const int QM = p.Q * p.M;
    for (int e = tid; e < BT * width; e += kThreads) {
        const int ii = e / width, x = e % width, i = row0 + ii, t = i / p.M, mu = i % p.M, s = n * p.Q + t;
        float val = 0.f;
        if (i < QM && s < p.S) val = to_f32(src[((((int64_t)b * p.S + s) * p.M + mu) * HG + h_or_g) * width + x]);
        dst[ii * ld + x] = val;
    }
}

// dW, CB, kern for the (I, J) block -> Ws = CB*kern, dCBs = dW*kern, dKs = dW*CB, Ks = kern (0 where masked).
__device__ __forceinline__ void block_products(const BwdTiles& t, const Params& p, const float* cum, const float* cs,
                                               const float* gs, int i0, int j0, int tid) {
    const int QM = p.Q * p.M;
#pragma unroll
    for (int k = 0; k < BT * BT / kThreads; ++k) {
        const int o = tid + k * kThreads, ii = o / BT, jj = o % BT, i = i0 + ii, j = j0 + jj;
        float dw = 0.f, cb = 0.f;
        for (int x = 0; x < p.P; ++x) dw = fmaf(t.dyI[ii * (p.P + 1) + x], t.vJ[jj * (p.P + 1) + x], dw);
        for (int x = 0; x < p.R; ++x) cb = fmaf(t.cI[ii * (p.R + 1) + x], t.bJ[jj * (p.R + 1) + x], cb);
        float kern = 0.f;
        if (i < QM && j < QM) {
            const int ti = i / p.M, tj = j / p.M;
            if (tj < ti) kern = expf(cum[ti] - cum[tj]) * cs[tj];
            else if (tj == ti) kern = gs[ti];
        }
        t.Ws[ii * (BT + 1) + jj] = cb * kern;
        t.dCBs[ii * (BT + 1) + jj] = dw * kern;
        t.dKs[ii * (BT + 1) + jj] = dw * cb;
        t.Ks[ii * (BT + 1) + jj] = kern;
    }
}

// Column-tile kernel: everything that is a sum over target rows i for a tile J of source columns:
// dv_J, dB_J, and the column-indexed scalar gradients (dcs, the negative half of dcum, dgs, dAend).
template <typename T>
__global__ void bwd_columns_kernel(Params p, BwdWork w, const T* dy, float* dv, float* db, float* dd) {
    extern __shared__ float sm[];
    BwdTiles t = carve_tiles(sm, p.P, p.R);
    const int tid = threadIdx.x;
    const int QM = p.Q * p.M, ntile = (QM + BT - 1) / BT;
    int64_t bx = blockIdx.x;
    const int jt = bx % ntile, h = (bx / ntile) % p.H, n = bx / ((int64_t)ntile * p.H), b = blockIdx.y;
    const int hpg = p.H / p.G, g = h / hpg, j0 = jt * BT;
    const int64_t cbase = (((int64_t)b * p.H + h) * p.NC + n) * p.Q;
    const float *cum = p.cum + cbase, *cs = p.cs + cbase, *gs = w.gs + cbase;
    const float aend = cum[p.Q - 1];
    const T* v = static_cast<const T*>(p.v);
    const T* bm_ = static_cast<const T*>(p.bmat);
    const T* cm = static_cast<const T*>(p.cmat);
    float* colacc = t.sc;  // [0..BT) dcs, [BT..2BT) -dcum, [2BT..3BT) dgs, [3BT..4BT) dw
    for (int e = tid; e < 4 * BT; e += kThreads) colacc[e] = 0.f;
    stage_rows(t.vJ, p.P + 1, v, p, b, n, h, p.H, p.P, j0, tid);
    stage_rows(t.bJ, p.R + 1, bm_, p, b, n, g, p.G, p.R, j0, tid);
    constexpr int MAXV = 16, MAXB = 32;  // per-thread outputs: BT*P/256 <= 16 (P <= 128), BT*R/256 <= 32 (R <= 256)
    float acc_v[MAXV], acc_b[MAXB];
#pragma unroll
    for (int k = 0; k < MAXV; ++k) acc_v[k] = 0.f;
#pragma unroll
    for (int k = 0; k < MAXB; ++k) acc_b[k] = 0.f;
    const int nv = BT * p.P, nb = BT * p.R;
    // target rows with t_i >= t_j: start at the tile holding the first fused index of time t(j0)
    // (a time step's M rows may straddle a tile boundary when M does not divide the tile size)
    for (int it = ((j0 / p.M) * p.M) / BT; it < ntile; ++it) {
        const int i0 = it * BT;
        __syncthreads();
        stage_rows(t.dyI, p.P + 1, dy, p, b, n, h, p.H, p.P, i0, tid);
        stage_rows(t.cI, p.R + 1, cm, p, b, n, g, p.G, p.R, i0, tid);
        __syncthreads();
        block_products(t, p, cum, cs, gs, i0, j0, tid);
        __syncthreads();
        // column scalars
        for (int e = tid; e < BT * BT; e += kThreads) {
            const int ii = e / BT, jj = e % BT, i = i0 + ii, j = j0 + jj;
            if (i < QM && j < QM) {
                const int ti = i / p.M, tj = j / p.M;
                const float dk = t.dKs[ii * (BT + 1) + jj];
                if (tj < ti) {
                    atomicAdd(&colacc[jj], dk * expf(cum[ti] - cum[tj]));
                    atomicAdd(&colacc[BT + jj], dk * t.Ks[ii * (BT + 1) + jj]);
                } else if (tj == ti) {
                    atomicAdd(&colacc[2 * BT + jj], dk);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < MAXV; ++k) {
            const int o = tid + k * kThreads;
            if (o < nv) {
                const int jj = o / p.P, x = o % p.P;
                float a = acc_v[k];
                for (int ii = 0; ii < BT; ++ii) a = fmaf(t.Ws[ii * (BT + 1) + jj], t.dyI[ii * (p.P + 1) + x], a);
                acc_v[k] = a;
            }
        }
#pragma unroll
        for (int k = 0; k < MAXB; ++k) {
            const int o = tid + k * kThreads;
            if (o < nb) {
                const int jj = o / p.R, x = o % p.R;
                float a = acc_b[k];
                for (int ii = 0; ii < BT; ++ii) a = fmaf(t.dCBs[ii * (BT + 1) + jj], t.cI[ii * (p.R + 1) + x], a);
                acc_b[k] = a;
            }
        }
    }
    // ---- chunk-state term: dS_n = dh_{n+1}
    __syncthreads();
    const float* dS = w.dstates + (((int64_t)b * p.NC + n) * p.H + h) * (int64_t)p.P * p.R;
    for (int e = tid; e < p.P * p.R; e += kThreads) t.big[e] = dS[e];
    // dy of the J tile for the skip term (reuses the dyI buffer)
    stage_rows(t.dyI, p.P + 1, dy, p, b, n, h, p.H, p.P, j0, tid);
    __syncthreads();
    float dd_part = 0.f;
#pragma unroll
    for (int k = 0; k < MAXV; ++k) {
        const int o = tid + k * kThreads;
        if (o < nv) {
            const int jj = o / p.P, x = o % p.P, j = j0 + jj, tj = j / p.M;
            const float wj = j < QM ? cs[tj] * expf(aend - cum[tj]) : 0.f;
            float t1 = 0.f;
            for (int r = 0; r < p.R; ++r) t1 = fmaf(t.big[x * p.R + r], t.bJ[jj * (p.R + 1) + r], t1);
            acc_v[k] = fmaf(wj, t1, acc_v[k]);
            atomicAdd(&colacc[3 * BT + jj], t.vJ[jj * (p.P + 1) + x] * t1);   // dw_j = v_j^T dS B_j
            const float dyv = t.dyI[jj * (p.P + 1) + x];
            if (p.d) {
                acc_v[k] = fmaf(p.d[h], dyv, acc_v[k]);
                dd_part = fmaf(dyv, t.vJ[jj * (p.P + 1) + x], dd_part);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < MAXB; ++k) {
        const int o = tid + k * kThreads;
        if (o < nb) {
            const int jj = o / p.R, x = o % p.R, j = j0 + jj, tj = j / p.M;
            const float wj = j < QM ? cs[tj] * expf(aend - cum[tj]) : 0.f;
            float t2 = 0.f;
            for (int pp = 0; pp < p.P; ++pp) t2 = fmaf(t.big[pp * p.R + x], t.vJ[jj * (p.P + 1) + pp], t2);
            acc_b[k] = fmaf(wj, t2, acc_b[k]);
        }
    }
    if (p.d && dd) {
        for (int off = 16; off > 0; off >>= 1) dd_part += __shfl_xor_sync(0xffffffffu, dd_part, off);
        if ((tid & 31) == 0) atomicAdd(&dd[h], dd_part);
    }
    __syncthreads();
    // ---- outputs
#pragma unroll
    for (int k = 0; k < MAXV; ++k) {
        const int o = tid + k * kThreads;
        if (o < nv) {
            const int jj = o / p.P, x = o % p.P, j = j0 + jj, tj = j / p.M, mu = j % p.M, s = n * p.Q + tj;
            if (j < QM && s < p.S) dv[((((int64_t)b * p.S + s) * p.M + mu) * p.H + h) * p.P + x] = acc_v[k];
        }
    }
#pragma unroll
    for (int k = 0; k < MAXB; ++k) {
        const int o = tid + k * kThreads;
        if (o < nb) {
            const int jj = o / p.R, x = o % p.R, j = j0 + jj, tj = j / p.M, mu = j % p.M, s = n * p.Q + tj;
            if (j < QM && s < p.S) {
                float* dst = db + ((((int64_t)b * p.S + s) * p.M + mu) * p.G + g) * p.R + x;
                if (hpg > 1) atomicAdd(dst, acc_b[k]); else *dst = acc_b[k];
            }
        }
    }
    for (int jj = tid; jj < BT; jj += kThreads) {
        const int j = j0 + jj;
        if (j < QM) {
            const int tj = j / p.M;
            const float e_end = expf(aend - cum[tj]), wj = cs[tj] * e_end, dw = colacc[3 * BT + jj];
            atomicAdd(&w.dcs[cbase + tj], colacc[jj] + dw * e_end);
            atomicAdd(&w.dcum[cbase + tj], -(colacc[BT + jj] + dw * wj));
            atomicAdd(&w.dgs[cbase + tj], colacc[2 * BT + jj]);
            atomicAdd(&w.daend[((int64_t)b * p.H + h) * p.NC + n], dw * wj);
        }
    }
}

// Row-tile kernel: everything that is a sum over source columns j for a tile I of target rows:
// dC_I and the positive half of dcum (intra-chunk term and state-readout term).
template <typename T>
__global__ void bwd_rows_kernel(Params p, BwdWork w, const T* dy, float* dc) {
    extern __shared__ float sm[];
    BwdTiles t = carve_tiles(sm, p.P, p.R);
    const int tid = threadIdx.x;
    const int QM = p.Q * p.M, ntile = (QM + BT - 1) / BT;
    int64_t bx = blockIdx.x;
    const int it = bx % ntile, h = (bx / ntile) % p.H, n = bx / ((int64_t)ntile * p.H), b = blockIdx.y;
    const int hpg = p.H / p.G, g = h / hpg, i0 = it * BT;
    const int64_t cbase = (((int64_t)b * p.H + h) * p.NC + n) * p.Q;
    const float *cum = p.cum + cbase, *cs = p.cs + cbase, *gs = w.gs + cbase;
    const T* v = static_cast<const T*>(p.v);
    const T* bm_ = static_cast<const T*>(p.bmat);
    const T* cm = static_cast<const T*>(p.cmat);
    float* rowacc = t.sc;  // [0..BT) +dcum
    for (int e = tid; e < 4 * BT; e += kThreads) rowacc[e] = 0.f;
    stage_rows(t.dyI, p.P + 1, dy, p, b, n, h, p.H, p.P, i0, tid);
    stage_rows(t.cI, p.R + 1, cm, p, b, n, g, p.G, p.R, i0, tid);
    constexpr int MAXC = 32;
    float acc_c[MAXC];
#pragma unroll
    for (int k = 0; k < MAXC; ++k) acc_c[k] = 0.f;
    const int nc_out = BT * p.R;
    // source columns with t_j <= t_i: up to the tile holding the last fused index of time t(i_last)
    const int i_last = min(i0 + BT, QM) - 1;
    const int jt_end = min(ntile - 1, (((i_last / p.M) + 1) * p.M - 1) / BT);
    for (int jt = 0; jt <= jt_end; ++jt) {
        const int j0 = jt * BT;
        __syncthreads();
        stage_rows(t.vJ, p.P + 1, v, p, b, n, h, p.H, p.P, j0, tid);
        stage_rows(t.bJ, p.R + 1, bm_, p, b, n, g, p.G, p.R, j0, tid);
        __syncthreads();
        block_products(t, p, cum, cs, gs, i0, j0, tid);
        __syncthreads();
        for (int e = tid; e < BT * BT; e += kThreads) {
            const int ii = e / BT, jj = e % BT, i = i0 + ii, j = j0 + jj;
            if (i < QM && j < QM && j / p.M < i / p.M)
                atomicAdd(&rowacc[ii], t.dKs[ii * (BT + 1) + jj] * t.Ks[ii * (BT + 1) + jj]);
        }
#pragma unroll
        for (int k = 0; k < MAXC; ++k) {
            const int o = tid + k * kThreads;
            if (o < nc_out) {
                const int ii = o / p.R, x = o % p.R;
                float a = acc_c[k];
                for (int jj = 0; jj < BT; ++jj) a = fmaf(t.dCBs[ii * (BT + 1) + jj], t.bJ[jj * (p.R + 1) + x], a);
                acc_c[k] = a;
            }
        }
    }
    // ---- state-readout term: dC_i += e_i h_n^T dy_i ; dcum_ti += C_i . (that)
    __syncthreads();
    const float* hin = p.states + (((int64_t)b * p.NC + n) * p.H + h) * (int64_t)p.P * p.R;
    for (int e = tid; e < p.P * p.R; e += kThreads) t.big[e] = hin[e];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < MAXC; ++k) {
        const int o = tid + k * kThreads;
        if (o < nc_out) {
            const int ii = o / p.R, x = o % p.R, i = i0 + ii;
            if (i < QM) {
                const float ei = expf(cum[i / p.M]);
                float t3 = 0.f;
                for (int pp = 0; pp < p.P; ++pp) t3 = fmaf(t.dyI[ii * (p.P + 1) + pp], t.big[pp * p.R + x], t3);
                t3 *= ei;
                acc_c[k] += t3;
                atomicAdd(&rowacc[ii], t.cI[ii * (p.R + 1) + x] * t3);
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < MAXC; ++k) {
        const int o = tid + k * kThreads;
        if (o < nc_out) {
            const int ii = o / p.R, x = o % p.R, i = i0 + ii, ti = i / p.M, mu = i % p.M, s = n * p.Q + ti;
            if (i < QM && s < p.S) {
                float* dst = dc + ((((int64_t)b * p.S + s) * p.M + mu) * p.G + g) * p.R + x;
                if (hpg > 1) atomicAdd(dst, acc_c[k]); else *dst = acc_c[k];
            }
        }
    }
    for (int ii = tid; ii < BT; ii += kThreads) {
        const int i = i0 + ii;
        if (i < QM) atomicAdd(&w.dcum[cbase + i / p.M], rowacc[ii]);
    }
}

// Finalise: dcum[Q-1] += dAend; d_da = suffix sum of dcum over the chunk; scatter to [b, s, h] outputs.
__global__ void bwd_finalize_kernel(Params p, BwdWork w, float* d_da, float* d_cs, float* d_gs, float* d_dt, float* d_a) {
    int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t total = (int64_t)p.B * p.NC * p.H;
    if (idx >= total) return;
    const int h = idx % p.H, n = (idx / p.H) % p.NC, b = idx / ((int64_t)p.H * p.NC);
    const int64_t cbase = (((int64_t)b * p.H + h) * p.NC + n) * p.Q;
    float run = w.daend[((int64_t)b * p.H + h) * p.NC + n];
    float da_acc = 0.f;
    for (int l = p.Q - 1; l >= 0; --l) {
        run += w.dcum[cbase + l];
        const int s = n * p.Q + l;
        if (s < p.S) {
            const int64_t g = ((int64_t)b * p.S + s) * p.H + h;
            if (d_da) d_da[g] = run;
            if (d_cs) d_cs[g] = w.dcs[cbase + l];
            if (d_gs) d_gs[g] = w.dgs[cbase + l];
            if (d_dt) {   // Mamba-2: da = dt * A_h, cs = gs = dt
                const float dt = p.dsrc[g];
                d_dt[g] = run * p.a[h] + w.dcs[cbase + l] + w.dgs[cbase + l];
                da_acc = fmaf(run, dt, da_acc);
            }
        }
    }
    if (d_a) atomicAdd(&d_a[h], da_acc);
}

static bool one_tile(const Params& p) { return p.P <= TP && p.R <= 128 && p.M <= TR; }

static size_t scan_bytes(int B, int S, int H, int q) { return align_up((size_t)B * H * cdiv(S, q) * q * sizeof(float), 256); }
static size_t state_bytes(int B, int S, int H, int P, int R, int q) { return align_up((size_t)B * cdiv(S, q) * H * P * R * sizeof(float), 256); }

// Workspace of the one-tile kernel and of the block kernels at chunk length q.
static size_t tile_bytes(int B, int S, int H, int P, int R, int q) { return 2 * scan_bytes(B, S, H, q) + 2 * state_bytes(B, S, H, P, R, q); }
static size_t blocks_bytes(int B, int S, int H, int P, int R, int q, bool mamba2) {
    const size_t ae = align_up((size_t)B * H * cdiv(S, q) * sizeof(float), 256);
    const size_t outs = mamba2 ? align_up((size_t)B * S * H * sizeof(float), 256) : 0;  // internal d_da of Mamba-2
    return 6 * scan_bytes(B, S, H, q) + 2 * state_bytes(B, S, H, P, R, q) + ae + outs;
}
size_t bwd_workspace_bytes(int B, int S, int H, int P, int R, int M, int Q, bool mamba2) {
    Params p{};
    p.P = P, p.R = R, p.M = M;
    const int q = inner_chunk(Q, M, false);
    return one_tile(p) ? tile_bytes(B, S, H, P, R, q) : blocks_bytes(B, S, H, P, R, q, mamba2);
}
size_t bwd_least_bytes(int B, int S, int H, int P, int R, int M, int Q, bool mamba2) {
    return std::min(bwd_workspace_bytes(B, S, H, P, R, M, Q, mamba2), blocks_bytes(B, S, H, P, R, Q, mamba2));
}

template <typename T, bool VEC, int W>
static int32_t launch_tile(const BwdParams& bp, const float* dstates, cudaStream_t stream) {
    const Params& p = bp.fwd;
    auto kernel = bwd_tile_kernel<T, VEC, W>;
    const size_t smem = sizeof(float) * (size_t)(3 * TR * (W + 4) + 4 * TR * LDX);
    if (int32_t e = check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "cudaFuncSetAttribute(bwd_tile)"))
        return e;
    kernel<<<dim3((unsigned)((int64_t)p.H * p.NC), p.B), kThreads, smem, stream>>>(bp, dstates);
    return check_launch("bwd_tile");
}
template <typename T>
static int32_t launch_tile(const BwdParams& bp, const float* dstates, cudaStream_t stream) {
    const Params& p = bp.fwd;
    const bool vec = p.P % 4 == 0 && p.R % 4 == 0, wide = p.R > 64;
    if (vec) return wide ? launch_tile<T, true, 128>(bp, dstates, stream) : launch_tile<T, true, 64>(bp, dstates, stream);
    return wide ? launch_tile<T, false, 128>(bp, dstates, stream) : launch_tile<T, false, 64>(bp, dstates, stream);
}

template <typename T>
static int32_t launch_blocks(BwdParams bp, BwdWork w, cudaStream_t stream) {
    Params& p = bp.fwd;
    const T* dy = static_cast<const T*>(bp.dy);
    const size_t smem = bwd_smem_bytes(p.P, p.R);
    cudaError_t e = cudaFuncSetAttribute(bwd_columns_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(bwd_rows_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(bwd)");
    if (int32_t er = launch_state_passing(p, nullptr, nullptr, nullptr, stream)) return er;
    dim3 grid4((unsigned)cdiv((int64_t)p.P * p.R, kThreads), p.H, p.B);
    bwd_state_passing_kernel<<<grid4, kThreads, 0, stream>>>(p, w, bp.dh_final, bp.dh0);
    if (int32_t er = check_launch("bwd_state_passing")) return er;
    const int64_t ntile = cdiv((int64_t)p.Q * p.M, BT);
    dim3 grid((unsigned)(ntile * p.H * p.NC), p.B);
    bwd_columns_kernel<T><<<grid, kThreads, smem, stream>>>(p, w, dy, bp.dv, bp.db, bp.dd);
    if (int32_t er = check_launch("bwd_columns")) return er;
    bwd_rows_kernel<T><<<grid, kThreads, smem, stream>>>(p, w, dy, bp.dc);
    if (int32_t er = check_launch("bwd_rows")) return er;
    int64_t total = (int64_t)p.B * p.NC * p.H;
    bwd_finalize_kernel<<<(unsigned)cdiv(total, 128), 128, 0, stream>>>(p, w, bp.d_da, bp.d_cs, bp.d_gs, bp.d_dt, bp.d_a);
    return check_launch("bwd_finalize");
}

int32_t run_bwd(BwdParams bp, void* workspace, size_t ws_bytes, cudaStream_t stream) {
    Params& p = bp.fwd;
    const bool mamba2 = bp.d_dt != nullptr;
    const size_t need = bwd_least_bytes(p.B, p.S, p.H, p.P, p.R, p.M, p.Q, mamba2);
    if (workspace == nullptr || ws_bytes < need)
        return fail(BM_ERR_WORKSPACE_TOO_SMALL, "workspace of %zu bytes given, %zu needed", ws_bytes, need);
    if (!aligned16(workspace)) return fail(BM_ERR_BAD_ALIGNMENT, "workspace is not 16-byte aligned");
    if (p.P > 128 || p.R > 256) return fail(BM_ERR_UNSUPPORTED, "backward supports headdim <= 128 and state_rank <= 256");
    if (bwd_smem_bytes(p.P, p.R) > 200 * 1024) return fail(BM_ERR_UNSUPPORTED, "headdim x state_rank too large for the backward tiles");
    if (p.B > 65535 || p.H > 65535) return fail(BM_ERR_UNSUPPORTED, "batch / nheads above 65535");
    // A workspace that does not hold the states of one-tile chunks is served by the block kernels at longer chunks.
    int q = inner_chunk(p.Q, p.M, false);
    const bool tile = one_tile(p) && ws_bytes >= tile_bytes(p.B, p.S, p.H, p.P, p.R, q);
    while (!tile && q < p.Q && ws_bytes < blocks_bytes(p.B, p.S, p.H, p.P, p.R, q, mamba2)) q = longer_chunk(q, p.Q, false);
    p.Q = q;
    p.NC = (int)cdiv(p.S, p.Q);
    p.states_out = nullptr, p.h_final = nullptr;   // the final state is not an output of the backward
    const size_t per = scan_bytes(p.B, p.S, p.H, p.Q), st = state_bytes(p.B, p.S, p.H, p.P, p.R, p.Q);
    char* wp = static_cast<char*>(workspace);
    p.cum = reinterpret_cast<float*>(wp); wp += per;
    p.cs = reinterpret_cast<float*>(wp); wp += per;
    p.states = reinterpret_cast<float*>(wp); wp += st;
    BwdWork w{};
    w.dstates = reinterpret_cast<float*>(wp); wp += st;
    if (!tile) {
        w.gs = reinterpret_cast<float*>(wp); wp += per;
        p.gs = w.gs;
        char* zero_begin = wp;   // accumulators, contiguous so that one memset clears them
        w.dcum = reinterpret_cast<float*>(wp); wp += per;
        w.dcs = reinterpret_cast<float*>(wp); wp += per;
        w.dgs = reinterpret_cast<float*>(wp); wp += per;
        w.daend = reinterpret_cast<float*>(wp); wp += align_up((size_t)p.B * p.H * p.NC * sizeof(float), 256);
        if (int32_t e = check_cuda(cudaMemsetAsync(zero_begin, 0, (size_t)(wp - zero_begin), stream), "cudaMemsetAsync(accumulators)")) return e;
        if (mamba2 && bp.d_da == nullptr) bp.d_da = reinterpret_cast<float*>(wp);
    }
    // gradients that several CTAs add into (B / C of a group's heads, D, A) are cleared by the first kernel
    const int64_t bc = p.H / p.G > 1 ? (int64_t)p.B * p.S * p.M * p.G * p.R : 0;
    if (int32_t e = launch_chunk_state(p, bp.dy, w.dstates, bp.db, bp.dc, bc, bp.dd, bp.d_a, stream)) return e;
    if (!tile) return p.dtype == BM_DTYPE_F32 ? launch_blocks<float>(bp, w, stream) : launch_blocks<__nv_bfloat16>(bp, w, stream);
    if (int32_t e = launch_state_passing(p, w.dstates, bp.dh_final, bp.dh0, stream)) return e;
    return p.dtype == BM_DTYPE_F32 ? launch_tile<float>(bp, w.dstates, stream) : launch_tile<__nv_bfloat16>(bp, w.dstates, stream);
}

}  // namespace exact
}  // namespace bm
