// Building blocks of the float32 chunked-SSD kernels (ssd_exact.cu, ssd_exact_bwd.cu): staging of a tile's rows into
// shared memory and register-tiled products of 64-row tiles on the float32 pipe.
//
// All products run with 256 threads as a 16 x 16 grid (ty = tid / 16, tx = tid % 16); a thread owns the rows
// 4 ty .. 4 ty + 3 of the output.  Operands come from shared memory as 128-bit reads: per 64 multiply-adds a thread
// issues 8 reads, and the row pitch of every k-contiguous operand is 4 floats more than a multiple of 32, so the 16
// rows a half-warp reads fall into distinct banks.  What bounds them is the operands' way to the float32 pipe: it is busy
// 38 to 54 % of the time, the shared-memory pipe 56 to 65 %, issue slots 50 to 72 % (ncu, b8 L2048 H16 P64 N128).
#pragma once
#include "ssd_exact.cuh"

namespace bm {
namespace exact {

constexpr int kThreads = 256;
constexpr int TR = 64;        // fused (time, rank) rows of a tile
constexpr int TP = 64;        // head-dimension columns of a block
constexpr int LDX = TP + 4;   // pitch of k-contiguous 64-wide tiles

// One B/C element for (row pointer, r) with the optional data-dependent rotation applied
// (src/modules/misc/rope.rs:50-170): pairwise mode rotates (2j, 2j+1), half mode (j, j + R/2);
// only the first rope_dim entries (pairwise) / first rope_dim/2 of each half rotate.
template <typename T>
__device__ __forceinline__ float bc_elem(const T* row, const float* ang, int r, int R, int rope_dim, int pairwise) {
    float self = to_f32(row[r]);
    if (ang == nullptr || rope_dim == 0) return self;
    if (pairwise) {
        if (r >= rope_dim) return self;
        int j = r >> 1;
        float th = wrap_angle(ang[j]);
        float c = cosf(th), s = sinf(th);
        float other = to_f32(row[r ^ 1]);
        return (r & 1) ? (s * other + c * self) : (c * self - s * other);
    }
    int half = R >> 1, na = rope_dim >> 1;
    if (r < na) {
        float th = wrap_angle(ang[r]);
        return cosf(th) * self - sinf(th) * to_f32(row[r + half]);
    }
    if (r >= half && r < half + na) {
        float th = wrap_angle(ang[r - half]);
        return sinf(th) * to_f32(row[r - half]) + cosf(th) * self;
    }
    return self;
}

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Four consecutive values as float32 (the caller has checked the alignment).
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    return make_float4(a.x, a.y, b.x, b.y);
}

// Rows of a tile: element index of row i's first entry in units of rows, (b S + s) M + mu, or -1 past the end; and its
// time step inside the chunk.  `i0`: first fused row of the tile inside the chunk.
struct TileRows {
    int64_t idx[TR];
    int t[TR];
};
__device__ __forceinline__ void fill_rows(TileRows& tr, const Params& p, int b, int n, int i0, int tid) {
    if (tid < TR) {
        const int i = i0 + tid, t = i / p.M, mu = i - t * p.M, s = n * p.Q + t;
        const bool live = i < p.Q * p.M && s < p.S;
        tr.idx[tid] = live ? ((int64_t)b * p.S + s) * p.M + mu : -1;
        tr.t[tid] = min(t, p.Q - 1);
    }
}

// Stages columns [c0, c0 + W) of the tile's rows of src [rows, HG, width] (slice hg) into dst with pitch ld; entries past
// the row or past the width become zero.  VEC: width and c0 are multiples of 4.  float32 tiles go by cp.async (the
// caller commits and waits), bf16 tiles are widened on the way.
template <typename T, bool VEC, int W>
__device__ __forceinline__ void stage(float* dst, int ld, const T* src, const TileRows& tr, int HG, int hg, int width, int c0, int tid) {
    constexpr int V4 = W / 4;
#pragma unroll 4
    for (int e = tid; e < TR * V4; e += kThreads) {
        const int i = e / V4, c = (e % V4) * 4;
        const int64_t ri = tr.idx[i];
        float* d = dst + i * ld + c;
        if (ri < 0 || c0 + c >= width) {
            *reinterpret_cast<float4*>(d) = make_float4(0.f, 0.f, 0.f, 0.f);
            continue;
        }
        const T* s = src + (ri * HG + hg) * width + c0 + c;
        if constexpr (VEC) {
            if constexpr (sizeof(T) == 4) cp_async16(d, reinterpret_cast<const float*>(s));
            else *reinterpret_cast<float4*>(d) = load4(s);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) d[k] = c0 + c + k < width ? to_f32(s[k]) : 0.f;
        }
    }
}
// The same for B / C with the rotation applied while loading (angles given).
template <typename T, int W>
__device__ __forceinline__ void stage_rotated(float* dst, int ld, const T* src, const TileRows& tr, const Params& p, int g, int h, int c0,
                                              int tid) {
    const int na = p.rope_dim >> 1;
    for (int e = tid; e < TR * W; e += kThreads) {
        const int i = e / W, c = e % W, r = c0 + c;
        const int64_t ri = tr.idx[i];
        float v = 0.f;
        if (ri >= 0 && r < p.R) v = bc_elem(src + (ri * p.G + g) * p.R, p.angles + (ri / p.M * p.H + h) * na, r, p.R, p.rope_dim, p.pairwise);
        dst[i * ld + c] = v;
    }
}
template <typename T, bool VEC, int W>
__device__ __forceinline__ void stage_bc(float* dst, int ld, const void* src, const TileRows& tr, const Params& p, int g, int h, int c0, int tid) {
    if (p.angles) stage_rotated<T, W>(dst, ld, static_cast<const T*>(src), tr, p, g, h, c0, tid);
    else stage<T, VEC, W>(dst, ld, static_cast<const T*>(src), tr, p.G, g, p.R, c0, tid);
}
// State block h[p0 .. p0 + 64)[c0 .. c0 + W) of a [P][R] float32 matrix; row p lands at row (p % 4) * 16 + p / 4, so that
// a thread of the k-contiguous product below finds the columns 4 tx .. 4 tx + 3 of its output 16 rows apart.
template <bool VEC, int W>
__device__ __forceinline__ void stage_state(float* dst, int ld, const float* src, int P, int R, int p0, int c0, int tid) {
    constexpr int V4 = W / 4;
#pragma unroll 4
    for (int e = tid; e < TP * V4; e += kThreads) {
        const int pp = e / V4, c = (e % V4) * 4;
        float* d = dst + ((pp & 3) * 16 + (pp >> 2)) * ld + c;
        if (p0 + pp >= P || c0 + c >= R) {
            *reinterpret_cast<float4*>(d) = make_float4(0.f, 0.f, 0.f, 0.f);
            continue;
        }
        const float* s = src + (int64_t)(p0 + pp) * R + c0 + c;
        if constexpr (VEC) {
            cp_async16(d, s);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) d[k] = c0 + c + k < R ? s[k] : 0.f;
        }
    }
}

__device__ __forceinline__ float f4(const float4& v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }

// acc[i][j] += sum_k A[i][k] B[j][k]: both operands k-contiguous; A at the thread's first row, B at row tx with the
// thread's NJ columns 16 rows apart.  K a multiple of 4.
template <int NJ>
__device__ __forceinline__ void mul_kk(const float* A, int lda, const float* B, int ldb, int K, float (&acc)[4][4]) {
#pragma unroll 2
    for (int k = 0; k < K; k += 4) {
        float4 a[4], b[NJ];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = load4(A + i * lda + k);
#pragma unroll
        for (int j = 0; j < NJ; ++j) b[j] = load4(B + j * 16 * ldb + k);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < NJ; ++j) acc[i][j] = fmaf(f4(a[i], kk), f4(b[j], kk), acc[i][j]);
    }
}
// acc[i][4 q + j] += sum_k A[i][k] B[k][64 q + 4 tx + j]: A k-contiguous, B row k at B + brow(k) ldb.  `PERM`: B's rows
// are stored in the order of stage_state.
template <int NQ, bool PERM>
__device__ __forceinline__ void mul_km(const float* A, int lda, const float* B, int ldb, int K, float (&acc)[4][4 * NQ]) {
#pragma unroll 2
    for (int k = 0; k < K; k += 4) {
        float4 a[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = load4(A + i * lda + k);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const float* row = B + (PERM ? kk * 16 + (k >> 2) : k + kk) * ldb;
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const float4 b = load4(row + q * 64);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float av = f4(a[i], kk);
                    acc[i][4 * q + 0] = fmaf(av, b.x, acc[i][4 * q + 0]);
                    acc[i][4 * q + 1] = fmaf(av, b.y, acc[i][4 * q + 1]);
                    acc[i][4 * q + 2] = fmaf(av, b.z, acc[i][4 * q + 2]);
                    acc[i][4 * q + 3] = fmaf(av, b.w, acc[i][4 * q + 3]);
                }
            }
        }
    }
}
// acc[i][4 q + j] += sum_k A[k][i] B[k][64 q + j]: both operands k-outer (A at the thread's first column, B at 4 tx).
template <int NQ>
__device__ __forceinline__ void mul_mm(const float* A, int lda, const float* B, int ldb, int k0, int K, float (&acc)[4][4 * NQ]) {
#pragma unroll 4
    for (int k = k0; k < K; ++k) {
        const float4 a = load4(A + k * lda);
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const float4 b = load4(B + k * ldb + q * 64);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float av = f4(a, i);
                acc[i][4 * q + 0] = fmaf(av, b.x, acc[i][4 * q + 0]);
                acc[i][4 * q + 1] = fmaf(av, b.y, acc[i][4 * q + 1]);
                acc[i][4 * q + 2] = fmaf(av, b.z, acc[i][4 * q + 2]);
                acc[i][4 * q + 3] = fmaf(av, b.w, acc[i][4 * q + 3]);
            }
        }
    }
}
// mul_kk over the first nj (1..4, warp-uniform) column groups only.
__device__ __forceinline__ void mul_kk_upto(int nj, const float* A, int lda, const float* B, int ldb, int K, float (&acc)[4][4]) {
    switch (nj) {
        case 1: mul_kk<1>(A, lda, B, ldb, K, acc); break;
        case 2: mul_kk<2>(A, lda, B, ldb, K, acc); break;
        case 3: mul_kk<3>(A, lda, B, ldb, K, acc); break;
        default: mul_kk<4>(A, lda, B, ldb, K, acc); break;
    }
}

// ---- launches shared by the forward and the backward -----------------------------------------------------------
// Chunk length the kernels use inside for a caller's chunk length Q: the result does not depend on it.
int inner_chunk(int Q, int M, bool want_states);
// The next longer one, where the scratch does not hold the states of chunks of q.
int longer_chunk(int q, int Q, bool want_states);
// K1 + K3: decay scan of every chunk and its state S_n (and, with `dy`, the readout gradient G_n into `dstates`); zeroes
// `zero_n` floats at each of zero_a / zero_b on the way (accumulators of a later kernel; may be NULL).
int32_t launch_chunk_state(const Params& p, const void* dy, float* dstates, float* zero_a, float* zero_b, int64_t zero_n, float* zero_h1,
                           float* zero_h2, cudaStream_t stream);
// K4 forward and, with `dstates`, the reverse recurrence of the backward in the same launch.
int32_t launch_state_passing(const Params& p, float* dstates, const float* dh_final, float* dh0, cudaStream_t stream);

}  // namespace exact
}  // namespace bm
