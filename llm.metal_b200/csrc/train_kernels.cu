// Row-wise and attention kernels of the LoRA-SFT step (everything but the GEMMs).
//
// Arithmetic follows shaders/q8_kernels.metal: rms_norm :133-158,
// rms_norm_train_backward :584-624, rope_train :495-538, rope_train_bwd
// :997-1040, attn_train_fwd :769-851, attn_bwd_dq :857-925, attn_bwd_dkv
// :931-968, repeat_kv / repeat_kv_bwd :476-492 / :973-992 (folded into the
// indexing), silu_mul :337-348, silu_mul_backward :540-556, softmax_ce_train
// :646-690, scale_tensor :627-633, clamp_tensor :1155-1161; the optimiser
// follows src/nn/fast_sft.c:1045-1107. All fp32 (the gradient norm in double).
//
// These kernels move little data next to the projections (a few MB per layer
// against hundreds of MB of weights); they are written for fusion -- no
// transposed or repeated copies, residual adds and scalings folded in -- rather
// than for peak bandwidth.
#include "common.cuh"
#include "../../include/llmb200_train_kernels.h"

extern unsigned long long g_b200_launches;

namespace {

// ---- embedding -----------------------------------------------------------------------------
__global__ void embed_rows_kernel(const float *emb, const uint32_t *tokens, int dim, int vocab, float scale, float *x)
{
    const int m = blockIdx.x;
    uint32_t t = tokens[m];
    if (t >= (uint32_t)vocab) t = 0;                                  // never read outside the table
    const float *src = emb + (size_t)t * dim;
    float *dst = x + (size_t)m * dim;
    for (int i = threadIdx.x; i < dim; i += blockDim.x) dst[i] = src[i] * scale;
}

// ---- RMSNorm over rows: a group of G threads per row (G = 32 for short rows, 256 for long ones) -----
template <int G>
__device__ __forceinline__ float group_sum_f(float v, float *sh)
{
    v = warp_sum(v);
    if (G == 32) return v;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sh[w] = v;
    __syncthreads();
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < G / 32; ++i) t += sh[i];
    return t;
}

template <int G>
__global__ void __launch_bounds__(256)
rms_norm_rows_kernel(const float *x, const float *gamma, float *out, __half *out_h, int rows, int dim, float eps)
{
    __shared__ float sh[8];
    const int row = blockIdx.x * (256 / G) + threadIdx.x / G;
    const int l = threadIdx.x % G;
    const bool on = row < rows;
    const float *xr = x + (size_t)(on ? row : 0) * dim;
    float ss = 0.f;
    if (on) for (int i = l; i < dim; i += G) { const float v = xr[i]; ss = fmaf(v, v, ss); }
    ss = group_sum_f<G>(ss, sh);
    if (!on) return;
    const float inv = rsqrtf(ss / (float)dim + eps);
    float *o = out + (size_t)row * dim;
    for (int i = l; i < dim; i += G) {
        const float v = xr[i] * inv * gamma[i];
        o[i] = v;
        if (out_h) out_h[(size_t)row * dim + i] = __float2half_rn(v);
    }
}

template <int G>
__global__ void __launch_bounds__(256)
rms_norm_bwd_rows_kernel(const float *x, const float *dy, long long dy_ld, const float *gamma, float *dx, int rows,
                         int dim, float eps, int accumulate, float clamp, __half *dx_h, float h_scale)
{
    __shared__ float sh[8];
    const int row = blockIdx.x * (256 / G) + threadIdx.x / G;
    const int l = threadIdx.x % G;
    const bool on = row < rows;
    const float *xr = x + (size_t)(on ? row : 0) * dim, *dr = dy + (size_t)(on ? row : 0) * dy_ld;
    float ss = 0.f, dot = 0.f;
    if (on) for (int i = l; i < dim; i += G) {
        const float v = xr[i];
        ss = fmaf(v, v, ss);
        dot = fmaf(dr[i] * gamma[i], v, dot);
    }
    ss = group_sum_f<G>(ss, sh);
    dot = group_sum_f<G>(dot, sh);
    if (!on) return;
    const float inv = rsqrtf(ss / (float)dim + eps);
    const float coeff = dot * inv * inv / (float)dim;
    float *o = dx + (size_t)row * dim;
    for (int i = l; i < dim; i += G) {
        float v = (gamma[i] * dr[i] - coeff * xr[i]) * inv;
        if (accumulate) v += o[i];
        if (clamp > 0.f) v = fminf(fmaxf(v, -clamp), clamp);
        o[i] = v;
        if (dx_h) dx_h[(size_t)row * dim + i] = __float2half_rn(v * h_scale);
    }
}

// The same sums in the same order for rows of up to 256 NV elements, a block per row: a thread's elements stay in registers, so that all of a row's
// loads are in flight at once and nothing is read twice. 512 rows of 2560: 8.6 us and, backward, 12.1 where the row was read again after the sums;
// 7.3 and 9.9 here.
template <int NV>
__global__ void __launch_bounds__(256)
rms_norm_held_kernel(const float *x, const float *gamma, float *out, __half *out_h, int dim, float eps)
{
    __shared__ float sh[8];
    const size_t at = (size_t)blockIdx.x * dim;
    float v[NV], ss = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = threadIdx.x + 256 * k;
        v[k] = i < dim ? x[at + i] : 0.f;
    }
#pragma unroll
    for (int k = 0; k < NV; ++k)
        if (threadIdx.x + 256 * k < dim) ss = fmaf(v[k], v[k], ss);
    ss = group_sum_f<256>(ss, sh);
    const float inv = rsqrtf(ss / (float)dim + eps);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = threadIdx.x + 256 * k;
        if (i < dim) {
            const float r = v[k] * inv * gamma[i];
            out[at + i] = r;
            if (out_h) out_h[at + i] = __float2half_rn(r);
        }
    }
}

template <int NV>
__global__ void __launch_bounds__(256)
rms_norm_bwd_held_kernel(const float *x, const float *dy, long long dy_ld, const float *gamma, float *dx, int dim, float eps, int accumulate,
                         float clamp, __half *dx_h, float h_scale)
{
    __shared__ float sh[8];
    const size_t at = (size_t)blockIdx.x * dim;
    const float *dr = dy + (size_t)blockIdx.x * dy_ld;
    float v[NV], d[NV], g[NV], ss = 0.f, dot = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = threadIdx.x + 256 * k;
        v[k] = i < dim ? x[at + i] : 0.f;
        d[k] = i < dim ? dr[i] : 0.f;
        g[k] = i < dim ? gamma[i] : 0.f;
    }
#pragma unroll
    for (int k = 0; k < NV; ++k)
        if (threadIdx.x + 256 * k < dim) {
            ss = fmaf(v[k], v[k], ss);
            dot = fmaf(d[k] * g[k], v[k], dot);
        }
    ss = group_sum_f<256>(ss, sh);
    dot = group_sum_f<256>(dot, sh);
    const float inv = rsqrtf(ss / (float)dim + eps);
    const float coeff = dot * inv * inv / (float)dim;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = threadIdx.x + 256 * k;
        if (i < dim) {
            float r = __fmaf_rn(g[k], d[k], -__fmul_rn(coeff, v[k])) * inv;      // as the element form contracts it
            if (accumulate) r += dx[at + i];
            if (clamp > 0.f) r = fminf(fmaxf(r, -clamp), clamp);
            dx[at + i] = r;
            if (dx_h) dx_h[at + i] = __float2half_rn(r * h_scale);
        }
    }
}

// ---- QK-norm + RoPE: one warp per (row, head) -----------------------------------------------
// Heads 0..n_q-1 are q heads, n_q..n_q+n_kv-1 the k heads; both sit in qkv at column head*hd.
template <int HD>
__global__ void qk_norm_rope_kernel(const float *qkv, long long ld, const float *qg, const float *kg,
                                    const float *inv_freq, int rows, int seq_len, int n_q, int n_kv, float eps,
                                    float *q_out, float *k_out)
{
    constexpr int PER = HD / 64;                       // rotation pairs per lane
    const int unit = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int nh = n_q + n_kv;
    if (unit >= rows * nh) return;
    const int row = unit / nh, h = unit % nh, l = threadIdx.x & 31;
    const float *src = qkv + (size_t)row * ld + (size_t)h * HD;
    const float *g = h < n_q ? qg : kg;
    float *dst = h < n_q ? q_out + ((size_t)row * n_q + h) * HD : k_out + ((size_t)row * n_kv + (h - n_q)) * HD;
    float a[PER], b[PER];
    float ss = 0.f;
#pragma unroll
    for (int c = 0; c < PER; ++c) {
        a[c] = src[l + 32 * c];
        b[c] = src[l + 32 * c + HD / 2];
        ss = fmaf(a[c], a[c], ss);
        ss = fmaf(b[c], b[c], ss);
    }
    ss = warp_sum(ss);
    const float inv = rsqrtf(ss / (float)HD + eps);
    const float pos = (float)(row % seq_len);
#pragma unroll
    for (int c = 0; c < PER; ++c) {
        const int d = l + 32 * c;
        const float x0 = a[c] * inv * g[d], x1 = b[c] * inv * g[d + HD / 2];
        float sn, cs;
        sincosf(pos * inv_freq[d], &sn, &cs);
        dst[d] = x0 * cs - x1 * sn;
        dst[d + HD / 2] = x0 * sn + x1 * cs;
    }
}

template <int HD>
__global__ void qk_norm_rope_bwd_kernel(float *dqkv, const float *qkv, long long ld, long long dld, const float *qg, const float *kg,
                                        const float *inv_freq, int rows, int seq_len, int n_q, int n_kv, float eps)
{
    constexpr int PER = HD / 64;
    const int unit = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int nh = n_q + n_kv;
    if (unit >= rows * nh) return;
    const int row = unit / nh, h = unit % nh, l = threadIdx.x & 31;
    const float *x = qkv + (size_t)row * ld + (size_t)h * HD;
    float *d = dqkv + (size_t)row * dld + (size_t)h * HD;
    const float *g = h < n_q ? qg : kg;
    const float pos = (float)(row % seq_len);
    float xa[PER], xb[PER], ga[PER], gb[PER];
    float ss = 0.f, dot = 0.f;
#pragma unroll
    for (int c = 0; c < PER; ++c) {
        const int i = l + 32 * c;
        float sn, cs;
        sincosf(pos * inv_freq[i], &sn, &cs);
        const float y0 = d[i], y1 = d[i + HD / 2];
        ga[c] = y0 * cs + y1 * sn;                     // rotation by -angle
        gb[c] = -y0 * sn + y1 * cs;
        xa[c] = x[i];
        xb[c] = x[i + HD / 2];
        ss = fmaf(xa[c], xa[c], ss);
        ss = fmaf(xb[c], xb[c], ss);
        dot = fmaf(ga[c] * g[i], xa[c], dot);
        dot = fmaf(gb[c] * g[i + HD / 2], xb[c], dot);
    }
    ss = warp_sum(ss);
    dot = warp_sum(dot);
    const float inv = rsqrtf(ss / (float)HD + eps);
    const float coeff = dot * inv * inv / (float)HD;
#pragma unroll
    for (int c = 0; c < PER; ++c) {
        const int i = l + 32 * c;
        d[i] = (g[i] * ga[c] - coeff * xa[c]) * inv;
        d[i + HD / 2] = (g[i + HD / 2] * gb[c] - coeff * xb[c]) * inv;
    }
}

// ---- causal attention, training form ---------------------------------------------------------------
// One block per (sequence, head, 64 queries), or 64 keys, walking the tiles it can see; fp32 values throughout. The products have two forms with
// the same layout over the lanes: fp32 multiply-adds on the CUDA cores, and the tensor cores (mma.sync m16n8k8), where an fp32
// operand is a TF32 number plus what that leaves (x = hi + lo, 22 bits) and a product is hi hi + hi lo + lo hi. The fragments of both
// operands are read from plain row-major tiles, in any orientation, with the split on the way; 16-bit planes would need every
// row's range. Scores and probabilities go to the matrices that are kept anyway and are read back by the thread that wrote them.
// The next tile's copies run under the current one's products. The longest rows start first.
// A layer forward and backward, 32 heads, 509 positions of 128: 515 us on the tensor cores, 718 us on the CUDA cores, one warp per query
// or key 2.2 ms. Bound by instructions (the split of every operand element; shared-memory reads of the fp32 form) and by the single-word
// accesses to the score matrix. Off float64 2e-7 .. 4e-7 as fp32 and no more on the tensor cores.
constexpr int AT = 64;                       // tile edge: queries and keys
constexpr int ATT_THREADS = 256;

__device__ __forceinline__ void tf32_parts(float x, uint32_t &hi, uint32_t &lo)
{
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
    lo = __float_as_uint(x - __uint_as_float(hi));
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// acc += A (16 x K) . B (K x 8 NT) of a warp: a(m, k) at A[m * am + k * ak], b(k, n) at B[k * bk + n * bn]. Lane l holds rows l / 4 and
// l / 4 + 8, columns 2 (l % 4) and the next of every eight. K: a multiple of 32.
// Tensor cores truncate what they add to an accumulator, 1.4e-8 of it a time: the corrections have one of their own, and the sums of 32 of k
// start from zero and join acc in fp32 adds.
template <int NT>
__device__ __forceinline__ void mma_add(float (&acc)[NT][4], const float *A, int am, int ak, const float *B, int bk, int bn, int K)
{
    const int r = (threadIdx.x & 31) >> 2, q = threadIdx.x & 3;
    float low[NT][4] = {};
#pragma unroll 1
    for (int k0 = 0; k0 < K; k0 += 32) {
        float t[NT][4] = {};
#pragma unroll 2
        for (int k = k0; k < k0 + 32; k += 8) {
            uint32_t ah[4], al[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) tf32_parts(A[(r + 8 * (e & 1)) * am + (k + q + 4 * (e >> 1)) * ak], ah[e], al[e]);
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                uint32_t h0, l0, h1, l1;
                tf32_parts(B[(k + q) * bk + (n * 8 + r) * bn], h0, l0);
                tf32_parts(B[(k + q + 4) * bk + (n * 8 + r) * bn], h1, l1);
                mma_tf32(low[n], al, h0, h1);
                mma_tf32(low[n], ah, l0, l1);
                mma_tf32(t[n], ah, h0, h1);
            }
        }
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[n][e] += t[n][e];
    }
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[n][e] += low[n][e];
}

// The same sums as fp32 multiply-adds in order of k, for operands whose k are contiguous (b(k, n) at B[n * bn + k]).
template <int NT>
__device__ __forceinline__ void fma_add(float (&acc)[NT][4], const float *A, int am, const float *B, int bn, int K)
{
    const int r = (threadIdx.x & 31) >> 2, q = threadIdx.x & 3;
#pragma unroll 2
    for (int k = 0; k < K; k += 4) {
        const float4 a0 = *reinterpret_cast<const float4 *>(A + r * am + k), a1 = *reinterpret_cast<const float4 *>(A + (r + 8) * am + k);
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float4 b = *reinterpret_cast<const float4 *>(B + (n * 8 + 2 * q + e) * bn + k);
                acc[n][e] = fmaf(a0.w, b.w, fmaf(a0.z, b.z, fmaf(a0.y, b.y, fmaf(a0.x, b.x, acc[n][e]))));
                acc[n][2 + e] = fmaf(a1.w, b.w, fmaf(a1.z, b.z, fmaf(a1.y, b.y, fmaf(a1.x, b.x, acc[n][2 + e]))));
            }
    }
}

// Whether any lane holds an infinity or NaN.
template <int NT>
__device__ __forceinline__ bool any_not_finite(const float (&t)[NT][4])
{
    float z = 0.f;
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) z = fmaf(t[n][e], 0.f, z);
    return __any_sync(0xffffffffu, z != z);
}

// Scores of 16 x 8 NT: rows of A times rows of B, HD long. TC: tensor cores; sums that come out infinite or NaN are formed again as
// fp32 sums, because the parts of an infinity are an infinity and a NaN.
template <bool TC, int NT>
__device__ __forceinline__ void score_tile(float (&acc)[NT][4], const float *A, int am, const float *B, int bn, int K)
{
    if (TC) {
        mma_add<NT>(acc, A, am, 1, B, 1, bn, K);
        if (!any_not_finite(acc)) return;
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[n][e] = 0.f;
    }
    fma_add<NT>(acc, A, am, B, bn, K);
}

// acc += weights (16 x 64) . rows (64 x 8 NT), row r + 8 a of the fragment over k in [from[a], to[a]), beyond which its weights are zero.
// Four columns of eight at a time in sums of their own that join acc in fp32 adds: tensor cores truncate when they
// accumulate, which over all tiles of a long row would add up (7e-6 of dK at 509 positions, 1e-6 so). fp32 sums leave the other k
// out, and so do those of the tensor cores when they come out infinite or NaN: zero times a later row's infinity is NaN.
template <bool TC, int NT>
__device__ __forceinline__ void weighted_rows(float (&acc)[NT][4], const float *A, int am, int ak, const float *B, int bk, const int (&from)[2],
                                              const int (&to)[2])
{
    const int r = (threadIdx.x & 31) >> 2, q = threadIdx.x & 3;
#pragma unroll
    for (int g = 0; g < NT; g += 4) {
        float t[4][4] = {};
        if (TC) mma_add<4>(t, A, am, ak, B + g * 8, bk, 1, AT);
        if (!TC || any_not_finite(t)) {
            if (TC) {
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) t[n][e] = 0.f;
            }
#pragma unroll 4
            for (int k = min(from[0], from[1]); k < max(to[0], to[1]); ++k) {
                const float w0 = A[r * am + k * ak], w1 = A[(r + 8) * am + k * ak];
                const bool on0 = k >= from[0] && k < to[0], on1 = k >= from[1] && k < to[1];
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    const float2 b = *reinterpret_cast<const float2 *>(B + k * bk + (g + n) * 8 + 2 * q);
                    if (on0) { t[n][0] = fmaf(w0, b.x, t[n][0]); t[n][1] = fmaf(w0, b.y, t[n][1]); }
                    if (on1) { t[n][2] = fmaf(w1, b.x, t[n][2]); t[n][3] = fmaf(w1, b.y, t[n][3]); }
                }
            }
        }
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[g + n][e] += t[n][e];
    }
}

// Asynchronous copy of n rows (zeros up to 64) of COLS floats, `ld` apart, to rows `pitch` apart; 16 bytes at a time where addresses allow.
template <int COLS>
__device__ __forceinline__ void tile_copy(float *dst, int pitch, const float *src, long long ld, int n, int cols = COLS)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if (((reinterpret_cast<uintptr_t>(src) & 15) | (ld & 3) | (cols & 3)) == 0) {
        for (int e = threadIdx.x; e < AT * (COLS / 4); e += ATT_THREADS) {
            const int i = e / (COLS / 4), c = e % (COLS / 4) * 4;
            const int on = i < n && c < cols ? 16 : 0;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d + (i * pitch + c) * 4), "l"(on ? src + i * ld + c : src), "r"(on) : "memory");
        }
    } else {
        for (int e = threadIdx.x; e < AT * COLS; e += ATT_THREADS) {
            const int i = e / COLS, c = e % COLS;
            const int on = i < n && c < cols ? 4 : 0;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + (i * pitch + c) * 4), "l"(on ? src + i * ld + c : src), "r"(on) : "memory");
        }
    }
}
__device__ __forceinline__ void tile_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void tile_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Pitches that keep fragment reads off each other's banks: along a row (k contiguous) 4 mod 32, down a column 8 mod 32.
template <int HD> struct AttnTiles {
    static constexpr int RP = HD + 4, CP = HD + 8, PP = AT + 4, BUF = AT * CP;
    static constexpr size_t bytes = ((size_t)AT * RP + 2 * BUF) * sizeof(float);      // one operand, two buffers; the weights replace the operand
};

// Sums and maxima of a row lie in four lanes of two warps (column halves).
__device__ __forceinline__ float quad_sum(float v)
{
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// Which tile (0: the heaviest), sequence and head the block works on. Tiles weigh 1 .. N / 64.
struct AttnItem { int tile, seq, head; };
template <int PER_SM>
__device__ __forceinline__ AttnItem attn_item(int n_seq, int heads)
{
    const int rank = rank_by_weight(PER_SM > 1);
    return {rank / (n_seq * heads), rank % n_seq, rank / n_seq % heads};
}

template <int HD, bool TC>
__global__ void __launch_bounds__(ATT_THREADS)
attn_fwd_kernel(const float *q, const float *k, const float *v, long long v_ld, int n_seq, int N, int n_q, int n_kv,
                float scale, float *probs, float *out, __half *out_h)
{
    using L = AttnTiles<HD>;
    extern __shared__ __align__(16) float sh[];
    __shared__ float stat[2][2][AT];
    float *Q = sh, *P = sh, *buf = sh + AT * L::RP;
    const AttnItem item = attn_item<HD == 256 ? 1 : 2>(n_seq, n_q);
    const int it = (N + AT - 1) / AT - 1 - item.tile, s = item.seq, h = item.head, kvh = h / (n_q / n_kv);
    const size_t row0 = (size_t)s * N;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rw = (warp & 3) * 16, half = warp >> 2;
    const int i0 = it * AT, ni = min(AT, N - i0), r0 = rw + (lane >> 2), c0 = half * 32 + 2 * (lane & 3);
    const float *kh = k + (row0 * n_kv + kvh) * HD, *vh = v + row0 * v_ld + (size_t)kvh * HD;
    float *pr = probs + (((size_t)s * n_q + h) * N + i0) * N;

    tile_copy<HD>(Q, L::RP, q + ((row0 + i0) * n_q + h) * HD, (long long)n_q * HD, ni);
    tile_copy<HD>(buf, L::RP, kh, (long long)n_kv * HD, min(AT, N));
    tile_commit();
    float mx[2] = {-1e30f, -1e30f}, l[2] = {0.f, 0.f};
    for (int jt = 0; jt <= it; ++jt) {
        const int j0 = jt * AT;
        if (jt < it) {
            tile_copy<HD>(buf + ((jt + 1) & 1) * L::BUF, L::RP, kh + (size_t)(j0 + AT) * n_kv * HD, (long long)n_kv * HD, min(AT, N - j0 - AT));
            tile_commit();
            tile_wait<1>();
        } else tile_wait<0>();
        __syncthreads();
        float acc[4][4] = {};
        score_tile<TC>(acc, Q + rw * L::RP, L::RP, buf + (jt & 1) * L::BUF + half * 32 * L::RP, L::RP, HD);
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            const int i = r0 + 8 * a;
            float m = mx[a];
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const int j = j0 + c0 + 8 * n + b;
                    float &x = acc[n][2 * a + b];
                    x *= scale;
                    if (i < ni && j <= i0 + i) { m = fmaxf(m, x); pr[(size_t)i * N + j] = x; }
                }
            float sum = 0.f;
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int b = 0; b < 2; ++b)
                    if (i < ni && j0 + c0 + 8 * n + b <= i0 + i) sum += expf(acc[n][2 * a + b] - m);
            l[a] = l[a] * expf(mx[a] - m) + sum;
            mx[a] = m;
        }
        __syncthreads();
    }
    tile_copy<HD>(buf, L::CP, vh, v_ld, min(AT, N));
    tile_commit();
    float inv[2];
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        float m = fmaxf(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], 1));
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
        const float sum = quad_sum(l[a] * expf(mx[a] - m));
        mx[a] = m; l[a] = sum;
        if ((lane & 3) == 0) { stat[0][half][r0 + 8 * a] = m; stat[1][half][r0 + 8 * a] = sum; }
    }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        const int i = r0 + 8 * a;
        const float m0 = stat[0][0][i], m1 = stat[0][1][i], m = fmaxf(m0, m1);
        mx[a] = m;
        inv[a] = i < ni ? 1.0f / (stat[1][0][i] * expf(m0 - m) + stat[1][1][i] * expf(m1 - m)) : 0.f;
    }
    float o[HD / 16][4] = {};
    for (int jt = 0; jt <= it; ++jt) {
        const int j0 = jt * AT;
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const int i = r0 + 8 * a, c = c0 + 8 * n + b, j = j0 + c;
                    float p = 0.f;
                    if (i < ni && j < N) {
                        if (j <= i0 + i) p = expf(pr[(size_t)i * N + j] - mx[a]) * inv[a];
                        pr[(size_t)i * N + j] = p;
                    }
                    P[i * L::PP + c] = p;
                }
        if (jt < it) {
            tile_copy<HD>(buf + ((jt + 1) & 1) * L::BUF, L::CP, vh + (size_t)(j0 + AT) * v_ld, v_ld, min(AT, N - j0 - AT));
            tile_commit();
            tile_wait<1>();
        } else tile_wait<0>();
        __syncthreads();
        const int from[2] = {0, 0}, to[2] = {r0 < ni ? min(AT, i0 + r0 - j0 + 1) : 0, r0 + 8 < ni ? min(AT, i0 + r0 + 8 - j0 + 1) : 0};
        weighted_rows<TC>(o, P + rw * L::PP, L::PP, 1, buf + (jt & 1) * L::BUF + half * (HD / 2), L::CP, from, to);
        __syncthreads();
    }
    const int ahead = min((it + 1) * AT, N);                   // columns that no row of the tile sees
    for (int i = warp; i < ni; i += ATT_THREADS / 32)
        for (int j = ahead + lane; j < N; j += 32) pr[(size_t)i * N + j] = 0.f;
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        const int i = r0 + 8 * a;
        if (i >= ni) continue;
        const size_t base = ((row0 + i0 + i) * n_q + h) * HD + half * (HD / 2) + 2 * (lane & 3);
#pragma unroll
        for (int n = 0; n < HD / 16; ++n)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                if (out) out[base + 8 * n + b] = o[n][2 * a + b];
                if (out_h) out_h[base + 8 * n + b] = __float2half_rn(o[n][2 * a + b]);
            }
    }
}

// d_score = p * (dO . V - sum_j p_j (dO . V_j)) * scale, and dQ = d_score . K, for 64 queries of a head.
template <int HD, bool TC>
__global__ void __launch_bounds__(ATT_THREADS)
attn_bwd_dq_kernel(const float *d_out, const float *probs, const float *k, const float *v, long long v_ld, int n_seq, int N, int n_q,
                   int n_kv, float scale, float *d_score, float *dqkv, long long ld)
{
    using L = AttnTiles<HD>;
    extern __shared__ __align__(16) float sh[];
    __shared__ float stat[2][AT];
    float *O = sh, *G = sh, *buf = sh + AT * L::RP;
    const AttnItem item = attn_item<HD == 256 ? 1 : 2>(n_seq, n_q);
    const int it = (N + AT - 1) / AT - 1 - item.tile, s = item.seq, h = item.head, kvh = h / (n_q / n_kv);
    const size_t row0 = (size_t)s * N;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rw = (warp & 3) * 16, half = warp >> 2;
    const int i0 = it * AT, ni = min(AT, N - i0), r0 = rw + (lane >> 2), c0 = half * 32 + 2 * (lane & 3);
    const float *kh = k + (row0 * n_kv + kvh) * HD, *vh = v + row0 * v_ld + (size_t)kvh * HD;
    const size_t tile_rows = (((size_t)s * n_q + h) * N + i0) * N;
    const float *pr = probs + tile_rows;
    float *ds = d_score + tile_rows;

    tile_copy<HD>(O, L::RP, d_out + ((row0 + i0) * n_q + h) * HD, (long long)n_q * HD, ni);
    tile_copy<HD>(buf, L::RP, vh, v_ld, min(AT, N));
    tile_commit();
    float dp[2] = {0.f, 0.f};
    for (int jt = 0; jt <= it; ++jt) {
        const int j0 = jt * AT;
        if (jt < it) {
            tile_copy<HD>(buf + ((jt + 1) & 1) * L::BUF, L::RP, vh + (size_t)(j0 + AT) * v_ld, v_ld, min(AT, N - j0 - AT));
            tile_commit();
            tile_wait<1>();
        } else tile_wait<0>();
        __syncthreads();
        float acc[4][4] = {};
        score_tile<TC>(acc, O + rw * L::RP, L::RP, buf + (jt & 1) * L::BUF + half * 32 * L::RP, L::RP, HD);
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const int i = r0 + 8 * a, j = j0 + c0 + 8 * n + b;
                    if (i < ni && j <= i0 + i) {
                        ds[(size_t)i * N + j] = acc[n][2 * a + b];
                        dp[a] = fmaf(pr[(size_t)i * N + j], acc[n][2 * a + b], dp[a]);
                    }
                }
        __syncthreads();
    }
    tile_copy<HD>(buf, L::CP, kh, (long long)n_kv * HD, min(AT, N));
    tile_commit();
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        dp[a] = quad_sum(dp[a]);
        if ((lane & 3) == 0) stat[half][r0 + 8 * a] = dp[a];
    }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 2; ++a) dp[a] = stat[0][r0 + 8 * a] + stat[1][r0 + 8 * a];
    float o[HD / 16][4] = {};
    for (int jt = 0; jt <= it; ++jt) {
        const int j0 = jt * AT;
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const int i = r0 + 8 * a, c = c0 + 8 * n + b, j = j0 + c;
                    float g = 0.f;
                    if (i < ni && j < N) {
                        if (j <= i0 + i) g = pr[(size_t)i * N + j] * (ds[(size_t)i * N + j] - dp[a]) * scale;
                        ds[(size_t)i * N + j] = g;
                    }
                    G[i * L::PP + c] = g;
                }
        if (jt < it) {
            tile_copy<HD>(buf + ((jt + 1) & 1) * L::BUF, L::CP, kh + (size_t)(j0 + AT) * n_kv * HD, (long long)n_kv * HD, min(AT, N - j0 - AT));
            tile_commit();
            tile_wait<1>();
        } else tile_wait<0>();
        __syncthreads();
        const int from[2] = {0, 0}, to[2] = {r0 < ni ? min(AT, i0 + r0 - j0 + 1) : 0, r0 + 8 < ni ? min(AT, i0 + r0 + 8 - j0 + 1) : 0};
        weighted_rows<TC>(o, G + rw * L::PP, L::PP, 1, buf + (jt & 1) * L::BUF + half * (HD / 2), L::CP, from, to);
        __syncthreads();
    }
    const int ahead = min((it + 1) * AT, N);
    for (int i = warp; i < ni; i += ATT_THREADS / 32)
        for (int j = ahead + lane; j < N; j += 32) ds[(size_t)i * N + j] = 0.f;
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        const int i = r0 + 8 * a;
        if (i >= ni) continue;
        float *dst = dqkv + (row0 + i0 + i) * ld + (size_t)h * HD + half * (HD / 2) + 2 * (lane & 3);
#pragma unroll
        for (int n = 0; n < HD / 16; ++n) { dst[8 * n] = o[n][2 * a]; dst[8 * n + 1] = o[n][2 * a + 1]; }
    }
}

// 64 keys x 64 columns of dK (d_score^T . Q) or dV (P^T . dO) of a KV head: summed over the later queries of each query head, then
// over the heads in order. The item's head = ((kv head * 2 + dK / dV) * (HD / 64) + columns).
template <bool TC>
__global__ void __launch_bounds__(ATT_THREADS)
attn_bwd_dkv_kernel(const float *d_score, const float *probs, const float *q, const float *d_out, int n_seq, int N, int n_q, int n_kv,
                    int hd, float *dqkv, long long ld)
{
    constexpr int CP = AT + 8, BUF = AT * CP;
    extern __shared__ __align__(16) float sh[];               // two buffers of (weights, rows)
    const int slices = hd / 64;
    const AttnItem item = attn_item<2>(n_seq, n_kv * 2 * slices);
    const int jt = item.tile, s = item.seq, slice = item.head % slices;
    const int which = (item.head / slices) & 1, kvh = item.head / (2 * slices), group = n_q / n_kv;
    const size_t row0 = (size_t)s * N;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rw = (warp & 3) * 16, half = warp >> 2;
    const int j0 = jt * AT, nj = min(AT, N - j0), tiles = (N - j0 + AT - 1) / AT, steps = group * tiles;
    auto stage = [&](int t) {
        const int h = kvh * group + t / tiles, i0 = j0 + t % tiles * AT, ni = min(AT, N - i0);
        float *w = sh + (t & 1) * 2 * BUF;
        tile_copy<AT>(w, CP, (which ? probs : d_score) + ((size_t)s * n_q + h) * N * N + (size_t)i0 * N + j0, N, ni, nj);
        tile_copy<AT>(w + BUF, CP, (which ? d_out : q) + ((row0 + i0) * n_q + h) * hd + slice * 64, (long long)n_q * hd, ni);
        tile_commit();
    };
    stage(0);
    float sum[4][4] = {};
    for (int t = 0; t < steps; ++t) {
        if (t + 1 < steps) { stage(t + 1); tile_wait<1>(); }
        else tile_wait<0>();
        __syncthreads();
        const float *w = sh + (t & 1) * 2 * BUF;
        const int i0 = j0 + t % tiles * AT, ni = min(AT, N - i0), first = j0 + rw + (lane >> 2) - i0;
        const int from[2] = {max(0, first), max(0, first + 8)}, to[2] = {ni, ni};
        weighted_rows<TC>(sum, w + rw, 1, CP, w + BUF + half * 32, CP, from, to);
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        const int j = rw + (lane >> 2) + 8 * a;
        if (j >= nj) continue;
        float *dst = dqkv + (row0 + j0 + j) * ld + (size_t)(n_q + (which ? n_kv : 0) + kvh) * hd + slice * 64 + half * 32 + 2 * (lane & 3);
#pragma unroll
        for (int n = 0; n < 4; ++n) { dst[8 * n] = sum[n][2 * a]; dst[8 * n + 1] = sum[n][2 * a + 1]; }
    }
}

// ---- SwiGLU ------------------------------------------------------------------------------------
struct Silu {
    static __device__ __forceinline__ float value(float g, float u) { return g / (1.0f + expf(-g)) * u; }
    static __device__ __forceinline__ void slopes(float g, float u, float dy, float &dg, float &du)
    {
        const float sig = 1.0f / (1.0f + expf(-g));
        dg = dy * u * (sig * (1.0f + g * (1.0f - sig)));
        du = dy * (g * sig);
    }
};
struct Gelu {
    static __device__ __forceinline__ float value(float g, float u)
    {
        float inner = 0.7978845608f * (g + 0.044715f * (g * g * g));
        inner = fminf(fmaxf(inner, -15.0f), 15.0f);
        return 0.5f * g * (1.0f + tanhf(inner)) * u;
    }
    static __device__ __forceinline__ void slopes(float g, float u, float dy, float &dg, float &du)
    {
        float inner = 0.7978845608f * (g + 0.044715f * (g * g * g));
        inner = fminf(fmaxf(inner, -15.0f), 15.0f);
        const float th = tanhf(inner);
        const float gelu_g = 0.5f * g * (1.0f + th);
        const float sech2 = 1.0f - th * th;
        const float grad = 0.5f * (1.0f + th) + 0.5f * g * sech2 * 0.7978845608f * (1.0f + 3.0f * 0.044715f * g * g);
        dg = dy * u * grad;
        du = dy * gelu_g;
    }
};
__global__ void silu_mul_rows_kernel(const float *gu, int inter, float *act, __half *act_h, size_t total)
{
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const size_t m = e / inter, i = e % inter;
        const float g = gu[m * 2 * inter + i], u = gu[m * 2 * inter + inter + i];
        const float v = Silu::value(g, u);
        if (act) act[e] = v;
        if (act_h) act_h[e] = __float2half_rn(v);
    }
}

__global__ void silu_mul_bwd_rows_kernel(const float *d_act, const float *gu, int inter, float *d_gu, __half *d_gu_h,
                                         float h_scale, size_t total)
{
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const size_t m = e / inter, i = e % inter;
        const float g = gu[m * 2 * inter + i], u = gu[m * 2 * inter + inter + i], dy = d_act[e];
        float dg, du;
        Silu::slopes(g, u, dy, dg, du);
        if (d_gu) { d_gu[m * 2 * inter + i] = dg; d_gu[m * 2 * inter + inter + i] = du; }
        if (d_gu_h) {
            d_gu_h[m * 2 * inter + i] = __float2half_rn(dg * h_scale);
            d_gu_h[m * 2 * inter + inter + i] = __float2half_rn(du * h_scale);
        }
    }
}

// GeGLU (Gemma3): gelu_mul / gelu_mul_backward, shaders/q8_kernels.metal:351-363, 561-580 -- the tanh form with
// its argument clamped to +-15, on the fused [rows, 2 * inter] gate|up layout.
__global__ void gelu_mul_rows_kernel(const float *gu, int inter, float *act, size_t total)
{
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const size_t m = e / inter, i = e % inter;
        const float g = gu[m * 2 * inter + i], u = gu[m * 2 * inter + inter + i];
        act[e] = Gelu::value(g, u);
    }
}

__global__ void gelu_mul_bwd_rows_kernel(const float *d_act, const float *gu, int inter, float *d_gu, size_t total)
{
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const size_t m = e / inter, i = e % inter;
        const float g = gu[m * 2 * inter + i], u = gu[m * 2 * inter + inter + i], dy = d_act[e];
        Gelu::slopes(g, u, dy, d_gu[m * 2 * inter + i], d_gu[m * 2 * inter + inter + i]);
    }
}

// out = a + b (residual_add :369-375 with its result in a third buffer)
__global__ void add_kernel(const float *a, const float *b, float *out, size_t n)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) out[i] = a[i] + b[i];
}

// The gated activations in whole aligned quads, rows over blockIdx.y: no division, 16 bytes an access. The element forms above divide twice in 64
// bits for every element: 512 x 9728 19 us (backward 21.4), 9.4 and 11.8 here.
__device__ __forceinline__ void put_quad(float *at, const float (&v)[4]) { *reinterpret_cast<float4 *>(at) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void put_quad(__half *at, const float (&v)[4], float scale)
{
    const __half2 a = __halves2half2(__float2half_rn(v[0] * scale), __float2half_rn(v[1] * scale));
    const __half2 b = __halves2half2(__float2half_rn(v[2] * scale), __float2half_rn(v[3] * scale));
    *reinterpret_cast<uint2 *>(at) = make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
}
template <typename F>
__global__ void __launch_bounds__(256) glu_quads_kernel(const float *gu, int inter, float *act, __half *act_h)
{
    const int i = 4 * (blockIdx.x * 256 + threadIdx.x);
    if (i >= inter) return;
    const size_t m = blockIdx.y;
    const float4 g = *reinterpret_cast<const float4 *>(gu + m * 2 * inter + i), u = *reinterpret_cast<const float4 *>(gu + m * 2 * inter + inter + i);
    const float v[4] = {F::value(g.x, u.x), F::value(g.y, u.y), F::value(g.z, u.z), F::value(g.w, u.w)};
    if (act) put_quad(act + m * inter + i, v);
    if (act_h) put_quad(act_h + m * inter + i, v, 1.0f);
}
template <typename F>
__global__ void __launch_bounds__(256) glu_bwd_quads_kernel(const float *d_act, const float *gu, int inter, float *d_gu, __half *d_gu_h, float h_scale)
{
    const int i = 4 * (blockIdx.x * 256 + threadIdx.x);
    if (i >= inter) return;
    const size_t m = blockIdx.y, at = m * 2 * inter + i;
    const float4 g = *reinterpret_cast<const float4 *>(gu + at), u = *reinterpret_cast<const float4 *>(gu + at + inter);
    const float4 dy = *reinterpret_cast<const float4 *>(d_act + m * inter + i);
    float dg[4], du[4];
    F::slopes(g.x, u.x, dy.x, dg[0], du[0]);
    F::slopes(g.y, u.y, dy.y, dg[1], du[1]);
    F::slopes(g.z, u.z, dy.z, dg[2], du[2]);
    F::slopes(g.w, u.w, dy.w, dg[3], du[3]);
    if (d_gu) { put_quad(d_gu + at, dg); put_quad(d_gu + at + inter, du); }
    if (d_gu_h) { put_quad(d_gu_h + at, dg, h_scale); put_quad(d_gu_h + at + inter, du, h_scale); }
}

// ---- LoRA up-projection added into the base projection -------------------------------------------
// One thread per output column keeps its row of B in registers and walks LORA_ROWS token rows whose
// mid vectors sit in shared memory.
constexpr int LORA_ROWS = 8;
template <int MAXR>
__global__ void __launch_bounds__(256)
lora_add_kernel(float *y, long long ld, int col0, int n_cols, const float *mid, long long mid_ld, const float *B,
                int rank, float sc, int rows)
{
    __shared__ float ms[LORA_ROWS][MAXR];
    const int m0 = blockIdx.y * LORA_ROWS;
    for (int e = threadIdx.x; e < LORA_ROWS * MAXR; e += blockDim.x) {
        const int i = e / MAXR, r = e % MAXR;
        ms[i][r] = (r < rank && m0 + i < rows) ? mid[(size_t)(m0 + i) * mid_ld + r] : 0.f;   // zero beyond the rank
    }
    __syncthreads();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n_cols) return;
    float b[MAXR], v[LORA_ROWS];
    float *at = y + (size_t)m0 * ld + col0 + c;
#pragma unroll
    for (int i = 0; i < LORA_ROWS; ++i) v[i] = m0 + i < rows ? at[i * ld] : 0.f;              // in flight under the row of B
    if (rank == MAXR && (reinterpret_cast<uintptr_t>(B) & 15) == 0) {
#pragma unroll
        for (int r = 0; r < MAXR; r += 4) *reinterpret_cast<float4 *>(b + r) = *reinterpret_cast<const float4 *>(B + (size_t)c * MAXR + r);
    } else {
#pragma unroll
        for (int r = 0; r < MAXR; ++r) b[r] = r < rank ? B[(size_t)c * rank + r] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < LORA_ROWS; ++i) {
        if (m0 + i >= rows) break;
        float acc = 0.f;
#pragma unroll
        for (int r = 0; r < MAXR; ++r) acc = fmaf(ms[i][r], b[r], acc);
        at[i * ld] = v[i] + sc * acc;
    }
}

// Refreshes the LoRA rows appended to the fused q/k/v weight and to its transposed copy.
//   w_ext  [qkv + xr, d]: rows qkv..qkv+R = A_q, rows qkv+R..qkv+2R = A_v
//   wt_ext [d + xr, qkv]: row d+r = sc * B_q[:, r] over the q columns, row d+R+r = sc * B_v[:, r] over the
//                         v columns, zero elsewhere
// so that the forward product also yields ln1 A^T and the backward product also yields sc * dq B_q and
// sc * dv B_v (src/nn/fast_sft.c:639-641, 948-949, 963-964) at no extra pass over the activations.
__device__ __forceinline__ void store_as(float *p, float v) { *p = v; }
__device__ __forceinline__ void store_as(__half *p, float v) { *p = __float2half_rn(v); }

template <typename T>
__global__ void lora_pack_kernel(T *w_ext, T *wt_ext, const float *A_q, const float *B_q, const float *A_v,
                                 const float *B_v, int d, int q_cols, int kv_cols, int rank, int xr, float sc)
{
    const int qkv = q_cols + 2 * kv_cols;
    const int row = blockIdx.y;                                    // 0 .. xr-1
    const int width = d > qkv ? d : qkv;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < width; c += gridDim.x * blockDim.x) {
        if (c < d) {
            float v = 0.f;
            if (row < rank) v = A_q[(size_t)row * d + c];
            else if (row < 2 * rank) v = A_v[(size_t)(row - rank) * d + c];
            store_as(w_ext + (size_t)(qkv + row) * d + c, v);
        }
        if (c < qkv) {
            float v = 0.f;
            if (row < rank) { if (c < q_cols) v = sc * B_q[(size_t)c * rank + row]; }
            else if (row < 2 * rank) { if (c >= q_cols + kv_cols) v = sc * B_v[(size_t)(c - q_cols - kv_cols) * rank + (row - rank)]; }
            store_as(wt_ext + (size_t)(d + row) * qkv + c, v);
        }
    }
}

// ---- rank-R LoRA gradients: C(p, r) = alpha * sum_m X[m, p] * Y[m, r], X wide, Y narrow (R <= MAXR) ------
// float_matmul_tn of the reference (shaders/q8_kernels.metal:1070-1094) for dB = sc * dY^T mid and
// dA = tmp^T ln1 (src/nn/fast_sft.c:946-950, 961-965). A block owns 16 columns p; its sixteen thread groups
// take every sixteenth row m and are summed in group order through shared memory, so the result does not
// depend on scheduling. A thread keeps its R sums in registers; the rows of Y are staged in shared memory
// 4096/MAXR at a time and read as broadcasts; four X loads are in flight per thread.
template <int MAXR>
__global__ void __launch_bounds__(256)
xty_skinny_kernel(const float *X, long long ld_x, const float *Y, long long ld_y, int rows, int P, int R, float alpha,
                  float *C, long long c_p, long long c_r)
{
    constexpr int CH = 4096 / MAXR;                      // rows of Y per shared-memory chunk
    constexpr int PW = 16, NG = 16;                      // columns per block, row groups per block
    static_assert(MAXR <= 16, "the cross-group buffer is sized for MAXR <= 16");
    __shared__ float ys[CH * MAXR];
    __shared__ float red[(NG - 1) * PW * (MAXR + 1)];
    const int pl = threadIdx.x % PW, mg = threadIdx.x / PW;
    const int p = blockIdx.x * PW + pl;
    const bool on = p < P;
    float acc[MAXR];
#pragma unroll
    for (int r = 0; r < MAXR; ++r) acc[r] = 0.f;
    for (int c0 = 0; c0 < rows; c0 += CH) {
        const int cn = min(CH, rows - c0);
        __syncthreads();
        for (int e = threadIdx.x; e < cn * MAXR; e += 256) {
            const int m = e / MAXR, r = e % MAXR;
            ys[e] = r < R ? Y[(size_t)(c0 + m) * ld_y + r] : 0.f;
        }
        __syncthreads();
        if (on) {
            int m = mg;
            for (; m + 3 * NG < cn; m += 4 * NG) {       // four rows of this group in flight
                const float x0 = X[(size_t)(c0 + m) * ld_x + p], x1 = X[(size_t)(c0 + m + NG) * ld_x + p];
                const float x2 = X[(size_t)(c0 + m + 2 * NG) * ld_x + p], x3 = X[(size_t)(c0 + m + 3 * NG) * ld_x + p];
#pragma unroll
                for (int r = 0; r < MAXR; ++r) {
                    acc[r] = fmaf(x0, ys[m * MAXR + r], acc[r]);
                    acc[r] = fmaf(x1, ys[(m + NG) * MAXR + r], acc[r]);
                    acc[r] = fmaf(x2, ys[(m + 2 * NG) * MAXR + r], acc[r]);
                    acc[r] = fmaf(x3, ys[(m + 3 * NG) * MAXR + r], acc[r]);
                }
            }
            for (; m < cn; m += NG) {
                const float x0 = X[(size_t)(c0 + m) * ld_x + p];
#pragma unroll
                for (int r = 0; r < MAXR; ++r) acc[r] = fmaf(x0, ys[m * MAXR + r], acc[r]);
            }
        }
    }
    if (mg > 0) {
#pragma unroll
        for (int r = 0; r < MAXR; ++r) red[((mg - 1) * PW + pl) * (MAXR + 1) + r] = acc[r];
    }
    __syncthreads();
    if (mg == 0 && on) {
#pragma unroll
        for (int r = 0; r < MAXR; ++r) {
            if (r < R) {
                float v = acc[r];
#pragma unroll
                for (int g = 0; g < NG - 1; ++g) v += red[(g * PW + pl) * (MAXR + 1) + r];
                C[(size_t)p * c_p + (size_t)r * c_r] = alpha * v;
            }
        }
    }
}

// ---- softmax cross-entropy: one block per row ----------------------------------------------------
// Two passes over the row instead of the reference's three: the first keeps a running (max, sum of
// exponentials) per thread (merged across the block in a fixed order), the second writes the gradient.
// Rows are read four values at a time when the vocabulary allows it.
__device__ __forceinline__ void lse_add(float &m, float &s, float v)
{
    if (v > m) { s = s * expf(m - v) + 1.0f; m = v; }
    else s += expf(v - m);
}

__global__ void __launch_bounds__(1024)
softmax_ce_rows_kernel(const float *logits, const uint32_t *targets, int vocab, float grad_scale, float *losses,
                       float *dlogits, __half *dlogits_h, float h_scale)
{
    __shared__ float sh_m[32], sh_s[32];
    const size_t off = (size_t)blockIdx.x * vocab;
    const float *lr = logits + off;
    uint32_t tgt = targets[blockIdx.x];
    if (tgt >= (uint32_t)vocab) tgt = 0;
    const bool vec = (vocab & 3) == 0 && ((reinterpret_cast<uintptr_t>(logits) | reinterpret_cast<uintptr_t>(dlogits)) & 15) == 0 &&
                     (reinterpret_cast<uintptr_t>(dlogits_h) & 7) == 0;
    float m = -1e30f, sum = 0.f;
    if (vec) {
        const float4 *lr4 = reinterpret_cast<const float4 *>(lr);
        for (int i = threadIdx.x; i < vocab / 4; i += blockDim.x) {
            const float4 v = lr4[i];
            lse_add(m, sum, v.x); lse_add(m, sum, v.y); lse_add(m, sum, v.z); lse_add(m, sum, v.w);
        }
    } else {
        for (int i = threadIdx.x; i < vocab; i += blockDim.x) lse_add(m, sum, lr[i]);
    }
    // merge (max, sum) pairs: lanes of a warp by shuffles, warps through shared memory in warp order
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float mo = __shfl_xor_sync(0xffffffffu, m, o), so = __shfl_xor_sync(0xffffffffu, sum, o);
        const float mn = fmaxf(m, mo);
        sum = sum * expf(m - mn) + so * expf(mo - mn);
        m = mn;
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
    if (l == 0) { sh_m[w] = m; sh_s[w] = sum; }
    __syncthreads();
    float M = sh_m[0];
    for (int i = 1; i < nw; ++i) M = fmaxf(M, sh_m[i]);
    float S = 0.f;
    for (int i = 0; i < nw; ++i) S += sh_s[i] * expf(sh_m[i] - M);
    const float lse = logf(S) + M;
    if (threadIdx.x == 0) losses[blockIdx.x] = lse - lr[tgt];
    float *dr = dlogits + off;
    if (vec) {
        const float4 *lr4 = reinterpret_cast<const float4 *>(lr);
        for (int i = threadIdx.x; i < vocab / 4; i += blockDim.x) {
            const float4 v = lr4[i];
            float d[4] = {expf(v.x - lse), expf(v.y - lse), expf(v.z - lse), expf(v.w - lse)};
            if ((uint32_t)i == tgt / 4) d[tgt & 3] -= 1.0f;
#pragma unroll
            for (int c = 0; c < 4; ++c) d[c] *= grad_scale;
            reinterpret_cast<float4 *>(dr)[i] = make_float4(d[0], d[1], d[2], d[3]);
            if (dlogits_h) {
                __half2 a = __floats2half2_rn(d[0] * h_scale, d[1] * h_scale), b = __floats2half2_rn(d[2] * h_scale, d[3] * h_scale);
                uint2 o;
                o.x = *reinterpret_cast<unsigned *>(&a);
                o.y = *reinterpret_cast<unsigned *>(&b);
                reinterpret_cast<uint2 *>(dlogits_h + off)[i] = o;
            }
        }
    } else {
        for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
            const float p = expf(lr[i] - lse);
            const float d = (p - ((uint32_t)i == tgt ? 1.0f : 0.0f)) * grad_scale;
            dr[i] = d;
            if (dlogits_h) dlogits_h[off + i] = __float2half_rn(d * h_scale);
        }
    }
}

// ---- GRPO: PPO-clip gradient of the sampled-token log-probability w.r.t. the logits ----------------
// One block per position (grpo_policy_grad, shaders/q8_kernels.metal:698-761): log-softmax of the row,
// new_logprob = logit[action] - logsumexp, ratio = exp(new - old), the clip decides whether the position
// contributes (weight = -advantage) or not (0), dlogits = weight * ratio * (softmax - onehot(action)).
// Positions with no contribution (prompt positions carry advantage 0) are written as zeros without a
// second pass over the logits.
__global__ void __launch_bounds__(1024)
grpo_policy_grad_rows_kernel(const float *logits, const uint32_t *actions, const float *old_logprobs, const float *advantages,
                             float *new_logprobs, float *dlogits, int vocab, float clip_eps)
{
    __shared__ float sh_m[32], sh_s[32];
    const size_t off = (size_t)blockIdx.x * vocab;
    const float *lr = logits + off;
    uint32_t action = actions[blockIdx.x];
    if (action >= (uint32_t)vocab) action = 0;                     // never index outside the row
    const bool vec = (vocab & 3) == 0 && ((reinterpret_cast<uintptr_t>(logits) | reinterpret_cast<uintptr_t>(dlogits)) & 15) == 0;
    float m = -1e30f, sum = 0.f;
    if (vec) {
        const float4 *lr4 = reinterpret_cast<const float4 *>(lr);
        for (int i = threadIdx.x; i < vocab / 4; i += blockDim.x) {
            const float4 v = lr4[i];
            lse_add(m, sum, v.x); lse_add(m, sum, v.y); lse_add(m, sum, v.z); lse_add(m, sum, v.w);
        }
    } else {
        for (int i = threadIdx.x; i < vocab; i += blockDim.x) lse_add(m, sum, lr[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float mo = __shfl_xor_sync(0xffffffffu, m, o), so = __shfl_xor_sync(0xffffffffu, sum, o);
        const float mn = fmaxf(m, mo);
        sum = sum * expf(m - mn) + so * expf(mo - mn);
        m = mn;
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
    if (l == 0) { sh_m[w] = m; sh_s[w] = sum; }
    __syncthreads();
    float M = sh_m[0];
    for (int i = 1; i < nw; ++i) M = fmaxf(M, sh_m[i]);
    float S = 0.f;
    for (int i = 0; i < nw; ++i) S += sh_s[i] * expf(sh_m[i] - M);
    const float lse = logf(S) + M;

    const float new_lp = lr[action] - lse;
    if (threadIdx.x == 0) new_logprobs[blockIdx.x] = new_lp;
    const float adv = advantages[blockIdx.x];
    const float ratio = expf(new_lp - old_logprobs[blockIdx.x]);
    const float clipped = fminf(fmaxf(ratio, 1.0f - clip_eps), 1.0f + clip_eps);
    const float weight = adv >= 0.f ? (ratio <= clipped ? -adv : 0.0f) : (ratio >= clipped ? -adv : 0.0f);
    const float coef = weight * ratio;

    float *dr = dlogits + off;
    if (vec) {
        const float4 *lr4 = reinterpret_cast<const float4 *>(lr);
        for (int i = threadIdx.x; i < vocab / 4; i += blockDim.x) {
            float d[4] = {0.f, 0.f, 0.f, 0.f};
            if (coef != 0.0f) {
                const float4 v = lr4[i];
                d[0] = expf(v.x - lse); d[1] = expf(v.y - lse); d[2] = expf(v.z - lse); d[3] = expf(v.w - lse);
                if ((uint32_t)i == action / 4) d[action & 3] -= 1.0f;
#pragma unroll
                for (int c = 0; c < 4; ++c) d[c] *= coef;
            }
            reinterpret_cast<float4 *>(dr)[i] = make_float4(d[0], d[1], d[2], d[3]);
        }
    } else {
        for (int i = threadIdx.x; i < vocab; i += blockDim.x)
            dr[i] = coef != 0.0f ? coef * (expf(lr[i] - lse) - ((uint32_t)i == action ? 1.0f : 0.0f)) : 0.0f;
    }
}

// f16_sgd_apply (shaders/q8_kernels.metal:1195-1206) on fp32 holders of binary16 values:
// w <- half(w - lr * g), g <- 0
__global__ void sgd_apply_f16_kernel(float *w, float *g, size_t n, float lr)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        w[i] = __half2float(__float2half_rn(w[i] - lr * g[i]));
        g[i] = 0.0f;
    }
}

// x *= alpha (scale_tensor, the 1/G of the group mean in the GRPO step)
__global__ void scale_kernel(float *x, float alpha, size_t n)
{
    const size_t i0 = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4, stride = (size_t)gridDim.x * blockDim.x * 4;
    if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {
        for (size_t i = i0; i < n; i += stride) {
            if (i + 4 <= n) {
                float4 v = *reinterpret_cast<float4 *>(x + i);
                v.x *= alpha; v.y *= alpha; v.z *= alpha; v.w *= alpha;
                *reinterpret_cast<float4 *>(x + i) = v;
            } else {
                for (size_t j = i; j < n; ++j) x[j] *= alpha;
            }
        }
    } else {
        for (size_t i = i0; i < n; i += stride)
            for (size_t j = i; j < n && j < i + 4; ++j) x[j] *= alpha;
    }
}

// ---- frozen weights: binary16 values held as fp32, and their transposes ---------------------------
__global__ void round_f16_kernel(float *w, size_t n)
{
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        w[i] = __half2float(__float2half_rn(w[i]));
}

// dst[c, r] = src[r, c]; 32 x 32 tiles through shared memory so that both sides coalesce.
__global__ void transpose_f32_kernel(const float *src, int rows, int cols, float *dst)
{
    __shared__ float t[32][33];
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    for (int i = threadIdx.y; i < 32; i += 8) {
        const int r = r0 + i, c = c0 + threadIdx.x;
        t[i][threadIdx.x] = (r < rows && c < cols) ? src[(size_t)r * cols + c] : 0.f;
    }
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += 8) {
        const int c = c0 + i, r = r0 + threadIdx.x;
        if (c < cols && r < rows) dst[(size_t)c * rows + r] = t[threadIdx.x][i];
    }
}

// ---- binary16 operand copies for the tensor-core products --------------------------------------------
// dst = half(src * scale), four elements per thread (n a multiple of 4 is the fast path).
__global__ void f32_to_f16_kernel(const float *src, size_t n, float scale, __half *dst)
{
    const size_t n4 = n / 4;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (size_t)gridDim.x * blockDim.x) {
        const float4 v = reinterpret_cast<const float4 *>(src)[i];
        __half2 a = __floats2half2_rn(v.x * scale, v.y * scale), b = __floats2half2_rn(v.z * scale, v.w * scale);
        uint2 o;
        o.x = *reinterpret_cast<unsigned *>(&a);
        o.y = *reinterpret_cast<unsigned *>(&b);
        reinterpret_cast<uint2 *>(dst)[i] = o;
    }
    if (blockIdx.x == 0 && threadIdx.x < (n & 3)) dst[n4 * 4 + threadIdx.x] = __float2half_rn(src[n4 * 4 + threadIdx.x] * scale);
}

__global__ void transpose_f16_kernel(const __half *src, int rows, int cols, __half *dst)
{
    __shared__ __half t[32][34];
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    for (int i = threadIdx.y; i < 32; i += 8) {
        const int r = r0 + i, c = c0 + threadIdx.x;
        t[i][threadIdx.x] = (r < rows && c < cols) ? src[(size_t)r * cols + c] : __float2half(0.f);
    }
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += 8) {
        const int c = c0 + i, r = r0 + threadIdx.x;
        if (c < cols && r < rows) dst[(size_t)c * rows + r] = t[threadIdx.x][i];
    }
}

// ---- gradient norm, clip, AdamW ------------------------------------------------------------------
__global__ void __launch_bounds__(256) sumsq_partials_kernel(const float *g, size_t n, double *partials)
{
    __shared__ double sh[8];
    double acc = 0.0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const double v = (double)g[i];
        acc += v * v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int i = 0; i < 8; ++i) t += sh[i];
        partials[blockIdx.x] = t;
    }
}

__global__ void __launch_bounds__(256)
clip_adamw_kernel(float *p, float *g, float *m, float *v, size_t n, const double *partials, int n_partials,
                  float max_norm, float lr, float beta1, float beta2, float eps, float wd, float bc1, float bc2,
                  int apply_update, float *norm_out)
{
    __shared__ float s_scale;
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int i = 0; i < n_partials; ++i) t += partials[i];          // same order in every block
        const float norm = (float)sqrt(t);
        s_scale = norm > max_norm ? max_norm / norm : 1.0f;
        if (blockIdx.x == 0 && norm_out) norm_out[0] = norm;
    }
    __syncthreads();
    const float scale = s_scale;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        float gr = g[i];
        if (scale != 1.0f) { gr *= scale; g[i] = gr; }
        if (apply_update) {
            const float mi = beta1 * m[i] + (1.0f - beta1) * gr;
            const float vi = beta2 * v[i] + (1.0f - beta2) * gr * gr;
            m[i] = mi;
            v[i] = vi;
            const float pi = p[i];
            p[i] = pi - lr * ((mi / bc1) / (sqrtf(vi / bc2) + eps) + wd * pi);
        }
    }
}

inline int done()
{
    ++g_b200_launches;
    return (int)cudaGetLastError();
}

template <typename K>
int opt_in_smem(K kern, size_t bytes)
{
    if (bytes <= 48 * 1024) return 0;
    if (bytes > 200 * 1024) return B200_E_TOOLARGE;
    return (int)cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

}  // namespace

// ================================== C ABI =========================================================

extern "C" int b200_round_f16(float *w, size_t n, void *stream)
{
    if (!w || n == 0) return B200_E_BADARG;
    const unsigned grid = (unsigned)((n + 255) / 256 < 148 * 16 ? (n + 255) / 256 : 148 * 16);
    round_f16_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(w, n);
    return done();
}

extern "C" int b200_transpose_f32(const float *src, int rows, int cols, float *dst, void *stream)
{
    if (!src || !dst || rows <= 0 || cols <= 0 || (rows + 31) / 32 > 65535) return B200_E_BADARG;
    dim3 grid((cols + 31) / 32, (rows + 31) / 32), block(32, 8);
    transpose_f32_kernel<<<grid, block, 0, (cudaStream_t)stream>>>(src, rows, cols, dst);
    return done();
}

extern "C" int b200_embed_rows(const float *emb, const uint32_t *tokens, int rows, int dim, int vocab, float scale,
                               float *x, void *stream)
{
    if (!emb || !tokens || !x || rows <= 0 || dim <= 0 || vocab <= 0) return B200_E_BADARG;
    embed_rows_kernel<<<rows, 256, 0, (cudaStream_t)stream>>>(emb, tokens, dim, vocab, scale, x);
    return done();
}

extern "C" int b200_rms_norm_rows_h(const float *x, const float *gamma, float *out, void *out_h, int rows, int dim,
                                    float eps, void *stream)
{
    if (!x || !gamma || !out || rows <= 0 || dim <= 0) return B200_E_BADARG;
    cudaStream_t st = (cudaStream_t)stream;
    __half *oh = static_cast<__half *>(out_h);
    if (dim >= 1024 && dim <= 2560) rms_norm_held_kernel<10><<<rows, 256, 0, st>>>(x, gamma, out, oh, dim, eps);
    else if (dim >= 1024 && dim <= 4096) rms_norm_held_kernel<16><<<rows, 256, 0, st>>>(x, gamma, out, oh, dim, eps);
    else if (dim >= 1024) rms_norm_rows_kernel<256><<<rows, 256, 0, st>>>(x, gamma, out, oh, rows, dim, eps);
    else rms_norm_rows_kernel<32><<<(rows + 7) / 8, 256, 0, st>>>(x, gamma, out, oh, rows, dim, eps);
    return done();
}

extern "C" int b200_rms_norm_rows(const float *x, const float *gamma, float *out, int rows, int dim, float eps,
                                  void *stream)
{
    return b200_rms_norm_rows_h(x, gamma, out, nullptr, rows, dim, eps, stream);
}

extern "C" int b200_rms_norm_bwd_rows_h(const float *x, const float *dy, long long dy_ld, const float *gamma, float *dx,
                                        int rows, int dim, float eps, int accumulate, float clamp, void *dx_h,
                                        float h_scale, void *stream)
{
    if (!x || !dy || !gamma || !dx || rows <= 0 || dim <= 0 || dy_ld < dim) return B200_E_BADARG;
    cudaStream_t st = (cudaStream_t)stream;
    __half *dh = static_cast<__half *>(dx_h);
    if (dim >= 1024 && dim <= 2560)
        rms_norm_bwd_held_kernel<10><<<rows, 256, 0, st>>>(x, dy, dy_ld, gamma, dx, dim, eps, accumulate, clamp, dh, h_scale);
    else if (dim >= 1024 && dim <= 4096)
        rms_norm_bwd_held_kernel<16><<<rows, 256, 0, st>>>(x, dy, dy_ld, gamma, dx, dim, eps, accumulate, clamp, dh, h_scale);
    else if (dim >= 1024)
        rms_norm_bwd_rows_kernel<256><<<rows, 256, 0, st>>>(x, dy, dy_ld, gamma, dx, rows, dim, eps, accumulate, clamp, dh,
                                                            h_scale);
    else
        rms_norm_bwd_rows_kernel<32><<<(rows + 7) / 8, 256, 0, st>>>(x, dy, dy_ld, gamma, dx, rows, dim, eps, accumulate,
                                                                    clamp, dh, h_scale);
    return done();
}

extern "C" int b200_rms_norm_bwd_rows(const float *x, const float *dy, long long dy_ld, const float *gamma, float *dx,
                                      int rows, int dim, float eps, int accumulate, float clamp, void *stream)
{
    return b200_rms_norm_bwd_rows_h(x, dy, dy_ld, gamma, dx, rows, dim, eps, accumulate, clamp, nullptr, 1.0f, stream);
}

extern "C" int b200_qk_norm_rope(const float *qkv, long long ld, const float *q_gamma, const float *k_gamma,
                                 const float *inv_freq, int rows, int seq_len, int n_q, int n_kv, int hd, float eps,
                                 float *q_out, float *k_out, void *stream)
{
    if (!qkv || !q_gamma || !k_gamma || !inv_freq || !q_out || !k_out || rows <= 0 || seq_len <= 0) return B200_E_BADARG;
    const long long units = (long long)rows * (n_q + n_kv);
    const unsigned grid = (unsigned)((units + 7) / 8);
    cudaStream_t st = (cudaStream_t)stream;
    switch (hd) {
    case 64: qk_norm_rope_kernel<64><<<grid, 256, 0, st>>>(qkv, ld, q_gamma, k_gamma, inv_freq, rows, seq_len, n_q, n_kv, eps, q_out, k_out); break;
    case 128: qk_norm_rope_kernel<128><<<grid, 256, 0, st>>>(qkv, ld, q_gamma, k_gamma, inv_freq, rows, seq_len, n_q, n_kv, eps, q_out, k_out); break;
    case 256: qk_norm_rope_kernel<256><<<grid, 256, 0, st>>>(qkv, ld, q_gamma, k_gamma, inv_freq, rows, seq_len, n_q, n_kv, eps, q_out, k_out); break;
    default: return B200_E_BADARG;
    }
    return done();
}

extern "C" int b200_qk_norm_rope_bwd(float *dqkv, const float *qkv, long long ld, long long dld, const float *q_gamma,
                                     const float *k_gamma, const float *inv_freq, int rows, int seq_len, int n_q,
                                     int n_kv, int hd, float eps, void *stream)
{
    if (!dqkv || !qkv || !q_gamma || !k_gamma || !inv_freq || rows <= 0 || seq_len <= 0) return B200_E_BADARG;
    const long long units = (long long)rows * (n_q + n_kv);
    const unsigned grid = (unsigned)((units + 7) / 8);
    cudaStream_t st = (cudaStream_t)stream;
    switch (hd) {
    case 64: qk_norm_rope_bwd_kernel<64><<<grid, 256, 0, st>>>(dqkv, qkv, ld, dld, q_gamma, k_gamma, inv_freq, rows, seq_len, n_q, n_kv, eps); break;
    case 128: qk_norm_rope_bwd_kernel<128><<<grid, 256, 0, st>>>(dqkv, qkv, ld, dld, q_gamma, k_gamma, inv_freq, rows, seq_len, n_q, n_kv, eps); break;
    case 256: qk_norm_rope_bwd_kernel<256><<<grid, 256, 0, st>>>(dqkv, qkv, ld, dld, q_gamma, k_gamma, inv_freq, rows, seq_len, n_q, n_kv, eps); break;
    default: return B200_E_BADARG;
    }
    return done();
}

static bool attn_shape_ok(int n_seq, int seq_len, int n_q, int n_kv, int hd)
{
    return n_seq > 0 && seq_len > 0 && n_q > 0 && n_kv > 0 && n_q % n_kv == 0 && (hd == 64 || hd == 128 || hd == 256);
}

template <int HD, bool TC>
static int attn_fwd_launch(const float *q, const float *k, const float *v, long long v_ld, int n_seq, int N, int n_q,
                           int n_kv, float scale, float *probs, float *out, __half *out_h, cudaStream_t st)
{
    constexpr size_t smem = AttnTiles<HD>::bytes;
    int rc = opt_in_smem(attn_fwd_kernel<HD, TC>, smem);
    if (rc) return rc;
    attn_fwd_kernel<HD, TC><<<(N + AT - 1) / AT * n_seq * n_q, ATT_THREADS, smem, st>>>(q, k, v, v_ld, n_seq, N, n_q, n_kv, scale, probs, out, out_h);
    return done();
}

template <bool TC>
static int attn_fwd(const float *q, const float *k, const float *v, long long v_ld, int n_seq, int seq_len, int n_q, int n_kv, int hd, float scale,
                    float *probs, float *out, void *out_h, void *stream)
{
    if (!q || !k || !v || !probs || (!out && !out_h) || !attn_shape_ok(n_seq, seq_len, n_q, n_kv, hd)) return B200_E_BADARG;
    if ((v_ld & 3) || ((uintptr_t)v & 15) || ((uintptr_t)k & 15)) return B200_E_BADARG;     // 16-byte row loads
    cudaStream_t st = (cudaStream_t)stream;
    __half *oh = static_cast<__half *>(out_h);
    if (hd == 64) return attn_fwd_launch<64, TC>(q, k, v, v_ld, n_seq, seq_len, n_q, n_kv, scale, probs, out, oh, st);
    if (hd == 128) return attn_fwd_launch<128, TC>(q, k, v, v_ld, n_seq, seq_len, n_q, n_kv, scale, probs, out, oh, st);
    return attn_fwd_launch<256, TC>(q, k, v, v_ld, n_seq, seq_len, n_q, n_kv, scale, probs, out, oh, st);
}

extern "C" int b200_attn_train_fwd_h(const float *q, const float *k, const float *v, long long v_ld, int n_seq,
                                     int seq_len, int n_q, int n_kv, int hd, float scale, float *probs, float *out,
                                     void *out_h, void *stream)
{
    return attn_fwd<false>(q, k, v, v_ld, n_seq, seq_len, n_q, n_kv, hd, scale, probs, out, out_h, stream);
}

extern "C" int b200_attn_train_fwd_tc(const float *q, const float *k, const float *v, long long v_ld, int n_seq,
                                      int seq_len, int n_q, int n_kv, int hd, float scale, float *probs, float *out,
                                      void *out_h, void *stream)
{
    return attn_fwd<true>(q, k, v, v_ld, n_seq, seq_len, n_q, n_kv, hd, scale, probs, out, out_h, stream);
}

extern "C" int b200_attn_train_fwd(const float *q, const float *k, const float *v, long long v_ld, int n_seq,
                                   int seq_len, int n_q, int n_kv, int hd, float scale, float *probs, float *out,
                                   void *stream)
{
    if (!out) return B200_E_BADARG;
    return b200_attn_train_fwd_h(q, k, v, v_ld, n_seq, seq_len, n_q, n_kv, hd, scale, probs, out, nullptr, stream);
}

template <int HD, bool TC>
static int attn_bwd_launch(const float *d_out, const float *probs, const float *q, const float *k, const float *v,
                           long long v_ld, int n_seq, int N, int n_q, int n_kv, float scale, float *d_score,
                           float *dqkv, long long ld, cudaStream_t st)
{
    constexpr size_t smem = AttnTiles<HD>::bytes, smem_kv = 4 * (size_t)AT * (AT + 8) * sizeof(float);
    int rc = opt_in_smem(attn_bwd_dq_kernel<HD, TC>, smem);
    if (!rc) rc = opt_in_smem(attn_bwd_dkv_kernel<TC>, smem_kv);
    if (rc) return rc;
    const int tiles = (N + AT - 1) / AT;
    attn_bwd_dq_kernel<HD, TC><<<tiles * n_seq * n_q, ATT_THREADS, smem, st>>>(d_out, probs, k, v, v_ld, n_seq, N, n_q, n_kv, scale, d_score, dqkv, ld);
    rc = done();
    if (rc) return rc;
    attn_bwd_dkv_kernel<TC><<<tiles * n_seq * n_kv * 2 * (HD / 64), ATT_THREADS, smem_kv, st>>>(d_score, probs, q, d_out, n_seq, N, n_q, n_kv, HD, dqkv, ld);
    return done();
}

template <bool TC>
static int attn_bwd(const float *d_out, const float *probs, const float *q, const float *k, const float *v, long long v_ld, int n_seq, int seq_len,
                    int n_q, int n_kv, int hd, float scale, float *d_score, float *dqkv, long long ld, void *stream)
{
    if (!d_out || !probs || !q || !k || !v || !d_score || !dqkv || !attn_shape_ok(n_seq, seq_len, n_q, n_kv, hd))
        return B200_E_BADARG;
    if ((v_ld & 3) || ((uintptr_t)v & 15)) return B200_E_BADARG;
    cudaStream_t st = (cudaStream_t)stream;
    if (hd == 64) return attn_bwd_launch<64, TC>(d_out, probs, q, k, v, v_ld, n_seq, seq_len, n_q, n_kv, scale, d_score, dqkv, ld, st);
    if (hd == 128) return attn_bwd_launch<128, TC>(d_out, probs, q, k, v, v_ld, n_seq, seq_len, n_q, n_kv, scale, d_score, dqkv, ld, st);
    return attn_bwd_launch<256, TC>(d_out, probs, q, k, v, v_ld, n_seq, seq_len, n_q, n_kv, scale, d_score, dqkv, ld, st);
}

extern "C" int b200_attn_train_bwd(const float *d_out, const float *probs, const float *q, const float *k,
                                   const float *v, long long v_ld, int n_seq, int seq_len, int n_q, int n_kv, int hd,
                                   float scale, float *d_score, float *dqkv, long long ld, void *stream)
{
    return attn_bwd<false>(d_out, probs, q, k, v, v_ld, n_seq, seq_len, n_q, n_kv, hd, scale, d_score, dqkv, ld, stream);
}

extern "C" int b200_attn_train_bwd_tc(const float *d_out, const float *probs, const float *q, const float *k,
                                      const float *v, long long v_ld, int n_seq, int seq_len, int n_q, int n_kv, int hd,
                                      float scale, float *d_score, float *dqkv, long long ld, void *stream)
{
    return attn_bwd<true>(d_out, probs, q, k, v, v_ld, n_seq, seq_len, n_q, n_kv, hd, scale, d_score, dqkv, ld, stream);
}

// Rows of at least 64 quads: a block of 256 threads takes one row, and narrower ones leave most of it idle (2000 x 64 2.9 us in quads and 2.0 by elements,
// 2000 x 128 2.9 and 2.6, 2000 x 256 3.0 and 3.4).
static bool whole_quads(int inter, int rows, const void *a, const void *b, const void *c)
{
    return (inter & 3) == 0 && inter >= 256 && rows <= 65535 && (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 15) == 0;
}

extern "C" int b200_silu_mul_rows_h(const float *gu, int rows, int inter, float *act, void *act_h, void *stream)
{
    if (!gu || (!act && !act_h) || rows <= 0 || inter <= 0) return B200_E_BADARG;
    const size_t total = (size_t)rows * inter;
    const unsigned grid = (unsigned)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
    if (whole_quads(inter, rows, gu, act, act_h)) {
        glu_quads_kernel<Silu><<<dim3((inter / 4 + 255) / 256, rows), 256, 0, (cudaStream_t)stream>>>(gu, inter, act, static_cast<__half *>(act_h));
        return done();
    }
    silu_mul_rows_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(gu, inter, act, static_cast<__half *>(act_h), total);
    return done();
}

extern "C" int b200_silu_mul_rows(const float *gu, int rows, int inter, float *act, void *stream)
{
    if (!act) return B200_E_BADARG;
    return b200_silu_mul_rows_h(gu, rows, inter, act, nullptr, stream);
}

extern "C" int b200_silu_mul_bwd_rows_h(const float *d_act, const float *gu, int rows, int inter, float *d_gu, void *d_gu_h,
                                        float h_scale, void *stream)
{
    if (!d_act || !gu || (!d_gu && !d_gu_h) || rows <= 0 || inter <= 0) return B200_E_BADARG;
    const size_t total = (size_t)rows * inter;
    const unsigned grid = (unsigned)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
    if (whole_quads(inter, rows, gu, d_gu, d_gu_h) && ((uintptr_t)d_act & 15) == 0) {
        glu_bwd_quads_kernel<Silu><<<dim3((inter / 4 + 255) / 256, rows), 256, 0, (cudaStream_t)stream>>>(d_act, gu, inter, d_gu, static_cast<__half *>(d_gu_h), h_scale);
        return done();
    }
    silu_mul_bwd_rows_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(d_act, gu, inter, d_gu, static_cast<__half *>(d_gu_h),
                                                                    h_scale, total);
    return done();
}

extern "C" int b200_silu_mul_bwd_rows(const float *d_act, const float *gu, int rows, int inter, float *d_gu,
                                      void *stream)
{
    if (!d_gu) return B200_E_BADARG;
    return b200_silu_mul_bwd_rows_h(d_act, gu, rows, inter, d_gu, nullptr, 1.0f, stream);
}

extern "C" int b200_gelu_mul_rows(const float *gu, int rows, int inter, float *act, void *stream)
{
    if (!gu || !act || rows <= 0 || inter <= 0) return B200_E_BADARG;
    const size_t total = (size_t)rows * inter;
    const unsigned grid = (unsigned)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
    if (whole_quads(inter, rows, gu, act, nullptr)) {
        glu_quads_kernel<Gelu><<<dim3((inter / 4 + 255) / 256, rows), 256, 0, (cudaStream_t)stream>>>(gu, inter, act, nullptr);
        return done();
    }
    gelu_mul_rows_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(gu, inter, act, total);
    return done();
}

extern "C" int b200_gelu_mul_bwd_rows(const float *d_act, const float *gu, int rows, int inter, float *d_gu, void *stream)
{
    if (!d_act || !gu || !d_gu || rows <= 0 || inter <= 0) return B200_E_BADARG;
    const size_t total = (size_t)rows * inter;
    const unsigned grid = (unsigned)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
    if (whole_quads(inter, rows, gu, d_gu, nullptr) && ((uintptr_t)d_act & 15) == 0) {
        glu_bwd_quads_kernel<Gelu><<<dim3((inter / 4 + 255) / 256, rows), 256, 0, (cudaStream_t)stream>>>(d_act, gu, inter, d_gu, nullptr, 1.0f);
        return done();
    }
    gelu_mul_bwd_rows_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(d_act, gu, inter, d_gu, total);
    return done();
}

extern "C" int b200_add(const float *a, const float *b, float *out, size_t n, void *stream)
{
    if (!a || !b || !out) return B200_E_BADARG;
    if (n == 0) return 0;
    const unsigned grid = (unsigned)((n + 255) / 256 < 148 * 16 ? (n + 255) / 256 : 148 * 16);
    add_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(a, b, out, n);
    return done();
}

extern "C" int b200_lora_add(float *y, long long ld, int col0, int n_cols, const float *mid, long long mid_ld,
                             const float *B, int rank, float sc, int rows, void *stream)
{
    if (!y || !mid || !B || rank <= 0 || rank > 64 || rows <= 0 || n_cols <= 0 || mid_ld < rank) return B200_E_BADARG;
    if ((rows + LORA_ROWS - 1) / LORA_ROWS > 65535) return B200_E_TOOLARGE;
    dim3 grid((n_cols + 255) / 256, (rows + LORA_ROWS - 1) / LORA_ROWS);
    cudaStream_t st = (cudaStream_t)stream;
    if (rank <= 16) lora_add_kernel<16><<<grid, 256, 0, st>>>(y, ld, col0, n_cols, mid, mid_ld, B, rank, sc, rows);
    else lora_add_kernel<64><<<grid, 256, 0, st>>>(y, ld, col0, n_cols, mid, mid_ld, B, rank, sc, rows);
    return done();
}

extern "C" int b200_lora_pack(float *w_ext, float *wt_ext, const float *A_q, const float *B_q, const float *A_v,
                              const float *B_v, int d, int q_cols, int kv_cols, int rank, int xr, float sc, void *stream)
{
    if (!w_ext || !wt_ext || !A_q || !B_q || !A_v || !B_v || d <= 0 || q_cols <= 0 || kv_cols <= 0 || rank <= 0 ||
        xr < 2 * rank)
        return B200_E_BADARG;
    const int width = d > q_cols + 2 * kv_cols ? d : q_cols + 2 * kv_cols;
    dim3 grid((width + 255) / 256, xr);
    lora_pack_kernel<float><<<grid, 256, 0, (cudaStream_t)stream>>>(w_ext, wt_ext, A_q, B_q, A_v, B_v, d, q_cols, kv_cols,
                                                                   rank, xr, sc);
    return done();
}

extern "C" int b200_lora_pack_f16(void *w_ext, void *wt_ext, const float *A_q, const float *B_q, const float *A_v,
                                  const float *B_v, int d, int q_cols, int kv_cols, int rank, int xr, float sc,
                                  void *stream)
{
    if (!w_ext || !wt_ext || !A_q || !B_q || !A_v || !B_v || d <= 0 || q_cols <= 0 || kv_cols <= 0 || rank <= 0 ||
        xr < 2 * rank)
        return B200_E_BADARG;
    const int width = d > q_cols + 2 * kv_cols ? d : q_cols + 2 * kv_cols;
    dim3 grid((width + 255) / 256, xr);
    lora_pack_kernel<__half><<<grid, 256, 0, (cudaStream_t)stream>>>(static_cast<__half *>(w_ext), static_cast<__half *>(wt_ext),
                                                                    A_q, B_q, A_v, B_v, d, q_cols, kv_cols, rank, xr, sc);
    return done();
}

extern "C" int b200_f32_to_f16(const float *src, size_t n, float scale, void *dst, void *stream)
{
    if (!src || !dst || n == 0 || ((uintptr_t)src & 15) || ((uintptr_t)dst & 7)) return B200_E_BADARG;
    const size_t n4 = (n + 3) / 4;
    const unsigned grid = (unsigned)((n4 + 255) / 256 < 148 * 16 ? (n4 + 255) / 256 : 148 * 16);
    f32_to_f16_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(src, n, scale, static_cast<__half *>(dst));
    return done();
}

extern "C" int b200_transpose_f16(const void *src, int rows, int cols, void *dst, void *stream)
{
    if (!src || !dst || rows <= 0 || cols <= 0 || (rows + 31) / 32 > 65535) return B200_E_BADARG;
    dim3 grid((cols + 31) / 32, (rows + 31) / 32), block(32, 8);
    transpose_f16_kernel<<<grid, block, 0, (cudaStream_t)stream>>>(static_cast<const __half *>(src), rows, cols,
                                                                  static_cast<__half *>(dst));
    return done();
}

extern "C" int b200_xty_skinny(const float *X, long long ld_x, const float *Y, long long ld_y, int rows, int P, int R,
                               float alpha, float *C, long long c_p, long long c_r, void *stream)
{
    if (!X || !Y || !C || rows <= 0 || P <= 0 || R <= 0 || ld_x < P || ld_y < R) return B200_E_BADARG;
    if (R > 16) return B200_E_UNSUPPORTED;               // wider ranks go through b200_gemm_f32
    xty_skinny_kernel<16><<<(unsigned)((P + 15) / 16), 256, 0, (cudaStream_t)stream>>>(X, ld_x, Y, ld_y, rows, P, R, alpha,
                                                                                        C, c_p, c_r);
    return done();
}

extern "C" int b200_softmax_ce_rows_h(const float *logits, const uint32_t *targets, int rows, int vocab,
                                      float grad_scale, float *losses, float *dlogits, void *dlogits_h, float h_scale,
                                      void *stream)
{
    if (!logits || !targets || !losses || !dlogits || rows <= 0 || vocab <= 0) return B200_E_BADARG;
    softmax_ce_rows_kernel<<<rows, 1024, 0, (cudaStream_t)stream>>>(logits, targets, vocab, grad_scale, losses, dlogits,
                                                                   static_cast<__half *>(dlogits_h), h_scale);
    return done();
}

extern "C" int b200_softmax_ce_rows(const float *logits, const uint32_t *targets, int rows, int vocab,
                                    float grad_scale, float *losses, float *dlogits, void *stream)
{
    return b200_softmax_ce_rows_h(logits, targets, rows, vocab, grad_scale, losses, dlogits, nullptr, 1.0f, stream);
}

extern "C" int b200_grpo_policy_grad(const float *logits, const uint32_t *actions, const float *old_logprobs,
                                     const float *advantages, float *new_logprobs, float *dlogits, int rows, int vocab,
                                     float clip_eps, void *stream)
{
    if (!logits || !actions || !old_logprobs || !advantages || !new_logprobs || !dlogits || rows <= 0 || vocab <= 0)
        return B200_E_BADARG;
    grpo_policy_grad_rows_kernel<<<rows, 1024, 0, (cudaStream_t)stream>>>(logits, actions, old_logprobs, advantages,
                                                                         new_logprobs, dlogits, vocab, clip_eps);
    return done();
}

extern "C" int b200_sgd_apply_f16(float *w, float *g, size_t n, float lr, void *stream)
{
    if (!w || !g) return B200_E_BADARG;
    if (n == 0) return 0;
    const size_t want = (n + 255) / 256;
    const unsigned grid = (unsigned)(want < 148 * 8 ? want : 148 * 8);
    sgd_apply_f16_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(w, g, n, lr);
    return done();
}

extern "C" int b200_scale(float *x, float alpha, size_t n, void *stream)
{
    if (!x) return B200_E_BADARG;
    if (n == 0) return 0;
    const size_t want = (n / 4 + 255) / 256;
    const unsigned grid = (unsigned)(want < 148 * 8 ? (want ? want : 1) : 148 * 8);
    scale_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(x, alpha, n);
    return done();
}

extern "C" int b200_sumsq_partials(const float *g, size_t n, double *partials, int n_partials, void *stream)
{
    if (!g || !partials || n == 0 || n_partials <= 0 || n_partials > 4096) return B200_E_BADARG;
    sumsq_partials_kernel<<<n_partials, 256, 0, (cudaStream_t)stream>>>(g, n, partials);
    return done();
}

extern "C" int b200_clip_adamw(float *p, float *g, float *m, float *v, size_t n, const double *partials,
                               int n_partials, float max_norm, float lr, float beta1, float beta2, float eps, float wd,
                               float bc1, float bc2, int apply_update, float *norm_out, void *stream)
{
    if (!g || !partials || n == 0 || n_partials <= 0) return B200_E_BADARG;
    if (apply_update && (!p || !m || !v)) return B200_E_BADARG;
    const unsigned grid = (unsigned)((n + 255) / 256 < 148 * 8 ? (n + 255) / 256 : 148 * 8);
    clip_adamw_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(p, g, m, v, n, partials, n_partials, max_norm, lr, beta1,
                                                             beta2, eps, wd, bc1, bc2, apply_update, norm_out);
    return done();
}
