// Row-wise kernels of a prompt pass for the models of the per-token path (Qwen3, Gemma3), and its attention (sm_100a).
//
// The matrix products between them are b200_rows_matmul; here is what feeds it. Every kernel that makes a product's operand
// writes it as one or two binary16 planes of the row times a power of two (2^14 <= largest element < 2^15), so that two planes
// carry 22 bits of each element down to 2^-16 of the row's largest, and 2^-39 of the largest below; the factor that takes the power
// of two out again goes beside it. One plane without a factor is the plain rounding that the batched engine's products take.
// All of them move each row once: bound by HBM / L2 bytes, a block per row so that a short prompt still spreads over SMs. In short
// prompts and in decode steps of a batch they and the products are bound by their launches instead, 2 to 4 us each: every kernel lets
// the next one in at once and waits for the one before it after its set-up, so that a product's weights are on
// their way into shared memory while the row kernel before it runs.
#include "stream_core.cuh"
#include "../../include/llmb200_train_kernels.h"

#include <math.h>

extern unsigned long long g_b200_launches;

namespace {

constexpr int ROW_THREADS = 256;
constexpr size_t ROW_HELD = 227 * 1024 - 256;    // bytes of a row that shared memory holds beside a kernel's own

__device__ __forceinline__ float block_max(float v, float *red)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    v = warp_max(v);
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    v = red[0];
    for (int i = 1; i < nw; ++i) v = fmaxf(v, red[i]);
    return v;
}

// What an element counts for in its row's largest magnitude: infinities and NaN nothing, they stay what they are under any factor.
__device__ __forceinline__ float magnitude(float v)
{
    const float a = fabsf(v);
    return a < INFINITY ? a : 0.0f;
}
__device__ __forceinline__ float magnitude4(float4 v) { return fmaxf(fmaxf(magnitude(v.x), magnitude(v.y)), fmaxf(magnitude(v.z), magnitude(v.w))); }

// The power of two that brings a row's largest finite magnitude into [2^14, 2^15): up, and its inverse for the results. Rows of
// zeros stay as they are.
__device__ __forceinline__ float row_up(float mx, float *down)
{
    int e = 0;
    if (mx > 0.0f) { e = 14 - ilogbf(mx); e = e > 120 ? 120 : e; }
    *down = ldexpf(1.0f, -e);
    return ldexpf(1.0f, e);
}

__device__ __forceinline__ void split_pair(float a, float b, uint32_t &hi, uint32_t &lo)
{
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}

// The second plane of an element whose first is an infinity or NaN holds nothing: infinity minus infinity would make it NaN.
__device__ __forceinline__ uint32_t finite_low(uint32_t hi, uint32_t lo)
{
    if ((hi & 0x7c00u) == 0x7c00u) lo &= 0xffff0000u;
    if ((hi & 0x7c000000u) == 0x7c000000u) lo &= 0x0000ffffu;
    return lo;
}

__device__ __forceinline__ void put4(const b200_row_planes &o, long long row, int i4, float4 v, float up)
{
    uint2 hi, lo;
    split_pair(v.x * up, v.y * up, hi.x, lo.x);
    split_pair(v.z * up, v.w * up, hi.y, lo.y);
    __half *d = static_cast<__half *>(o.d_x) + row * o.ld + 4 * i4;
    *reinterpret_cast<uint2 *>(d) = hi;
    if (o.planes == 2) *reinterpret_cast<uint2 *>(d + (long long)o.plane_rows * o.ld) = make_uint2(finite_low(hi.x, lo.x), finite_low(hi.y, lo.y));
}

// x += (post ? post-normed y : y); planes of the RMS-normed x. index: row m of the output is row index[m] of x (no update then).
// HELD: the row stays in shared memory between the walks over it; wider rows are read again from where they lie.
template <bool HELD>
__global__ void __launch_bounds__(ROW_THREADS)
rows_norm_kernel(float *x, int dim, const float *y, const float *post, const float *gamma, const int *index, float eps, const b200_row_planes o)
{
    extern __shared__ __align__(16) float row_sh[];
    __shared__ float red[33];
    const int m = blockIdx.x, n4 = dim >> 2;
    pdl_launch_dependents();
    pdl_wait();
    float4 *xr = reinterpret_cast<float4 *>(x + (long long)(index ? index[m] : m) * dim);
    float4 *sh = reinterpret_cast<float4 *>(row_sh);
    const float4 *yr = y ? reinterpret_cast<const float4 *>(y + (long long)m * dim) : nullptr;
    float yinv = 1.0f;
    if (yr && post) {
        float ss = 0.0f;
        for (int i = threadIdx.x; i < n4; i += ROW_THREADS) {
            const float4 v = yr[i];
            if (HELD) sh[i] = v;
            ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
        }
        yinv = 1.0f / sqrtf(block_sum(ss, red) / (float)dim + eps);
    }
    float ss = 0.0f;
    for (int i = threadIdx.x; i < n4; i += ROW_THREADS) {
        float4 v = xr[i];
        if (yr) {
            float4 a = HELD && post ? sh[i] : yr[i];
            if (post) {
                const float4 g = reinterpret_cast<const float4 *>(post)[i];
                a.x *= yinv * g.x; a.y *= yinv * g.y; a.z *= yinv * g.z; a.w *= yinv * g.w;
            }
            v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
            xr[i] = v;
        }
        if (HELD) sh[i] = v;
        ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
    }
    const float inv = 1.0f / sqrtf(block_sum(ss, red) / (float)dim + eps);
    auto normed = [&](int i) {
        const float4 g = reinterpret_cast<const float4 *>(gamma)[i];
        float4 v = HELD ? sh[i] : xr[i];
        v.x *= inv * g.x; v.y *= inv * g.y; v.z *= inv * g.z; v.w *= inv * g.w;
        return v;
    };
    float mx = 0.0f;
    for (int i = threadIdx.x; i < n4; i += ROW_THREADS) {
        const float4 v = normed(i);
        if (HELD) sh[i] = v;
        mx = fmaxf(mx, magnitude4(v));
    }
    float up = 1.0f, down;
    if (o.d_scale) {
        up = row_up(block_max(mx, red), &down);
        if (threadIdx.x == 0) o.d_scale[m] = down;
    }
    for (int i = threadIdx.x; i < n4; i += ROW_THREADS) put4(o, m, i, HELD ? sh[i] : normed(i), up);
}

// Planes of act(gate) * up. Rows of 2 * inter: (gate, up) side by side in pairs, or all gates and then all ups. HELD as above; it matters
// with a factor only.
template <bool HELD>
__global__ void __launch_bounds__(ROW_THREADS)
rows_glu_kernel(const float *gu, int inter, int pairs, int gelu, const b200_row_planes o)
{
    extern __shared__ __align__(16) float row_sh[];
    __shared__ float red[33];
    const int m = blockIdx.x, n4 = inter >> 2;
    pdl_launch_dependents();
    pdl_wait();
    const float4 *g4 = reinterpret_cast<const float4 *>(gu + (long long)m * 2 * inter);
    float4 *sh = reinterpret_cast<float4 *>(row_sh);
    auto value = [&](int i) {
        const float4 a = __ldcs(g4 + (pairs ? 2 * i : i)), b = __ldcs(g4 + (pairs ? 2 * i + 1 : n4 + i));
        const float g[4] = {a.x, pairs ? a.z : a.y, pairs ? b.x : a.z, pairs ? b.z : a.w};
        const float u[4] = {pairs ? a.y : b.x, pairs ? a.w : b.y, pairs ? b.y : b.z, b.w};
        float v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = (gelu ? act_gelu_tanh(g[k]) : g[k] / (1.0f + expf(-g[k]))) * u[k];
        return make_float4(v[0], v[1], v[2], v[3]);
    };
    if (!o.d_scale) {                        // the row's elements do not depend on one another: several blocks share it
        for (int i = blockIdx.y * ROW_THREADS + threadIdx.x; i < n4; i += gridDim.y * ROW_THREADS) put4(o, m, i, value(i), 1.0f);
        return;
    }
    float mx = 0.0f, down;
    for (int i = threadIdx.x; i < n4; i += ROW_THREADS) {
        const float4 v = value(i);
        if (HELD) sh[i] = v;
        mx = fmaxf(mx, magnitude4(v));
    }
    const float up = row_up(block_max(mx, red), &down);
    if (threadIdx.x == 0) o.d_scale[m] = down;
    for (int i = threadIdx.x; i < n4; i += ROW_THREADS) put4(o, m, i, HELD ? sh[i] : value(i), up);
}

// Planes of plain rows.
__global__ void __launch_bounds__(ROW_THREADS)
rows_split_kernel(const float *x, int dim, const b200_row_planes o)
{
    __shared__ float red[33];
    const int m = blockIdx.x, n4 = dim >> 2;
    pdl_launch_dependents();
    pdl_wait();
    const float4 *xr = reinterpret_cast<const float4 *>(x + (long long)m * dim);
    float up = 1.0f, down;
    if (o.d_scale) {
        float mx = 0.0f;
        for (int i = threadIdx.x; i < n4; i += ROW_THREADS) {
            const float4 v = xr[i];
            mx = fmaxf(mx, magnitude4(v));
        }
        up = row_up(block_max(mx, red), &down);
        if (threadIdx.x == 0) o.d_scale[m] = down;
    }
    for (int i = blockIdx.y * ROW_THREADS + threadIdx.x; i < n4; i += gridDim.y * ROW_THREADS) put4(o, m, i, xr[i], up);
}

__global__ void __launch_bounds__(ROW_THREADS) rows_gather_kernel(const float *x, int dim, const int *index, float *out)
{
    pdl_launch_dependents();
    pdl_wait();
    const float4 *src = reinterpret_cast<const float4 *>(x + (long long)index[blockIdx.x] * dim);
    float4 *dst = reinterpret_cast<float4 *>(out + (long long)blockIdx.x * dim);
    for (int i = threadIdx.x; i < dim >> 2; i += ROW_THREADS) dst[i] = src[i];
}

// One warp per (row, head): query heads are normed, rotated and stored as two planes with a factor per row and head; key heads
// are normed and rotated into the binary16 cache, value heads copied there.
template <int HD>
__global__ void __launch_bounds__(128) rows_qkv_kernel(const b200_rows_attn_args p)
{
    constexpr int H2 = HD / 64;                               // pairs (d, d + HD/2) per lane
    const int lane = threadIdx.x & 31, m = blockIdx.x, h = blockIdx.y * 4 + (threadIdx.x >> 5), heads = p.n_q + 2 * p.n_kv;
    pdl_launch_dependents();
    pdl_wait();
    if (h >= heads) return;
    const int seq = m / p.seq_len, pos = p.pos0 + m % p.seq_len;
    const float *src = p.d_qkv + (long long)m * heads * HD + (long long)h * HD;
    float a[H2], b[H2];
#pragma unroll
    for (int j = 0; j < H2; ++j) { a[j] = src[lane + 32 * j]; b[j] = src[lane + 32 * j + HD / 2]; }
    if (h < p.n_q + p.n_kv) {
        const float *gm = h < p.n_q ? p.d_q_gamma : p.d_k_gamma;
        if (gm) {
            float ss = 0.0f;
#pragma unroll
            for (int j = 0; j < H2; ++j) ss = fmaf(a[j], a[j], fmaf(b[j], b[j], ss));
            const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)HD + p.eps);
#pragma unroll
            for (int j = 0; j < H2; ++j) { a[j] *= gm[lane + 32 * j] * inv; b[j] *= gm[lane + 32 * j + HD / 2] * inv; }
        }
#pragma unroll
        for (int j = 0; j < H2; ++j) {
            float sn, cs;
            sincosf((float)pos * p.d_inv_freq[lane + 32 * j], &sn, &cs);
            const float r0 = a[j] * cs - b[j] * sn, r1 = a[j] * sn + b[j] * cs;
            a[j] = r0; b[j] = r1;
        }
    }
    if (h < p.n_q) {
        float mx = 0.0f, down;
#pragma unroll
        for (int j = 0; j < H2; ++j) mx = fmaxf(mx, fmaxf(magnitude(a[j]), magnitude(b[j])));
        const float up = row_up(warp_max(mx), &down);
        const long long at = ((long long)m * p.n_q + h) * HD, plane = (long long)p.n_rows * p.n_q * HD;
        __half *q = static_cast<__half *>(p.d_q);
#pragma unroll
        for (int j = 0; j < H2; ++j) {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const float f = (k ? b[j] : a[j]) * up;
                const __half hi = __float2half_rn(f);
                const long long i = at + lane + 32 * j + k * (HD / 2);
                q[i] = hi;
                const float rest = f - __half2float(hi);
                q[plane + i] = __float2half_rn(fabsf(rest) < INFINITY ? rest : 0.0f);          // as finite_low
            }
        }
        if (lane == 0) p.d_q_scale[(long long)m * p.n_q + h] = down;
    } else {
        const int kvh = (h - p.n_q) % p.n_kv;
        __half *c = static_cast<__half *>(h < p.n_q + p.n_kv ? p.d_k_cache : p.d_v_cache) + (long long)seq * p.cache_seq_stride +
                    ((long long)kvh * p.max_seq + pos) * HD;
#pragma unroll
        for (int j = 0; j < H2; ++j) { c[lane + 32 * j] = __float2half_rn(a[j]); c[lane + 32 * j + HD / 2] = __float2half_rn(b[j]); }
    }
}

__device__ __forceinline__ void cp16(uint32_t dst, const void *src, bool on)
{
    const int n = on ? 16 : 0;                               // 0: the 16 bytes are zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void ldsm4(uint32_t a, uint32_t (&r)[4])
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ldsm4_t(uint32_t a, uint32_t (&r)[4])
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// z takes zero times eight binary16 values: it is NaN from the first infinity or NaN among them on.
__device__ __forceinline__ void zero_times8(__half2 &z, uint4 v)
{
    const __half2 zero = __floats2half2_rn(0.0f, 0.0f);
    z = __hfma2(*reinterpret_cast<const __half2 *>(&v.x), zero, z);
    z = __hfma2(*reinterpret_cast<const __half2 *>(&v.y), zero, z);
    z = __hfma2(*reinterpret_cast<const __half2 *>(&v.z), zero, z);
    z = __hfma2(*reinterpret_cast<const __half2 *>(&v.w), zero, z);
}
__device__ __forceinline__ float ex2(float x)                // 2^x, 2 ulp, 0 for -inf
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// A tile's scores and weighted sums in plain multiply-adds, laid out over the lanes as the tensor cores' fragments are; arrays through
// memory and out of line, so that the tiles that never need them keep their registers.
template <int HD, int BKEY>
__device__ __noinline__ void plain_scores(const __half *q, int plane, const __half *k, float *s)      // q: this lane's first row; the other 8 below
{
    constexpr int KS = HD + 8;
    for (int e = 0; e < BKEY / 2; ++e) {
        const __half *x = q + (e >> 1 & 1) * 8 * KS, *y = k + (e / 4 * 8 + (threadIdx.x & 3) * 2 + (e & 1)) * KS;
        float t = 0.0f;
        for (int d = 0; d < HD; ++d) t = fmaf(__half2float(x[d]) + __half2float(x[plane + d]), __half2float(y[d]), t);
        s[e] = t;
    }
}
template <int DV, int BKEY>
__device__ __noinline__ void plain_sums(const __half *v, int last, const float *w, float *o)           // last: the last key that the first row sees
{
    constexpr int VS = DV + 8;
    const int lane = threadIdx.x & 31;
    for (int key = 0; key < BKEY; ++key) {
        const int e = key / 8 * 4 + (key & 1), from = (lane & ~3) | (key % 8 / 2);
        const float p0 = __shfl_sync(0xffffffffu, w[e], from), p1 = __shfl_sync(0xffffffffu, w[e + 2], from);
        for (int i = 0; i < DV / 8; ++i) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(v + key * VS + i * 8 + (lane & 3) * 2));
            if (key <= last) { o[4 * i] = fmaf(p0, f.x, o[4 * i]); o[4 * i + 1] = fmaf(p0, f.y, o[4 * i + 1]); }
            if (key <= last + 8) { o[4 * i + 2] = fmaf(p1, f.x, o[4 * i + 2]); o[4 * i + 3] = fmaf(p1, f.y, o[4 * i + 3]); }
        }
    }
}

// Causal attention of the new rows over the binary16 cache: online softmax on mma.sync tiles, 16 query rows a warp, 32 keys a step
// with the next step's copies in flight. Keys and values are binary16 as they lie; queries and weights are fp32 numbers as two
// binary16 planes (22 bits), one product each, twice the products of a 16-bit attention. Sums start from zero every 32 of the head
// or of the keys and join in fp32 adds; corrections are summed apart. Off float64 1.6e-7 .. 1.7e-7, the per-token kernel 1.4e-7 .. 1.7e-7.
// Weights are formed times 2^14, which keeps the small ones' second plane away from binary16's lowest numbers; the factor cancels in the
// division by their sum. Tiles that hold an infinity or NaN (values beyond binary16) are summed in plain multiply-adds over the keys that a row
// sees: a later key's weight of zero would not keep them out, nor a second plane of zero.
// mma.sync and not tcgen05: the split of the weights stays in registers. 32 heads of 128: 512 / 1531 rows 46 / 246 us (42 / 208 when
// corrections and all of a score went through one accumulator, 4.9e-7 off); bound by instructions beside the products.
template <int HD, int NW>
__global__ void __launch_bounds__(NW * 32, HD == 256 ? 1 : HD == 128 && NW == 4 ? 3 : 16 / NW) rows_attn_kernel(const b200_rows_attn_args p)
{
    constexpr int DV = HD < 128 ? HD : 128, KS = HD + 8, VS = DV + 8, BQ = NW * 16, NT = NW * 32, BKEY = 32;
    static_assert(BKEY * (HD / 8) % NT == 0 && BKEY * (DV / 8) % NT == 0, "every thread copies as many chunks");
    extern __shared__ __align__(16) unsigned char smem[];
    __half *qsm = reinterpret_cast<__half *>(smem);          // [2 planes][BQ][KS]
    __half *ksm = qsm + 2 * BQ * KS;                         // [2][BKEY][KS]
    __half *vsm = ksm + 2 * BKEY * KS;                       // [2][BKEY][VS]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tiles_q = (p.seq_len + BQ - 1) / BQ, per_tile = gridDim.x / tiles_q, rank = rank_by_weight(HD < 256), part = rank % per_tile;
    const int h = part % p.n_q, c0 = part / p.n_q % (HD / DV) * DV, seq = part / (p.n_q * (HD / DV));
    const int m0 = (tiles_q - 1 - rank / per_tile) * BQ;                      // rows that see the most keys start first
    const int rows = min(BQ, p.seq_len - m0), first = p.pos0 + m0, last = first + rows - 1;
    const long long head = (long long)seq * p.cache_seq_stride + (long long)(h / (p.n_q / p.n_kv)) * p.max_seq * HD;
    const __half *keys = static_cast<const __half *>(p.d_k_cache) + head, *values = static_cast<const __half *>(p.d_v_cache) + head + c0;
    const long long row0 = (long long)seq * p.seq_len + m0, plane = (long long)p.n_rows * p.n_q * HD;
    const __half *qg = static_cast<const __half *>(p.d_q) + (row0 * p.n_q + h) * HD;
    const int tiles = last / BKEY + 1;
    pdl_launch_dependents();
    pdl_wait();

    for (int e = tid; e < 2 * BQ * (HD / 8); e += NT) {
        const int c = e % (HD / 8), r = e / (HD / 8) % BQ, u = e / (HD / 8 * BQ);
        const bool on = r < rows;
        cp16(smem_u32(qsm + (u * BQ + r) * KS + c * 8), on ? qg + u * plane + (long long)r * p.n_q * HD + c * 8 : qg, on);
    }
    auto stage = [&](int tile, int slot) {
        const int k0 = tile * BKEY, n = last - k0;           // rows past n hold zeros
        for (int e = tid; e < BKEY * (HD / 8); e += NT) {
            const int r = e / (HD / 8), c = e % (HD / 8);
            cp16(smem_u32(ksm + (slot * BKEY + r) * KS + c * 8), r <= n ? keys + (long long)(k0 + r) * HD + c * 8 : keys, r <= n);
        }
        for (int e = tid; e < BKEY * (DV / 8); e += NT) {
            const int r = e / (DV / 8), c = e % (DV / 8);
            cp16(smem_u32(vsm + (slot * BKEY + r) * VS + c * 8), r <= n ? values + (long long)(k0 + r) * HD + c * 8 : values, r <= n);
        }
        cp_commit();
    };
    stage(0, 0);

    float o[DV / 8][4];
#pragma unroll
    for (int i = 0; i < DV / 8; ++i)
#pragma unroll
        for (int k = 0; k < 4; ++k) o[i][k] = 0.0f;
    float mx[2] = {-INFINITY, -INFINITY}, l[2] = {0.0f, 0.0f}, sc[2];
    const int r0 = warp * 16 + (lane >> 2);                  // this thread's rows: r0 and r0 + 8
    const float scale = 1.4426950408889634f / sqrtf((float)HD);
#pragma unroll
    for (int r = 0; r < 2; ++r) sc[r] = r0 + 8 * r < rows ? p.d_q_scale[(row0 + r0 + 8 * r) * p.n_q + h] * scale : 0.0f;
    const uint32_t qaddr = smem_u32(qsm + (warp * 16 + (lane & 15)) * KS + (lane >> 4) * 8);

    for (int tile = 0; tile < tiles; ++tile) {
        const int slot = tile & 1;
        if (tile + 1 < tiles) { stage(tile + 1, slot ^ 1); cp_wait<1>(); }
        else cp_wait<0>();
        // every thread looks through what it copied itself: the barrier that follows tells all of them
        __half2 z = __floats2half2_rn(0.0f, 0.0f);
#pragma unroll
        for (int e = 0; e < BKEY * (HD / 8); e += NT)
            zero_times8(z, lds_128(smem_u32(ksm + (slot * BKEY + (tid + e) / (HD / 8)) * KS + (tid + e) % (HD / 8) * 8)));
#pragma unroll
        for (int e = 0; e < BKEY * (DV / 8); e += NT)
            zero_times8(z, lds_128(smem_u32(vsm + (slot * BKEY + (tid + e) / (DV / 8)) * VS + (tid + e) % (DV / 8) * 8)));
        const bool plainly = __syncthreads_or(!__hbeq2(z, z));
        const int k0 = tile * BKEY, w_first = first + warp * 16;
        if (k0 <= w_first + 15) {                            // else all of it is ahead of the warp's rows
            float s[BKEY / 8][4];
#pragma unroll
            for (int i = 0; i < BKEY / 8; ++i)
#pragma unroll
                for (int k = 0; k < 4; ++k) s[i][k] = 0.0f;
            if (plainly) {
                float t[BKEY / 8 * 4];
                plain_scores<HD, BKEY>(qsm + r0 * KS, BQ * KS, ksm + slot * BKEY * KS, t);
#pragma unroll
                for (int i = 0; i < BKEY / 2; ++i) s[i / 4][i % 4] = t[i];
            } else {
                const uint32_t kaddr = smem_u32(ksm + slot * BKEY * KS + ((lane & 7) + ((lane >> 4) << 3)) * KS + ((lane >> 3) & 1) * 8);
                float low[BKEY / 8][4] = {};
#pragma unroll 1
                for (int d0 = 0; d0 < HD; d0 += 32) {
                    float t[BKEY / 8][4] = {};
#pragma unroll
                    for (int kk = d0; kk < d0 + 32; kk += 16) {
                        uint32_t a[4], a2[4];
                        ldsm4(qaddr + kk * 2, a);
                        ldsm4(qaddr + (BQ * KS + kk) * 2, a2);
#pragma unroll
                        for (int n = 0; n < BKEY / 16; ++n) {
                            uint32_t b[4];
                            ldsm4(kaddr + (uint32_t)(n * 16 * KS + kk) * 2, b);
                            mma_f16(t[2 * n], a, b[0], b[1]);
                            mma_f16(t[2 * n + 1], a, b[2], b[3]);
                            mma_f16(low[2 * n], a2, b[0], b[1]);
                            mma_f16(low[2 * n + 1], a2, b[2], b[3]);
                        }
                    }
#pragma unroll
                    for (int n = 0; n < BKEY / 8; ++n)
#pragma unroll
                        for (int k = 0; k < 4; k += 2) add_pair(s[n][k], s[n][k + 1], t[n][k], t[n][k + 1]);
                }
#pragma unroll
                for (int n = 0; n < BKEY / 8; ++n)
#pragma unroll
                    for (int k = 0; k < 4; k += 2) add_pair(s[n][k], s[n][k + 1], low[n][k], low[n][k + 1]);
            }
            if (k0 + BKEY - 1 > w_first) {
                const int d0 = first + r0 - k0 - (lane & 3) * 2;
#pragma unroll
                for (int n = 0; n < BKEY / 8; ++n)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (d0 + (k >> 1) * 8 - n * 8 - (k & 1) < 0) s[n][k] = -INFINITY;
            }
            float mt[2] = {mx[0], mx[1]};
#pragma unroll
            for (int n = 0; n < BKEY / 8; ++n) {
                mt[0] = fmaxf(mt[0], fmaxf(s[n][0], s[n][1]));
                mt[1] = fmaxf(mt[1], fmaxf(s[n][2], s[n][3]));
            }
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                mt[r] = fmaxf(mt[r], __shfl_xor_sync(0xffffffffu, mt[r], 1));
                mt[r] = fmaxf(mt[r], __shfl_xor_sync(0xffffffffu, mt[r], 2));
            }
            // differences first: the score at the maximum weighs exactly one (times 2^14), whatever its size; no difference of infinities
            const float top[2] = {mt[0] == -INFINITY ? 0.0f : mt[0], mt[1] == -INFINITY ? 0.0f : mt[1]};
            const float corr[2] = {ex2((mx[0] - top[0]) * sc[0]), ex2((mx[1] - top[1]) * sc[1])};
            const bool moved = mt[0] != mx[0] || mt[1] != mx[1];
            mx[0] = mt[0]; mx[1] = mt[1];
            float ls[2] = {0.0f, 0.0f};
#pragma unroll
            for (int n = 0; n < BKEY / 8; ++n)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    s[n][k] = ex2((s[n][k] - top[k >> 1]) * sc[k >> 1]) * 16384.0f;      // the factor in the exponent would cost its bits
                    ls[k >> 1] += s[n][k];
                }
            l[0] = fmaf(l[0], corr[0], ls[0]);
            l[1] = fmaf(l[1], corr[1], ls[1]);
            if (__any_sync(0xffffffffu, moved)) {
#pragma unroll
                for (int i = 0; i < DV / 8; ++i) { mul_pair(o[i][0], o[i][1], corr[0], corr[0]); mul_pair(o[i][2], o[i][3], corr[1], corr[1]); }
            }
            if (plainly) {
                float w[BKEY / 8 * 4], t[DV / 8 * 4];
#pragma unroll
                for (int i = 0; i < BKEY / 2; ++i) w[i] = s[i / 4][i % 4];
#pragma unroll
                for (int i = 0; i < DV / 2; ++i) t[i] = o[i / 4][i % 4];
                plain_sums<DV, BKEY>(vsm + slot * BKEY * VS, first + r0 - k0, w, t);
#pragma unroll
                for (int i = 0; i < DV / 2; ++i) o[i / 4][i % 4] = t[i];
            } else {
                const uint32_t vaddr = smem_u32(vsm + slot * BKEY * VS + (lane & 15) * VS + (lane >> 4) * 8);
                uint32_t a[BKEY / 16][4], a2[BKEY / 16][4];
#pragma unroll
                for (int kk = 0; kk < BKEY / 16; ++kk) {
                    split_pair(s[2 * kk][0], s[2 * kk][1], a[kk][0], a2[kk][0]);
                    split_pair(s[2 * kk][2], s[2 * kk][3], a[kk][1], a2[kk][1]);
                    split_pair(s[2 * kk + 1][0], s[2 * kk + 1][1], a[kk][2], a2[kk][2]);
                    split_pair(s[2 * kk + 1][2], s[2 * kk + 1][3], a[kk][3], a2[kk][3]);
                }
                // the step's sums start from zero, corrections first, and join the rows' in fp32 adds: tensor cores truncate when they
                // accumulate, which over a long prompt would add up (5e-6 of a row at 700 keys otherwise)
#pragma unroll
                for (int n = 0; n < DV / 16; ++n) {
                    float t[2][4] = {};
                    uint32_t b[BKEY / 16][4];
#pragma unroll
                    for (int kk = 0; kk < BKEY / 16; ++kk) ldsm4_t(vaddr + (uint32_t)(kk * 16 * VS + n * 16) * 2, b[kk]);
#pragma unroll
                    for (int kk = 0; kk < BKEY / 16; ++kk) { mma_f16(t[0], a2[kk], b[kk][0], b[kk][1]); mma_f16(t[1], a2[kk], b[kk][2], b[kk][3]); }
#pragma unroll
                    for (int kk = 0; kk < BKEY / 16; ++kk) { mma_f16(t[0], a[kk], b[kk][0], b[kk][1]); mma_f16(t[1], a[kk], b[kk][2], b[kk][3]); }
#pragma unroll
                    for (int k = 0; k < 4; k += 2) { add_pair(o[2 * n][k], o[2 * n][k + 1], t[0][k], t[0][k + 1]); add_pair(o[2 * n + 1][k], o[2 * n + 1][k + 1], t[1][k], t[1][k + 1]); }
                }
            }
        }
        __syncthreads();                                     // the slot is overwritten by the next round's copies
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
        if (r0 + 8 * r >= rows) continue;
        const float inv = 1.0f / l[r];
        float *out = p.d_out + ((row0 + r0 + 8 * r) * p.n_q + h) * HD + c0 + (lane & 3) * 2;
#pragma unroll
        for (int i = 0; i < DV / 8; ++i) *reinterpret_cast<float2 *>(out + i * 8) = make_float2(o[i][2 * r] * inv, o[i][2 * r + 1] * inv);
    }
}

template <typename K>
int allow_smem(K kern, size_t smem)          // beside less than 1 KB of a kernel's own
{
    if (smem > 227 * 1024) return B200_E_TOOLARGE;
    return smem > 47 * 1024 ? (int)cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) : 0;
}

template <int HD, int NW>
int launch_attn(const b200_rows_attn_args &a, cudaStream_t st)
{
    constexpr int DV = HD < 128 ? HD : 128;
    constexpr size_t smem = (size_t)(2 * NW * 16 * (HD + 8) + 2 * 32 * (HD + 8) + 2 * 32 * (DV + 8)) * 2;
    const int rc = allow_smem(rows_attn_kernel<HD, NW>, smem);
    if (rc) return rc;
    ++g_b200_launches;
    return (int)launch_chained(rows_attn_kernel<HD, NW>, dim3((a.seq_len + NW * 16 - 1) / (NW * 16) * a.n_q * (HD / DV) * (a.n_rows / a.seq_len)),
                               dim3(NW * 32), smem, st, a);
}

template <int HD>
int rows_attn(const b200_rows_attn_args &a, cudaStream_t st)
{
    ++g_b200_launches;
    const int rc = (int)launch_chained(rows_qkv_kernel<HD>, dim3(a.n_rows, (a.n_q + 2 * a.n_kv + 3) / 4), dim3(128), 0, st, a);
    // 128 query rows a block where that still fills the machine (a tile of keys serves twice the rows), 64 otherwise
    const long long blocks = (long long)((a.seq_len + 127) / 128) * a.n_q * (HD > 128 ? 2 : 1) * (a.n_rows / a.seq_len);
    return rc ? rc : blocks >= 148 ? launch_attn<HD, 8>(a, st) : launch_attn<HD, 4>(a, st);
}

// Blocks per row where they can share it: about two waves of them, each with an element group for every thread.
int share_row(int rows, int dim)
{
    const int most = (dim / 4 + ROW_THREADS - 1) / ROW_THREADS, want = (148 * 4 + rows - 1) / rows;
    return want < most ? want : most;
}

bool planes_ok(const b200_row_planes *o, int rows, int dim)
{
    return o && o->d_x && (o->planes == 1 || (o->planes == 2 && o->plane_rows >= rows && o->d_scale)) && o->ld >= dim && (o->ld & 3) == 0 &&
           (reinterpret_cast<uintptr_t>(o->d_x) & 15) == 0;
}

}  // namespace

extern "C" int b200_rows_norm_planes(float *x, int rows, int dim, const float *y, const float *post_gamma, const float *gamma,
                                     const int *index, float eps, const b200_row_planes *out, void *stream)
{
    if (!x || !gamma || rows <= 0 || dim <= 0 || (dim & 3) || (index && y) || (post_gamma && !y) || !planes_ok(out, rows, dim)) return B200_E_BADARG;
    const size_t smem = (size_t)dim * 4 <= ROW_HELD ? (size_t)dim * 4 : 0;
    const auto kern = smem ? rows_norm_kernel<true> : rows_norm_kernel<false>;
    const int rc = allow_smem(kern, smem);
    if (rc) return rc;
    ++g_b200_launches;
    return (int)launch_chained(kern, dim3(rows), dim3(ROW_THREADS), smem, (cudaStream_t)stream, x, dim, y, post_gamma, gamma, index, eps, *out);
}

extern "C" int b200_rows_glu_planes(const float *gu, int rows, int inter, int pairs, int gelu, const b200_row_planes *out, void *stream)
{
    if (!gu || rows <= 0 || inter <= 0 || (inter & 3) || !planes_ok(out, rows, inter)) return B200_E_BADARG;
    const size_t smem = out->d_scale && (size_t)inter * 4 <= ROW_HELD ? (size_t)inter * 4 : 0;
    const auto kern = smem ? rows_glu_kernel<true> : rows_glu_kernel<false>;
    const int rc = allow_smem(kern, smem);
    if (rc) return rc;
    ++g_b200_launches;
    return (int)launch_chained(kern, dim3(rows, out->d_scale ? 1 : share_row(rows, inter)), dim3(ROW_THREADS), smem, (cudaStream_t)stream, gu, inter,
                               pairs, gelu, *out);
}

extern "C" int b200_rows_split_planes(const float *x, int rows, int dim, const b200_row_planes *out, void *stream)
{
    if (!x || rows <= 0 || dim <= 0 || (dim & 3) || !planes_ok(out, rows, dim)) return B200_E_BADARG;
    ++g_b200_launches;
    return (int)launch_chained(rows_split_kernel, dim3(rows, out->d_scale ? 1 : share_row(rows, dim)), dim3(ROW_THREADS), 0, (cudaStream_t)stream,
                               x, dim, *out);
}

extern "C" int b200_rows_gather(const float *x, int rows, int dim, const int *index, float *out, void *stream)
{
    if (!x || !index || !out || rows <= 0 || dim <= 0 || (dim & 3) || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & 15))
        return B200_E_BADARG;
    ++g_b200_launches;
    return (int)launch_chained(rows_gather_kernel, dim3(rows), dim3(ROW_THREADS), 0, (cudaStream_t)stream, x, dim, index, out);
}

extern "C" int b200_rows_attn(const b200_rows_attn_args *a, void *stream)
{
    if (!a || !a->d_qkv || !a->d_inv_freq || !a->d_k_cache || !a->d_v_cache || !a->d_q || !a->d_q_scale || !a->d_out) return B200_E_BADARG;
    if (a->n_rows <= 0 || a->seq_len <= 0 || a->n_rows % a->seq_len || a->n_q <= 0 || a->n_kv <= 0 || a->n_q % a->n_kv) return B200_E_BADARG;
    if (a->pos0 < 0 || a->pos0 + a->seq_len > a->max_seq || a->n_rows / a->seq_len > 65535) return B200_E_TOOLARGE;
    switch (a->hd) {
    case 64: return rows_attn<64>(*a, (cudaStream_t)stream);
    case 128: return rows_attn<128>(*a, (cudaStream_t)stream);
    case 256: return rows_attn<256>(*a, (cudaStream_t)stream);
    default: return B200_E_UNSUPPORTED;
    }
}
