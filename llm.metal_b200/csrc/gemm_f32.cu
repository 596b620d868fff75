// CUDA-core fp32 GEMM with arbitrary unit-stride orientation of both operands.
//
// Carries the small and oddly shaped products of the LoRA-SFT step (the rank-R
// LoRA matmuls of src/nn/fast_sft.c:639-643, 946-966: float_matmul,
// float_matmul_tn, float_matmul_nt of shaders/q8_kernels.metal:1043-1152), every
// product of full-parameter training and of fp32 models, and is
// the any-shape fallback of the tensor-core GEMM for the frozen projections
// (f16_matmul :383-407, f16_matmul_nt :411-435). fp32 multiply-add throughout,
// k ascending within a block.
//
// Tile 64 x 64, 32 of k a step, 128 threads with 8 x 4 outputs each (48 bytes of shared memory per 32 multiply-adds and k). The next
// step's operands are in registers under the current one's products, two shared-memory buffers, one barrier a step; several
// blocks share an SM. The loader walks whichever dimension of an operand has stride 1 so that global reads coalesce; the
// transposing stores are spread over the banks by xor-ing k into the low bits of the position.
// A training step has 64 rows, so a product is few tiles with a long k (64 x 1152 x 6912: 18): up to eight blocks of a cluster
// share a tile along k, and each adds up an eighth of it from the others' shared memory, in rank order.
// Two full-parameter steps of 64 tokens (two layers of 1152 x 6912, vocabulary 8192): 14.9 ms with one block a tile and no prefetch, 4.1 ms with
// this kernel (3.5 with the tiled attention since).
// Bound by the latency of a step's operands where an SM has one block (64 x 1152 x 13824: 93 us), by the fp32 pipes elsewhere.
#include "common.cuh"
#include "../../include/llmb200_train_kernels.h"

extern unsigned long long g_b200_launches;

namespace {

constexpr int BM = 64, BN = 64, BK = 32, TM = 8, TN = 4, THREADS = 128, PITCH = BM + 4;
constexpr int PER = BM * BK / THREADS;           // elements of an operand tile per thread

__device__ __forceinline__ float finish(const b200_gemm_args &p, float v, const float *r)
{
    v *= p.alpha;
    if (r) v += *r;
    if (p.relu2) { v = fmaxf(v, 0.0f); v *= v; }
    return p.round_f16 ? __half2float(__float2half_rn(v)) : v;
}

// One operand: element (m, k) at base[m * row + k * col]; KC: contiguous along k.
template <bool KC>
struct Operand {
    const float *at;
    long long step;
    int m, k, m_end, k_end;                      // this thread's first element and the ends of the matrix
    __device__ __forceinline__ Operand(const float *base, long long row, long long col, int m0, int k0, int rows, int k_stop)
    {
        const int t = threadIdx.x;
        m = m0 + (KC ? t / BK : t % BM);
        k = k0 + (KC ? t % BK : t / BM);
        at = base + (long long)m * row + (long long)k * col;
        step = KC ? (THREADS / BK) * row : (THREADS / BM) * col;
        m_end = rows; k_end = k_stop;
    }
    __device__ __forceinline__ void load(float (&r)[PER]) const
    {
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const bool on = KC ? (m + i * (THREADS / BK) < m_end && k < k_end) : (m < m_end && k + i * (THREADS / BM) < k_end);
            r[i] = on ? __ldg(at + i * step) : 0.0f;
        }
    }
    __device__ __forceinline__ void next(long long col) { at += BK * col; k += BK; }
    __device__ __forceinline__ static void store(float (*s)[PITCH], const float (&r)[PER])
    {
        const int t = threadIdx.x;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int mm = KC ? t / BK + i * (THREADS / BK) : t % BM, kk = KC ? t % BK : t / BM + i * (THREADS / BM);
            s[kk][mm ^ (kk >> 3)] = r[i];
        }
    }
};

// AK: A is contiguous along k (a_col == 1); otherwise along m. BKC: B contiguous along k (b_row == 1).
template <bool AK, bool BKC>
__global__ void __launch_bounds__(THREADS, 3) gemm_f32_kernel(const __grid_constant__ b200_gemm_args p, int per_split)
{
    __shared__ __align__(16) float As[2][BK][PITCH], Bs[2][BK][PITCH];
    const int tid = threadIdx.x, m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tx = tid % 16, ty = tid / 16;      // columns 4 tx .., rows 8 ty ..
    const int k_begin = blockIdx.z * per_split, k_end = min(p.K, k_begin + per_split);
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    Operand<AK> a(p.A, p.a_row, p.a_col, m0, k_begin, p.M, k_end);
    Operand<BKC> b(p.B, p.b_col, p.b_row, n0, k_begin, p.N, k_end);
    float ra[PER], rb[PER];
    a.load(ra); b.load(rb);
    for (int k0 = k_begin, buf = 0; k0 < k_end; k0 += BK, buf ^= 1) {
        a.store(As[buf], ra); b.store(Bs[buf], rb);
        __syncthreads();
        a.next(p.a_col); b.next(p.b_row);
        if (k0 + BK < k_end) { a.load(ra); b.load(rb); }
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float av[TM], bv[TN];
#pragma unroll
            for (int q = 0; q < TM / 4; ++q) {
                const float4 v = *reinterpret_cast<const float4 *>(&As[buf][k][ty * TM + 4 * q]);
                const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) av[4 * q + (i ^ (k >> 3))] = f[i];
            }
            const float4 v = *reinterpret_cast<const float4 *>(&Bs[buf][k][tx * TN]);
            const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) bv[i ^ (k >> 3)] = f[i];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        // the other buffer was last read before this step's barrier: no second one
    }

    if (gridDim.z > 1) {
        __syncthreads();
        float *part = &As[0][0][0];              // [64][64]
#pragma unroll
        for (int i = 0; i < TM; ++i)
            *reinterpret_cast<float4 *>(part + (ty * TM + i) * BN + tx * TN) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        cluster_sync();
        const uint32_t base = (uint32_t)__cvta_generic_to_shared(part);
        const int rows = BM / gridDim.z, first = blockIdx.z * rows;
        for (int e = first * BN + 4 * tid; e < (first + rows) * BN; e += 4 * THREADS) {
            const int gm = m0 + e / BN, gn = n0 + e % BN;
            const float4 q = sum_ranks4(base + (uint32_t)e * 4, gridDim.z, 0, 1);
            const float v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (gm < p.M && gn + j < p.N)
                    p.C[(long long)gm * p.ldc + gn + j] = finish(p, v[j], p.R ? p.R + (long long)gm * p.ldr + gn + j : nullptr);
        }
        cluster_sync();
        return;
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty * TM + i, gn = n0 + tx * TN;
        if (gm >= p.M) continue;
        const float *r = p.R ? p.R + (long long)gm * p.ldr + gn : nullptr;
        float *c = p.C + (long long)gm * p.ldc + gn;
        if (gn + TN <= p.N && ((reinterpret_cast<uintptr_t>(c) | reinterpret_cast<uintptr_t>(r)) & 15) == 0) {
            const float4 q = r ? *reinterpret_cast<const float4 *>(r) : make_float4(0.f, 0.f, 0.f, 0.f);
            const float f[4] = {q.x, q.y, q.z, q.w};
            float o[4];
#pragma unroll
            for (int j = 0; j < TN; ++j) o[j] = finish(p, acc[i][j], r ? f + j : nullptr);
            *reinterpret_cast<float4 *>(c) = make_float4(o[0], o[1], o[2], o[3]);
        } else {
#pragma unroll
            for (int j = 0; j < TN; ++j)
                if (gn + j < p.N) c[j] = finish(p, acc[i][j], r ? r + j : nullptr);
        }
    }
}

}  // namespace

extern "C" int b200_gemm_f32(const b200_gemm_args *a, void *stream)
{
    if (!a || !a->A || !a->B || !a->C || a->M <= 0 || a->N <= 0 || a->K <= 0) return B200_E_BADARG;
    if ((a->a_row != 1 && a->a_col != 1) || (a->b_row != 1 && a->b_col != 1)) return B200_E_BADARG;
    const bool ak = a->a_col == 1, bk = a->b_row == 1;
    // Blocks per tile: enough for about four on every SM, as long as each keeps 128 of k.
    const long long tiles = (long long)((a->N + BN - 1) / BN) * ((a->M + BM - 1) / BM);
    int splits = 1;
    while (splits < 8 && tiles * splits * 2 <= 148 * 4 && a->K / (splits * 2) >= 128) splits *= 2;
    const int per = ((a->K + splits - 1) / splits + BK - 1) / BK * BK;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((a->N + BN - 1) / BN, (a->M + BM - 1) / BM, splits);
    cfg.blockDim = dim3(THREADS);
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 1; at.val.clusterDim.y = 1; at.val.clusterDim.z = splits;
    cfg.attrs = &at;
    cfg.numAttrs = splits > 1;
    cudaError_t rc;
    if (ak && bk) rc = cudaLaunchKernelEx(&cfg, gemm_f32_kernel<true, true>, *a, per);
    else if (ak) rc = cudaLaunchKernelEx(&cfg, gemm_f32_kernel<true, false>, *a, per);
    else if (bk) rc = cudaLaunchKernelEx(&cfg, gemm_f32_kernel<false, true>, *a, per);
    else rc = cudaLaunchKernelEx(&cfg, gemm_f32_kernel<false, false>, *a, per);
    ++g_b200_launches;
    return rc != cudaSuccess ? (int)rc : (int)cudaGetLastError();
}
