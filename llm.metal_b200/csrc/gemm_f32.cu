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
// Tile 64 x 64, 32 of k a step, 128 threads with 8 x 4 outputs each. Steps arrive with cp.async, three ahead of the one that is multiplied, in the
// order that memory has them: rows of k where an operand is contiguous along k, rows of m (n) otherwise; 16 bytes at a time where
// addresses allow. A thread reads four of k of its operands with 16-byte loads in either order (12 loads for 128 multiply-adds) and multiplies in pairs
// (fma.rn.f32x2): pairs of k where both operands have them side by side, pairs of outputs otherwise. Pitches keep the loads of a
// warp off each other's banks.
// A training step has 64 rows, so a product is few tiles with a long k (64 x 1152 x 6912: 18): the blocks of a cluster
// share a tile along k, and each adds up a share of it from the others' shared memory, in rank order.
// Bound by the fp32 pipes, busy half of the time, and shared memory's port, a third of it; 13824 x 1152 x 64 60 us, 74 with operands of the next step
// in registers and one multiply-add an instruction, the form that short products keep.
#include "common.cuh"
#include "../../include/llmb200_train_kernels.h"

extern unsigned long long g_b200_launches;

namespace {

constexpr int BM = 64, BN = 64, BK = 32, TM = 8, TN = 4, GROUP = 128, STEPS = 4;
constexpr int PITCH_K = BK + 4, PITCH_M = BM + 4;        // floats between rows of k, and between rows of m
constexpr int TILE = BM * PITCH_K, STAGE = 2 * TILE;     // floats of an operand's tile and of a step (32 rows of PITCH_M are less)

__device__ __forceinline__ float finish(const b200_gemm_args &p, float v, const float *r)
{
    v *= p.alpha;
    if (r) v += *r;
    if (p.relu2) { v = fmaxf(v, 0.0f); v *= v; }
    return p.round_f16 ? __half2float(__float2half_rn(v)) : v;
}

__device__ __forceinline__ void copy16(float *dst, const float *src, int n)          // n floats of four, zeros beyond
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(4 * n) : "memory");
}
__device__ __forceinline__ void copy4(float *dst, const float *src, int n)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(4 * n) : "memory");
}

// Copies `lines` lines of `len` floats (a multiple of four) from line l0, place e0 on; zeros beyond the ends. Lines are `ld` apart in memory.
template <int LINES, int LEN, int PITCH, int THREADS>
__device__ __forceinline__ void copy_tile(float *dst, const float *base, long long ld, int l0, int l_end, int e0, int e_end, bool vec)
{
    if (vec) {
#pragma unroll
        for (int c = threadIdx.x; c < LINES * LEN / 4; c += THREADS) {
            const int l = c / (LEN / 4), e = c % (LEN / 4) * 4;
            const int n = l0 + l < l_end ? max(0, min(4, e_end - e0 - e)) : 0;
            copy16(dst + l * PITCH + e, n ? base + (long long)(l0 + l) * ld + e0 + e : base, n);
        }
    } else {
#pragma unroll 4
        for (int c = threadIdx.x; c < LINES * LEN; c += THREADS) {
            const int l = c / LEN, e = c % LEN;
            const int n = l0 + l < l_end && e0 + e < e_end;
            copy4(dst + l * PITCH + e, n ? base + (long long)(l0 + l) * ld + e0 + e : base, n);
        }
    }
}
// One operand's tile of a step: 64 of m (n), 32 of k. KC: contiguous along k.
template <bool KC, int THREADS>
__device__ __forceinline__ void copy_operand(float *dst, const float *base, long long ld, int m0, int m_end, int k0, int k_end, bool vec)
{
    if (KC) copy_tile<BM, BK, PITCH_K, THREADS>(dst, base, ld, m0, m_end, k0, k_end, vec);
    else copy_tile<BK, BM, PITCH_M, THREADS>(dst, base, ld, k0, k_end, m0, m_end, vec);
}

// The sums of the block's tile lie in part, [64][PITCH_M]: the blocks of the cluster each add up and store a share of the rows, in rank order.
template <int THREADS>
__device__ __forceinline__ void store_tile(const b200_gemm_args &p, const float *part, int m0, int n0)
{
    const int tid = threadIdx.x;
    const int ranks = gridDim.z, rows = (BM + ranks - 1) / ranks, first = blockIdx.z * rows, last = min(first + rows, BM);
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(part);
    const bool vec = ((reinterpret_cast<uintptr_t>(p.C) | reinterpret_cast<uintptr_t>(p.R)) & 15) == 0 && ((p.ldc | (p.R ? p.ldr : 0)) & 3) == 0;
#pragma unroll 4
    for (int e = first * BN + 4 * tid; e < last * BN; e += 4 * THREADS) {
        const int lm = e / BN, ln = e % BN, gm = m0 + lm, gn = n0 + ln;
        if (gm >= p.M || gn >= p.N) continue;
        const float *r = p.R ? p.R + (long long)gm * p.ldr + gn : nullptr;
        float *c = p.C + (long long)gm * p.ldc + gn;
        const bool whole = vec && gn + 4 <= p.N;
        float f[4] = {};
        if (whole && r) *reinterpret_cast<float4 *>(f) = *reinterpret_cast<const float4 *>(r);
        const float4 q = ranks > 1 ? sum_ranks4(base + (uint32_t)(lm * PITCH_M + ln) * 4, ranks, 0, 1) : *reinterpret_cast<const float4 *>(part + lm * PITCH_M + ln);
        const float v[4] = {q.x, q.y, q.z, q.w};
        if (whole) {
            float o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) o[j] = finish(p, v[j], r ? f + j : nullptr);
            *reinterpret_cast<float4 *>(c) = make_float4(o[0], o[1], o[2], o[3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (gn + j < p.N) c[j] = finish(p, v[j], r ? r + j : nullptr);
        }
    }
    if (ranks > 1) cluster_sync();                                       // nobody leaves while a peer still reads
}

// AK: A is contiguous along k (a_col == 1); otherwise along m. BKC: B contiguous along k (b_row == 1). KG: groups of threads that share the steps.
template <bool AK, bool BKC, int KG>
__global__ void __launch_bounds__(GROUP * KG, KG == 1 ? 3 : 1) gemm_f32_kernel(const __grid_constant__ b200_gemm_args p, int per_split)
{
    constexpr int THREADS = GROUP * KG;
    extern __shared__ __align__(16) float sh[];                          // steps; then the tile's sums
    const int tid = threadIdx.x, kg = tid / GROUP, t = tid % GROUP, m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tx = t % 16, ty = t / 16;
    const int k_begin = blockIdx.z * per_split, k_end = min(p.K, k_begin + per_split), n_steps = max(0, (k_end - k_begin + BK - 1) / BK);
    const long long a_ld = AK ? p.a_row : p.a_col, b_ld = BKC ? p.b_col : p.b_row;
    const bool a_vec = ((reinterpret_cast<uintptr_t>(p.A) & 15) | (a_ld & 3)) == 0, b_vec = ((reinterpret_cast<uintptr_t>(p.B) & 15) | (b_ld & 3)) == 0;
    // this thread's outputs: rows and columns that its loads of a warp find on different banks
    auto row_of = [&](int i) { return AK ? ty + 8 * i : TM * ty + i; };
    auto col_of = [&](int j) { return BKC ? tx + 16 * j : TN * tx + j; };

    auto stage = [&](int step) {
        if (step < n_steps) {
            float *s = sh + step % STEPS * STAGE;
            const int k0 = k_begin + step * BK;
            copy_operand<AK, THREADS>(s, p.A, a_ld, m0, p.M, k0, k_end, a_vec);
            copy_operand<BKC, THREADS>(s + TILE, p.B, b_ld, n0, p.N, k0, k_end, b_vec);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // Sums in pairs: of k (BOTH), of columns, or of rows.
    constexpr bool BOTH = AK && BKC;
    constexpr int PI = !AK && BKC ? TM / 2 : TM, PJ = !BKC ? TN / 2 : TN;
    float2 acc[PI][PJ];
#pragma unroll
    for (int i = 0; i < PI; ++i)
#pragma unroll
        for (int j = 0; j < PJ; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < STEPS - 1; ++i) stage(i);
    for (int step = 0; step < n_steps; ++step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STEPS - 2) : "memory");
        __syncthreads();                                                 // everybody's copies have landed, and nobody reads the step before any more
        stage(step + STEPS - 1);
        const float *As = sh + step % STEPS * STAGE, *Bs = As + TILE;
#pragma unroll 2
        for (int k = kg * (BK / KG); k < (kg + 1) * (BK / KG); k += 4) {
            float a[TM][4], b[TN][4];                                    // [.][k]
            if (AK) {
#pragma unroll
                for (int i = 0; i < TM; ++i) *reinterpret_cast<float4 *>(a[i]) = *reinterpret_cast<const float4 *>(As + (ty + 8 * i) * PITCH_K + k);
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int i = 0; i < TM; i += 4) {
                        const float4 v = *reinterpret_cast<const float4 *>(As + (k + q) * PITCH_M + TM * ty + i);
                        a[i][q] = v.x; a[i + 1][q] = v.y; a[i + 2][q] = v.z; a[i + 3][q] = v.w;
                    }
            }
            if (BKC) {
#pragma unroll
                for (int j = 0; j < TN; ++j) *reinterpret_cast<float4 *>(b[j]) = *reinterpret_cast<const float4 *>(Bs + (tx + 16 * j) * PITCH_K + k);
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 v = *reinterpret_cast<const float4 *>(Bs + (k + q) * PITCH_M + TN * tx);
                    b[0][q] = v.x; b[1][q] = v.y; b[2][q] = v.z; b[3][q] = v.w;
                }
            }
            if constexpr (BOTH) {
#pragma unroll
                for (int q = 0; q < 4; q += 2)
#pragma unroll
                    for (int i = 0; i < TM; ++i)
#pragma unroll
                        for (int j = 0; j < TN; ++j) acc[i][j] = __ffma2_rn(make_float2(a[i][q], a[i][q + 1]), make_float2(b[j][q], b[j][q + 1]), acc[i][j]);
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int i = 0; i < PI; ++i)
#pragma unroll
                        for (int j = 0; j < PJ; ++j) {
                            if constexpr (!BKC) acc[i][j] = __ffma2_rn(make_float2(a[i][q], a[i][q]), make_float2(b[2 * j][q], b[2 * j + 1][q]), acc[i][j]);
                            else acc[i][j] = __ffma2_rn(make_float2(a[2 * i][q], a[2 * i + 1][q]), make_float2(b[j][q], b[j][q]), acc[i][j]);
                        }
            }
        }
    }

    // the tile's sums, in shared memory so that whole rows go out whatever the threads hold; the second group's first
    float *part = sh;                                                    // [64][PITCH_M]
    auto sum = [&](int i, int j) {
        if constexpr (BOTH) return acc[i][j].x + acc[i][j].y;
        else if constexpr (!BKC) return j & 1 ? acc[i][j / 2].y : acc[i][j / 2].x;
        else return i & 1 ? acc[i / 2][j].y : acc[i / 2][j].x;
    };
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int g = KG - 1; g >= 0; --g) {
        if (kg == g) {
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    float *at = part + row_of(i) * PITCH_M + col_of(j);
                    *at = g == KG - 1 ? sum(i, j) : sum(i, j) + *at;
                }
        }
        if (g > 0) __syncthreads();
    }
    if (gridDim.z > 1) cluster_sync();
    else __syncthreads();
    store_tile<THREADS>(p, part, m0, n0);
}

// One operand: element (m, k) at base[m * row + k * col]; KC: contiguous along k.
template <bool KC>
struct Operand {
    static constexpr int PER = BM * BK / GROUP;  // elements of an operand tile per thread
    const float *at;
    long long step;
    int m, k, m_end, k_end;                      // this thread's first element and the ends of the matrix
    __device__ __forceinline__ Operand(const float *base, long long row, long long col, int m0, int k0, int rows, int k_stop)
    {
        const int t = threadIdx.x;
        m = m0 + (KC ? t / BK : t % BM);
        k = k0 + (KC ? t % BK : t / BM);
        at = base + (long long)m * row + (long long)k * col;
        step = KC ? (GROUP / BK) * row : (GROUP / BM) * col;
        m_end = rows; k_end = k_stop;
    }
    __device__ __forceinline__ void load(float (&r)[PER]) const
    {
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const bool on = KC ? (m + i * (GROUP / BK) < m_end && k < k_end) : (m < m_end && k + i * (GROUP / BM) < k_end);
            r[i] = on ? __ldg(at + i * step) : 0.0f;
        }
    }
    __device__ __forceinline__ void next(long long col) { at += BK * col; k += BK; }
    __device__ __forceinline__ static void store(float (*s)[PITCH_M], const float (&r)[PER])
    {
        const int t = threadIdx.x;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int mm = KC ? t / BK + i * (GROUP / BK) : t % BM, kk = KC ? t % BK : t / BM + i * (GROUP / BM);
            s[kk][mm ^ (kk >> 3)] = r[i];
        }
    }
};

// The form for what the kernel above gains nothing on (the rule is in b200_gemm_f32): the next step's operands are in registers under the current
// one's products, two shared-memory buffers, one barrier a step; the transposing stores are spread over the banks by xor-ing k into the low
// bits of the position.
template <bool AK, bool BKC>
__global__ void __launch_bounds__(GROUP, 3) gemm_f32_turning_kernel(const __grid_constant__ b200_gemm_args p, int per_split)
{
    __shared__ __align__(16) float As[2][BK][PITCH_M], Bs[2][BK][PITCH_M];
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
    float ra[Operand<AK>::PER], rb[Operand<BKC>::PER];
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
        for (int e = first * BN + 4 * tid; e < (first + rows) * BN; e += 4 * GROUP) {
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

enum { TURNING, ASYNC, ASYNC_ALONE };
cudaError_t launch_f32(const b200_gemm_args &a, int splits, int per, int form, cudaStream_t st)
{
    typedef void (*Kernel)(const b200_gemm_args, int);
    static const Kernel kernels[3][4] = {                        // rows of A along k: + 2, of B: + 1
        {gemm_f32_turning_kernel<false, false>, gemm_f32_turning_kernel<false, true>, gemm_f32_turning_kernel<true, false>, gemm_f32_turning_kernel<true, true>},
        {gemm_f32_kernel<false, false, 1>, gemm_f32_kernel<false, true, 1>, gemm_f32_kernel<true, false, 1>, nullptr},
        {gemm_f32_kernel<false, false, 4>, gemm_f32_kernel<false, true, 4>, gemm_f32_kernel<true, false, 4>, gemm_f32_kernel<true, true, 4>}};
    const Kernel kern = kernels[form][2 * (a.a_col == 1) + (a.b_row == 1)];
    const int steps = (per + BK - 1) / BK;
    size_t smem = form == TURNING ? 0 : (size_t)(steps < STEPS ? steps : STEPS) * STAGE * sizeof(float);
    if (form == ASYNC_ALONE && smem < 116 * 1024) smem = 116 * 1024;           // no second block beside it
    const cudaError_t set = form == TURNING ? cudaSuccess : cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 116 * 1024);
    if (set != cudaSuccess) return set;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((a.N + BN - 1) / BN, (a.M + BM - 1) / BM, splits);
    cfg.blockDim = dim3(form == ASYNC_ALONE ? 4 * GROUP : GROUP);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 1; at.val.clusterDim.y = 1; at.val.clusterDim.z = splits;
    cfg.attrs = &at;
    cfg.numAttrs = splits > 1;
    return cudaLaunchKernelEx(&cfg, kern, a, per);
}

}  // namespace

extern "C" int b200_gemm_f32(const b200_gemm_args *a, void *stream)
{
    if (!a || !a->A || !a->B || !a->C || a->M <= 0 || a->N <= 0 || a->K <= 0) return B200_E_BADARG;
    if ((a->a_row != 1 && a->a_col != 1) || (a->b_row != 1 && a->b_col != 1)) return B200_E_BADARG;
    // Blocks per tile: up to about four on every SM, as long as each keeps 128 of k. Where that is no more than the SMs, clusters would still put several
    // on one and leave others idle (64 x 1152 x 13824 in 8: half of them): then as many as fit with an SM to each, four groups of threads in
    // it (79 us, 106 before; 64 x 1152 x 6912 41 and 55). Where that is the same number of blocks it pays for a long k that is not along the rows of
    // both operands (64 x 512 x 4096 in 8: 21.3 us and 22.3; along both 22.7 and 20.6; 64 x 512 x 1536 along both 11.6 and 10.1).
    static const int resident[9] = {0, 148, 148, 135, 132, 130, 132, 105, 120};          // clusters of 1 .. 8, a block on an SM
    const long long tiles = (long long)((a->N + BN - 1) / BN) * ((a->M + BM - 1) / BM);
    const bool both = a->a_col == 1 && a->b_row == 1;
    int splits = 1, form = TURNING;
    while (splits < 8 && tiles * splits * 2 <= 148 * 4 && a->K / (splits * 2) >= 128) splits *= 2;
    if (splits > 1 && tiles * splits <= 148 && a->K >= 512) {
        int fit = 0;
        for (int s = 2; s <= 8; ++s)
            if (a->K / s >= 128 && tiles * s <= resident[s]) fit = s;
        if (fit && (fit != splits || (a->K / fit >= 512 && !both))) { splits = fit; form = ASYNC_ALONE; }
    }
    // One block a tile: copies that run ahead pay where waves of tiles follow one another and an operand at least is contiguous along its rows
    // (13824 x 1152 x 64 60 us, 74 turning; one of them along k 70 and 73); with few waves, and in splits of a short k, its longer start costs 5 - 25 %
    // (64 x 1536 x 1152 14.9 us and 13.5, 64 x 1152 x 256 10.6 and 8.8).
    if (splits == 1 && tiles >= 4 * 148 && !both) form = ASYNC;
    const int per = ((a->K + splits - 1) / splits + BK - 1) / BK * BK;
    const cudaError_t rc = launch_f32(*a, splits, per, form, (cudaStream_t)stream);
    ++g_b200_launches;
    return rc != cudaSuccess ? (int)rc : (int)cudaGetLastError();
}
