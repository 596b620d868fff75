// The large products of 16-bit operands on pairs of SMs (sm_100a): C[M,N] = alpha * A[M,K] * B[N,K]^T (+ R), as gemm_tf32.cu
// defines it, for more than 128 rows. b200_gemm_f16 / _bf16 come here when that is modelled faster.
//
// What bounds these products is operand staging: an SM takes in about 58 bytes a clock, and a 128 x 176 tile by itself wants 110
// to keep its tensor core busy. Here two SMs work on a 256 x bn tile (tcgen05 cta_group::2): each loads its own 128 rows of A and
// half of the rows of B, and the tensor cores read the other half from the neighbour's shared memory, so a 256-wide
// tile wants 64. Persistent: a pair walks its tiles, two accumulators in tensor memory take turns, and the epilogue of one
// tile runs under the products of the next.
// Results leave through shared memory (store_block), and the issuing lane counts its places in the ring: stored by the thread that read the row, 16
// bytes in 32 lines, and with a division per ring step, chains of 20 took: 512 x 6144 x 2560 23.7 us, 17.5 now (with an addend 33.6 and 18.9),
// 512 x 2560 x 4096 27.7 and 24.3, 2048 x 2560 x 4096 47.3 and 38.1, 2048 x 12288 x 2048 94 and 85, 512 x 4096 x 512 12.4 and 12.4; bfloat16
// results 777 x 9728 x 512 18.0 and 14.7 (24 with 8 bytes a store).
//
// Pair, per SM: warp 0 loads with TMA (both SMs' copies complete on the barrier of the first, the leader), one lane of the
// leader's warp 1 issues the products for both and commits to both, warps 2-5 store their SM's 128 rows. Products of few tiles are
// split along k over the pairs of one cluster (two to four); each leaves its sums in shared memory and adds up a share of
// the rows, in rank order. (Adding into C one after the other instead: 55 us for 512 x 2560 x 4096, the second pair waits for
// the first one's stores and reads them back.)
// Every wait is bounded; on a timeout the block raises *d_err, lets copies in flight land, frees its tensor memory and returns.
#include "tcgen05.cuh"
#include "gemm_pair.cuh"

#include <cuda_bf16.h>

#include <type_traits>

extern unsigned long long g_b200_launches;

namespace {

constexpr int SM_ROWS = 128;             // rows of A per SM = tensor-memory lanes
constexpr int KB = 64;                   // k of a 128-byte operand row
constexpr int PAIR_THREADS = 192;
constexpr int PAIR_SLOTS = 8;
constexpr int KSUB = 2;                  // operand rows per slot: half the hand-overs
constexpr uint32_t A_TILE = SM_ROWS * KB * 2;
struct PairArgs {
    float *C; long long ldc;
    const float *R; long long ldr;
    __nv_bfloat16 *Ch; long long ldch;
    int M, N, K, bn, slots, splits, tiles_m, tiles, fmt, relu2;
    float alpha;
    unsigned *d_err;
};

// The place in a ring and the phase of the barriers there.
struct Turn {
    int at = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void next(int n) { if (++at == n) { at = 0; phase ^= 1; } }
};

__device__ __forceinline__ uint32_t on_rank(uint32_t addr, uint32_t rank)
{
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    return a;
}
// into this SM's shared memory, completing on a barrier that may be the neighbour's
__device__ __forceinline__ void pair_load(void *dst, const CUtensorMap *map, int x, int y, uint32_t bar)
{
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void pair_umma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void pair_commit(uint64_t *bar, uint32_t leader)       // on the barrier at this place in both SMs
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"((unsigned short)(3u << leader)) : "memory");
}
__device__ __forceinline__ void arrive_at(uint32_t bar)
{
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

// What is stored of a sum: alpha times it, and then what is added (two roundings in every path).
__device__ __forceinline__ float scaled(const PairArgs &p, float v) { return __fmul_rn(p.alpha, v); }

// 32 rows (row0 on, one a lane in r) by 32 columns (n on) of a tile, by one warp: through 2 KB of shared memory, so that a store covers 64 bytes of
// eight rows and not 16 of 32, and what is added is read so; fp32 in two halves of 16 columns, bfloat16 packed first. The 16-byte pieces of a row are
// exchanged by the row's number: eight lanes meet all banks both ways. The unusual paths are loops, every launch fetches this code anew. Against whole
// lines of four rows (4 KB) it leaves a ring slot more to tiles 176 wide, and 600 products of M 192 .. 2048, N 512 .. 12288, K 256 .. 9728 take
// 1 % (C), 3 % (C + R) less.
__device__ __forceinline__ void store_block(const PairArgs &p, uint4 *stage, int row0, int n, int n_end, const uint32_t *r, bool vec)
{
    const int lane = threadIdx.x & 31, c = lane & 3, r0 = lane >> 2;
    auto piece = [&](int row, int k) { return stage + row * 4 + (k ^ ((row >> 1) & 3)); };
    if (p.Ch) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            uint32_t w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float x = __uint_as_float(r[8 * k + 2 * j]), y = __uint_as_float(r[8 * k + 2 * j + 1]);
                const __nv_bfloat162 h = __floats2bfloat162_rn(p.alpha * (p.relu2 ? act_relu2(x) : x), p.alpha * (p.relu2 ? act_relu2(y) : y));
                w[j] = *reinterpret_cast<const uint32_t *>(&h);
            }
            *piece(lane, k) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        __syncwarp();
        n += 8 * c;
        __nv_bfloat16 *h = p.Ch + (long long)(row0 + r0) * p.ldch + n;
        if (n + 8 <= n_end) {
            uint4 v[4];                                      // all of them before the first store, which might alias
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = *piece(8 * i + r0, c);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (row0 + 8 * i + r0 < p.M) *reinterpret_cast<uint4 *>(h + (long long)(8 * i) * p.ldch) = v[i];
        } else {
#pragma unroll 1
            for (int i = 0; i < 4 && row0 + 8 * i + r0 < p.M; ++i)
#pragma unroll 1
                for (int j = 0; n + j < n_end; ++j) h[(long long)(8 * i) * p.ldch + j] = reinterpret_cast<const __nv_bfloat16 *>(piece(8 * i + r0, c))[j];
        }
        __syncwarp();
        return;
    }
    n += 4 * c;
    float4 add[8];
    if (p.R && vec) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int row = row0 + 8 * (k & 3) + r0, col = n + 16 * (k >> 2);
            add[k] = row < p.M && col + 4 <= n_end ? __ldcg(reinterpret_cast<const float4 *>(p.R + (long long)row * p.ldr + col)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
#pragma unroll
    for (int half = 0; half < 2; ++half, n += 16) {
#pragma unroll
        for (int k = 0; k < 4; ++k) *piece(lane, k) = make_uint4(r[16 * half + 4 * k], r[16 * half + 4 * k + 1], r[16 * half + 4 * k + 2], r[16 * half + 4 * k + 3]);
        __syncwarp();
        if (vec && n + 4 <= n_end) {
            float4 v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = *reinterpret_cast<const float4 *>(piece(8 * i + r0, c));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = row0 + 8 * i + r0;
                v[i] = make_float4(scaled(p, v[i].x), scaled(p, v[i].y), scaled(p, v[i].z), scaled(p, v[i].w));
                if (p.R) { const float4 q = add[4 * half + i]; v[i].x += q.x; v[i].y += q.y; v[i].z += q.z; v[i].w += q.w; }
                if (row < p.M) *reinterpret_cast<float4 *>(p.C + (long long)row * p.ldc + n) = v[i];
            }
        } else {
#pragma unroll 1
            for (int i = 0; i < 4; ++i) {
                const int row = row0 + 8 * i + r0;
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (row < p.M && n + j < n_end) {
                        float v = scaled(p, reinterpret_cast<const float *>(piece(8 * i + r0, c))[j]);
                        if (p.R) v += __ldcg(p.R + (long long)row * p.ldr + n + j);
                        p.C[(long long)row * p.ldc + n + j] = v;
                    }
            }
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(PAIR_THREADS)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ PairArgs p)
{
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full_bar[PAIR_SLOTS], empty_bar[PAIR_SLOTS], done_bar[2], free_bar[2];
    __shared__ uint32_t tmem_base_sh;
    __shared__ int abort_sh;
    uint8_t *ring = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);          // (an offset: accesses stay known as shared ones)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = blockIdx.x & 1;
    const int split = (int)(blockIdx.x >> 1) % p.splits;                 // clusters hold the splits of a tile
    const uint32_t leader = 2 * split;
    const int first = (int)(blockIdx.x >> 1) / p.splits, stride = (int)(gridDim.x >> 1) / p.splits;
    const uint32_t B_TILE = (uint32_t)p.bn / 2 * KB * 2, SLOT = (A_TILE + B_TILE) * KSUB;
    const int nkb_all = (p.K + KB * KSUB - 1) / (KB * KSUB), per = (nkb_all + p.splits - 1) / p.splits;
    const int kb0 = split * per, nkb = min(per, nkb_all - kb0);
    volatile int *abort_flag = &abort_sh;

    if (threadIdx.x == 0) {
        abort_sh = 0;
        for (int s = 0; s < p.slots; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(&done_bar[a], 1); mbar_init(&free_bar[a], 8); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();                                             // the neighbour's barriers exist
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_sh;
    auto give_up = [&](unsigned code) { if (!*abort_flag) { *abort_flag = 1; if (p.d_err) atomicExch(p.d_err, code); } };

    // a pair (with splits: a cluster, which has one) takes every stride-th tile
    if (warp == 0) {
        if (lane == 0) {
            Turn t;                                          // places and phases are counted: a division a step would be on the critical path
            for (int tile = first; tile < p.tiles && !*abort_flag; tile += stride) {
                const int m0 = tile % p.tiles_m * 2 * SM_ROWS + (int)rank * SM_ROWS, n0 = tile / p.tiles_m * p.bn + (int)rank * (p.bn / 2);
                for (int kb = 0; kb < nkb; ++kb, t.next(p.slots)) {
                    const int s = t.at;
                    if (!wait_or_abort(&empty_bar[s], t.phase ^ 1, abort_flag)) { give_up(0x7301u); break; }
                    uint8_t *a = ring + (size_t)s * SLOT, *b = a + (size_t)A_TILE * KSUB;
                    const uint32_t bar = on_rank(smem_u32(&full_bar[s]), leader);
                    if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * SLOT);
#pragma unroll
                    for (int q = 0; q < KSUB; ++q) {
                        const int x = ((kb0 + kb) * KSUB + q) * KB;
                        pair_load(a + (size_t)q * A_TILE, &map_a, x, m0, bar);
                        pair_load(b + (size_t)q * B_TILE, &map_b, x, n0, bar);
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            const uint32_t idesc = (1u << 4) | ((uint32_t)p.fmt << 7) | ((uint32_t)p.fmt << 10) | ((uint32_t)(p.bn >> 3) << 17) | (16u << 24);
            Turn u;
            int t = 0;
            for (int tile = first; tile < p.tiles && !*abort_flag; tile += stride, ++t) {
                const int acc = t & 1;
                if (!wait_or_abort(&free_bar[acc], ((t >> 1) & 1) ^ 1, abort_flag)) { give_up(0x7305u); break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                bool ok = true;
                for (int kb = 0; kb < nkb; ++kb, u.next(p.slots)) {
                    const int s = u.at;
                    if (!wait_or_abort(&full_bar[s], u.phase, abort_flag)) { give_up(0x7302u); ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a = smem_u32(ring + (size_t)s * SLOT), b = a + A_TILE * KSUB;
#pragma unroll
                    for (int q = 0; q < KSUB; ++q) {
                        const uint64_t ad = smem_desc_sw128(a + q * A_TILE), bd = smem_desc_sw128(b + q * B_TILE);
#pragma unroll
                        for (int j = 0; j < 4; ++j) pair_umma(tmem_base + acc * 256, ad + 2 * j, bd + 2 * j, idesc, (kb | q | j) != 0);
                    }
                    pair_commit(&empty_bar[s], leader);
                }
                if (!ok) break;
                pair_commit(&done_bar[acc], leader);
            }
        }
    } else {
        const int quad = warp & 3;
        uint4 *stage = reinterpret_cast<uint4 *>(ring + (size_t)p.slots * SLOT);
        const bool vec = ((p.ldc & 3) == 0) && ((reinterpret_cast<uintptr_t>(p.C) & 15) == 0) &&
                         (!p.R || (((p.ldr & 3) == 0) && ((reinterpret_cast<uintptr_t>(p.R) & 15) == 0)));
        int t = 0;
        for (int tile = first; tile < p.tiles; tile += stride, ++t) {
            const int acc = t & 1;
            const int row0 = tile % p.tiles_m * 2 * SM_ROWS + (int)rank * SM_ROWS + quad * 32, n0 = tile / p.tiles_m * p.bn;
            const bool ok = __all_sync(0xffffffffu, wait_or_abort(&done_bar[acc], (t >> 1) & 1, abort_flag));
            if (!ok) { if (lane == 0) give_up(0x7303u); break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int n_end = min(p.N, n0 + p.bn);
#pragma unroll 1
            for (int c = 0; n0 + c < n_end; c += 32) {
                uint32_t r[32];
                tmem_ld32(tmem_base + ((uint32_t)quad << 21) + (uint32_t)(acc * 256 + c), r);
                if (p.splits > 1) {
                    // rows bn + 4 floats apart: 16-byte stores of eight rows fall on 32 banks
                    float *part = reinterpret_cast<float *>(ring) + (quad * 32 + lane) * (p.bn + 4) + c;
#pragma unroll
                    for (int j = 0; j < 32; j += 4)
                        if (c + j < p.bn)
                            *reinterpret_cast<float4 *>(part + j) = make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]),
                                                                                __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3]));
                } else store_block(p, stage + (warp - 2) * 128, row0, n0 + c, n_end, r, vec);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) arrive_at(on_rank(smem_u32(&free_bar[acc]), leader));
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (p.splits > 1) {                                      // one tile: first
        cluster_sync();                                         // the sums of all splits lie in shared memory
        const int n0 = first / p.tiles_m * p.bn, cols = min(p.N - n0, p.bn), share = SM_ROWS / p.splits;
        const int r0 = split * share, r1 = split + 1 == p.splits ? SM_ROWS : r0 + share;
        const int m0 = first % p.tiles_m * 2 * SM_ROWS + (int)rank * SM_ROWS;
        const uint32_t part = smem_u32(ring);
        const bool vec = ((p.ldc & 3) == 0) && ((reinterpret_cast<uintptr_t>(p.C) & 15) == 0);
        auto add_up = [&](auto with) {                       // (apart: the loop without an addend stays as short as it is)
            constexpr bool ADD = decltype(with)::value;
            for (int r = r0 + warp; r < r1 && m0 + r < p.M && !*abort_flag; r += PAIR_THREADS / 32) {
                float *c = p.C + (long long)(m0 + r) * p.ldc + n0;
                const float *q = ADD ? p.R + (long long)(m0 + r) * p.ldr + n0 : nullptr;
#pragma unroll 2
                for (int n = 4 * lane; n < cols; n += 128) {
                    float add[4] = {};
                    if (ADD) {                               // on their way under the sums of the other splits
#pragma unroll
                        for (int j = 0; j < 4; ++j) add[j] = n + j < cols ? __ldcg(q + n + j) : 0.0f;
                    }
                    const float4 s4 = sum_ranks4(part + (uint32_t)(r * (p.bn + 4) + n) * 4, p.splits, rank, 2);
                    float f[4] = {scaled(p, s4.x), scaled(p, s4.y), scaled(p, s4.z), scaled(p, s4.w)};
                    if (ADD) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) f[j] += add[j];
                    }
                    if (vec && n + 4 <= cols) *reinterpret_cast<float4 *>(c + n) = make_float4(f[0], f[1], f[2], f[3]);
                    else {
#pragma unroll 1
                        for (int j = 0; j < 4; ++j)
                            if (n + j < cols) c[n + j] = j == 0 ? f[0] : j == 1 ? f[1] : j == 2 ? f[2] : f[3];
                    }
                }
            }
        };
        if (p.R) add_up(std::true_type{});
        else add_up(std::false_type{});
        cluster_sync();                                      // nobody leaves while its sums are read
    }
    if (*abort_flag)
        for (int i = 0; i < 200; ++i) __nanosleep(1000);     // copies in flight land before the memory is released
    cluster_sync();                                             // the neighbour is done with this SM's memory
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

}  // namespace

// Tile width and split: the least modelled time. A step of 64 of k takes 2 clocks a column of products or its operand bytes
// at 58 a clock, whichever is more; the last epilogue is not hidden (some 20 clocks a column), and sums of splits go
// through shared memory. The width is a multiple of 16 up to 256. CLUSTERS: how many clusters of 2, 4, 6, 8 blocks are resident
// on 148 SMs (the occupancy calculator's figures).
// What comes back is held against the form of one SM per tile: clocks of the shape taken, fitted to 200 products (M 129 .. 2048, N 256 .. 19456,
// K 256 .. 16384, chains of 20 launches) when the thread that read a row stored it, 8 % rms then; times have come down since (store_block), those of
// a short k most, so that pairs are taken a little late. Left as they are: narrower tiles in fewer splits would be up to 10 % faster (512 x 2560 x
// 4096 24 us in two, 22 in one), but their accumulators take twice the additions, which the tensor cores truncate.
double gemm_pair_shape(int M, int N, int K, bool may_split, PairShape *out)
{
    if (M <= SM_ROWS || N < 256) return 1e30;
    const int pairs = tc_sm_count() / 2, mt = (M + 2 * SM_ROWS - 1) / (2 * SM_ROWS), nkb = (K + KB - 1) / KB;
    constexpr int CLUSTERS[5] = {0, 74, 33, 22, 15};
    double least = 1e30, clocks = 1e30;
    for (int bn = 64; bn <= 256; bn += 16) {
        const long long tiles = (long long)mt * ((N + bn - 1) / bn);
        double step = 2.0 * bn;
        if (step < (A_TILE + bn * 64.0) / 58.0) step = (A_TILE + bn * 64.0) / 58.0;
        for (int s = 1; s <= 4; ++s) {
            if (s > 1 && (!may_split || nkb / s < 8)) break;
            const long long place = (long long)CLUSTERS[s] * pairs / 74, waves = (tiles + place - 1) / place;
            if (s > 1 && waves > 1) break;
            const double steps = waves * ((nkb + s - 1) / s) * step, cost = steps + 1500.0 + bn * 20.0 + (s > 1 ? 1500.0 + bn * 15.0 : 0.0);
            if (cost < least) {
                least = cost; out->bn = bn; out->splits = s;
                clocks = 1.32 * steps + 3450.0 * waves + 3250.0 + bn * 74.0 + (s > 1 ? 3450.0 + bn * 43.0 : 0.0);
            }
        }
    }
    return clocks;
}

int gemm_pair_launch(const b200_gemm_args *a, int fmt, const PairShape &sh, cudaStream_t st)
{
    PairArgs p = {};
    p.C = a->C; p.ldc = a->ldc; p.R = a->R; p.ldr = a->ldr;
    p.Ch = static_cast<__nv_bfloat16 *>(a->Ch); p.ldch = a->ldch;
    p.M = a->M; p.N = a->N; p.K = a->K; p.bn = sh.bn; p.splits = sh.splits; p.fmt = fmt; p.relu2 = a->relu2;
    p.alpha = a->alpha; p.d_err = a->d_err;
    p.tiles_m = (a->M + 2 * SM_ROWS - 1) / (2 * SM_ROWS);
    p.tiles = p.tiles_m * ((a->N + p.bn - 1) / p.bn);
    const size_t slot = (size_t)(A_TILE + p.bn * 64) * KSUB;
    // a split without a step would have nothing to commit: as many as there are slots of k for
    const int nkb = (a->K + KB * KSUB - 1) / (KB * KSUB);
    while (p.splits > 1 && (p.splits - 1) * ((nkb + p.splits - 1) / p.splits) >= nkb) --p.splits;
    // of 227 KB: barriers (512 bytes), alignment, and 2 KB a storing warp for results on their way out; none for splits, whose sums lie in the ring
    const size_t stage = p.splits > 1 ? 0 : 4 * 2048;
    p.slots = (int)((227 * 1024 - 512 - 1024 - stage) / slot);
    if (p.slots > PAIR_SLOTS) p.slots = PAIR_SLOTS;
    const size_t smem = slot * p.slots + stage + 1024;
    CUtensorMap ma, mb;
    const CUtensorMapDataType type = fmt ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    if (!tc_make_map(&ma, a->A, a->M, a->K, a->a_row * 2, KB, SM_ROWS, type)) return B200_E_UNSUPPORTED;
    if (!tc_make_map(&mb, a->B, a->N, a->K, a->b_col * 2, KB, p.bn / 2, type)) return B200_E_UNSUPPORTED;
    cudaError_t rc = cudaFuncSetAttribute(gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (rc != cudaSuccess) return (int)rc;
    const int pairs = tc_sm_count() / 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (p.splits > 1 ? p.tiles * p.splits : p.tiles < pairs ? p.tiles : pairs));
    cfg.blockDim = dim3(PAIR_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 2 * p.splits; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    rc = cudaLaunchKernelEx(&cfg, gemm_pair_kernel, ma, mb, p);
    if (rc != cudaSuccess) return (int)rc;
    ++g_b200_launches;
    return (int)cudaGetLastError();
}
