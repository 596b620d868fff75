// Rows of activations times a packed weight matrix, C[m][n] = (x_m . w_n) (+ R[m][n]), on the tensor cores with fp32 operands and sums
// (sm_100a): prompts, and sequences that advance together.
//
// The weights are the M side of the tile (128 weight rows, tcgen05 M = 128), the activation rows its N side (16..128, a multiple
// of 16), so a few activation rows cost a few columns and not a padded tile of 128. fp32 operands are sums of binary16 planes:
//   * an activation row is scaled by a power of two (largest element in [2^14, 2^15)) and split into one or two planes
//     (b200_rows_norm_planes and its relatives write them); two planes hold 22 bits of an element down to 2^-16 of the largest, 2^-39
//     of the largest below;
//   * a Q8_0 weight is scale x int8, at most 11 + 7 bits. It is made in the kernel: hi = rn(d q), lo = d q - hi by one binary16
//     fused multiply-add, exact; d carries a power of two of the row, so nothing of the row's large elements underflows.
//     Products: hi x0 + lo x0 + hi x1 (what is left out is 2^-22 of a term). F16 weights: w x0 + w x1.
// The accumulators are fp32 in tensor memory; the epilogue takes the powers of two out again.
// The tensor cores truncate what they add to an accumulator, always towards zero: a sum through one accumulator loses 1.4e-7 of itself per
// 64 columns (F16; 2.2e-7 Q8_0). So an accumulator takes the products of 64 columns only, corrections first, and warps of their own add it
// to fp32 sums in registers, rounding, while the next step fills another one: two to four go round. Against float64 that is 1.3e-7 ..
// 2.6e-7 of a result at 512 .. 9728 columns, where the per-token kernels' fp32 sums are 0.8e-7 .. 1.2e-7 off and up to three accumulators of
// 256 additions each, without drains, were 0.3e-6 .. 5e-6. Every second step would be 3e-7 .. 4e-7. One plane: a single chain, 1e-6 .. 1e-5 beside
// the 2e-4 of its rounded operand.
// Measured, two planes, drained every step and before (three accumulators): Q8_0 19456 x 2560, 48 / 512 / 1531 rows 53 / 209 / 518 us and
// 51 / 224 / 569; F16 42 / 133 / 302 and 38 / 122 / 291: bound by operand staging (48 KB a step of a 128-column tile at 52 bytes a clock) and the
// wait of two blocks on an SM with two accumulators each for their drains.
//
// Block: warp 0 fills the ring with TMA (activation planes; F16 weight tiles), one lane of warp 1 issues tcgen05.mma, the last four
// warps (eight in the wide Q8_0 form, half of the columns each) drain the accumulators and store the result. What the issuing lane does between
// two steps is on the critical path: places and phases are counted, not divided (0.2 us a step otherwise).
// Q8_0: the four warps of a team make the weight tile of a step in tensor memory, where the products read it as their A operand, 32 rows
// each (a thread its row); two teams take turns in the wide form. A warp copies its rows' 64 bytes and scales to shared memory
// several of its steps ahead (cp.async, four lanes a row; nobody else reads them: no barrier), and stores the two planes with
// tcgen05.st. binary16 arithmetic on pairs makes that two instructions an element. Through shared memory the planes would cost 256
// cycles of its bandwidth to write and 384 to read per step, beside 256 .. 768 of products; with register prefetch instead of cp.async a
// step took 3000 cycles.
// Few tiles: the blocks of a cluster share one along k, leave their sums in shared memory and each adds up a share of the
// columns, in rank order (deterministic, nothing goes through HBM).
//
// Every wait is bounded; on a timeout the block raises *d_err, joins the cluster's barriers and returns.
#include "stream_core.cuh"
#include "tcgen05.cuh"
#include "../../include/llmb200_train_kernels.h"

extern unsigned long long g_b200_launches;

namespace {

constexpr int WM = 128;                  // weight rows of a tile = TMEM lanes
constexpr int KB = 64;                   // columns per ring slot = one 128-byte swizzle row of binary16
constexpr int MAX_ACC = 4;
constexpr uint32_t RAW_WARP = 32 * 68;    // quants (64 bytes a row) and scales (4) of a warp's 32 rows and a step
constexpr int MAX_SLOTS = 8;
constexpr uint32_t W_TILE = WM * KB * 2;

struct RowsMat {
    const uint8_t *w; long long w_stride;
    const float *w_scale, *x_scale;
    int rows, cols, n, planes, plane_rows;
    float *out; long long out_ld;
    const float *resid; long long resid_ld;
    unsigned *d_err;
    int bn, slots, tmem_cols, splits;
    int acc_cols, n_acc, every;          // accumulators that go round: columns between them, how many, and the steps that one takes
};

__device__ __forceinline__ void cp_async(uint32_t dst, const void *src, int bytes_on)      // 16 bytes, zeros unless on
{
    asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes_on) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void *src, int bytes_on)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes_on) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t *r)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
// A from tensor memory: lane = row, two elements of k per column
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t acc)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(acc) : "memory");
}

// Four int8 weights times d as two planes of binary16 pairs.
__device__ __forceinline__ void q8_planes(uint32_t u, __half2 d, uint32_t *hi, uint32_t *lo)
{
    const uint32_t b = u ^ 0x80808080u;
    const __half2 bias = __half2half2(__ushort_as_half(0x6480));          // 1152: 1024 (the bytes' exponent) + 128
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const uint32_t p = __byte_perm(b, 0x64646464u, i ? 0x4342u : 0x4140u);
        const __half2 q = __hsub2(*reinterpret_cast<const __half2 *>(&p), bias);
        const __half2 vh = __hmul2(d, q), vl = __hfma2(d, q, __hneg2(vh));
        hi[i] = *reinterpret_cast<const uint32_t *>(&vh);
        lo[i] = *reinterpret_cast<const uint32_t *>(&vl);
    }
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t *r)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// The forms of the kernel. F16 weights: tiles of up to 128 columns, one or two blocks on an SM; of up to 32 with a third of the registers, so that
// the kernels before and behind find room beside them (a batch's steps are chains of short launches: 0.49 and 0.53 ms a step).
// Q8_0: a block with eight warps for the weight tiles and eight that drain has an SM to itself; tiles of up to 64 columns take half
// of both and run two on an SM.
enum Form { F16_WIDE, F16_NARROW, Q8_WIDE, Q8_NARROW };
constexpr int form_bn(Form f) { return f == F16_NARROW ? 32 : f == Q8_NARROW ? 64 : 128; }
template <Form F> struct Shape_of {
    static constexpr bool q8 = F == Q8_WIDE || F == Q8_NARROW;
    static constexpr int max_bn = form_bn(F);
    static constexpr int teams = F == Q8_WIDE ? 2 : 1;                   // of four warps that make weight tiles, in turns
    static constexpr int depth = F == Q8_WIDE ? 3 : 6;                   // of a team's steps that are on their way into shared memory
    static constexpr int drain_warps = F == Q8_WIDE ? 8 : 4, drain_cols = max_bn * 4 / drain_warps;
    static constexpr int first_drain = 2 + (q8 ? 4 * teams : 0), threads = 32 * (first_drain + drain_warps);
    static constexpr uint32_t raw = q8 ? 4 * teams * RAW_WARP : 0;       // bytes of a step of every team
};

// The place in a ring and the phase of the barriers there.
struct Turn {
    int at = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void next(int n) { if (++at == n) { at = 0; phase ^= 1; } }
};

template <Form F>
__global__ void __launch_bounds__(Shape_of<F>::threads, F == Q8_WIDE ? 1 : 2)
rows_matmul_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ RowsMat p)
{
    using Of = Shape_of<F>;
    constexpr bool Q8 = Of::q8;
    constexpr uint32_t W_SLOT = Q8 ? 0 : W_TILE, RAW = Of::raw;
    constexpr int DRAIN_WARPS = Of::drain_warps, DRAIN_COLS = Of::drain_cols, FIRST_DRAIN = Of::first_drain, TEAMS = Of::teams, DEPTH = Of::depth;
    constexpr int LEAVE = (FIRST_DRAIN - 2 + DRAIN_WARPS) * 32;          // builders and drains of a shared tile
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full_bar[MAX_SLOTS], empty_bar[MAX_SLOTS], full_acc[MAX_ACC], free_acc[MAX_ACC];
    __shared__ uint32_t tmem_base_sh;
    __shared__ int abort_sh;
    __shared__ float xs_sh[Of::max_bn];
    uint8_t *ring = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int BN = p.bn, slots = p.slots;
    const uint32_t X_TILE = (uint32_t)BN * KB * 2, SLOT = W_SLOT + X_TILE * p.planes;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.x * BN, m0 = blockIdx.y * WM;
    const int nkb_all = (p.cols + KB - 1) / KB, per = (nkb_all + p.splits - 1) / p.splits;
    const int kb0 = blockIdx.z * per, nkb = max(0, min(per, nkb_all - kb0));     // 0: this block only adds zeros
    volatile int *abort_flag = &abort_sh;

    if (threadIdx.x == 0) {
        abort_sh = 0;
        for (int s = 0; s < slots; ++s) { mbar_init(&full_bar[s], 1 + (Q8 ? 4 : 0)); mbar_init(&empty_bar[s], 1); }
        for (int a = 0; a < p.n_acc; ++a) { mbar_init(&full_acc[a], 1); mbar_init(&free_acc[a], DRAIN_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base_sh)), "r"((uint32_t)p.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_sh;
    pdl_launch_dependents();
    auto give_up = [&](unsigned code) { if (!*abort_flag) { *abort_flag = 1; if (p.d_err) atomicExch(p.d_err, code); } };

    if (warp == 0) {
        if (lane == 0) {
            // weights do not depend on earlier kernels: the first slots' tiles are asked for before the wait
            const int ahead = Q8 ? 0 : min(slots, nkb);
            for (int kb = 0; kb < ahead; ++kb) {
                mbar_expect_tx(&full_bar[kb], SLOT);
                tma_load_2d(ring + (size_t)kb * SLOT, &map_w, (kb0 + kb) * KB, m0, &full_bar[kb]);
            }
            pdl_wait();
            Turn t;
            for (int kb = 0; kb < nkb; ++kb, t.next(slots)) {
                const int s = t.at;
                if (!wait_or_abort(&empty_bar[s], t.phase ^ 1, abort_flag)) { give_up(0x7201u); break; }
                uint8_t *dst = ring + (size_t)s * SLOT;
                const int x = (kb0 + kb) * KB;
                if (kb >= ahead) {
                    mbar_expect_tx(&full_bar[s], Q8 ? X_TILE * p.planes : SLOT);
                    if (!Q8) tma_load_2d(dst, &map_w, x, m0, &full_bar[s]);
                }
                for (int u = 0; u < p.planes; ++u)
                    tma_load_2d(dst + W_SLOT + u * X_TILE, &map_x, x, u * p.plane_rows + n0, &full_bar[s]);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // D fp32, A and B binary16, both K-major, N = BN, M = 128
            const uint32_t idesc = (1u << 4) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(WM >> 4) << 24);
            Turn t, acc;
            uint32_t on = 0;                                              // steps that the accumulator holds: the first one starts from zero
            for (int kb = 0; kb < nkb; ++kb, t.next(slots)) {
                const int s = t.at, a = acc.at;
                if (!on && !wait_or_abort(&free_acc[a], acc.phase ^ 1, abort_flag)) { give_up(0x7205u); break; }
                if (!wait_or_abort(&full_bar[s], t.phase, abort_flag)) { give_up(0x7202u); break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t wa = smem_u32(ring + (size_t)s * SLOT), xa = wa + W_SLOT, d = tmem_base + (uint32_t)a * p.acc_cols;
                const uint64_t x0 = smem_desc_sw128(xa), x1 = smem_desc_sw128(xa + X_TILE);
                if constexpr (Q8) {
                    const uint32_t hi = tmem_base + (uint32_t)p.n_acc * p.acc_cols + (uint32_t)s * 64, lo = hi + 32;
#pragma unroll
                    for (int j = 0; j < 4; ++j) umma_f16_ts(d, lo + 8 * j, x0 + 2 * j, idesc, on | (j > 0));
                    if (p.planes == 2) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) umma_f16_ts(d, hi + 8 * j, x1 + 2 * j, idesc, 1);
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) umma_f16_ts(d, hi + 8 * j, x0 + 2 * j, idesc, 1);
                } else {
                    const uint64_t wd = smem_desc_sw128(wa);
                    if (p.planes == 2) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) umma_f16(d, wd + 2 * j, x1 + 2 * j, idesc, on | (j > 0));
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) umma_f16(d, wd + 2 * j, x0 + 2 * j, idesc, on | (p.planes == 2 || j > 0));
                }
                umma_commit(&empty_bar[s]);
                if (++on == (uint32_t)p.every || kb == nkb - 1) { umma_commit(&full_acc[a]); acc.next(p.n_acc); on = 0; }
            }
        }
    } else if (warp < FIRST_DRAIN) {
        if constexpr (Q8) {
            const int quad = warp & 3, turn = (warp - 2) >> 2, row = m0 + quad * 32 + lane, nblk = p.cols / 32;
            const float up = row < p.rows ? 1.0f / p.w_scale[row] : 0.0f;             // a power of two
            const uint32_t raw = smem_u32(ring + (size_t)slots * SLOT) + (uint32_t)(warp - 2) * RAW_WARP;
            // 16-byte chunk c of row r lies at r * 64 + (c ^ (r / 2 % 4)) * 16: reads of a chunk by 32 rows are conflict-free
            auto fetch = [&](int kb, int slot) {
                const uint32_t dst = raw + (uint32_t)slot * RAW;
                const int b = (kb0 + kb) * 2, c = lane & 3;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int r = i * 8 + (lane >> 2), m = m0 + quad * 32 + r;
                    const int on = kb < nkb && m < p.rows && b + (c >> 1) < nblk;
                    cp_async(dst + r * 64 + ((c ^ (r >> 1)) & 3) * 16, on ? p.w + (long long)m * p.w_stride + (size_t)b * 32 + c * 16 : p.w, on ? 16 : 0);
                }
                // the scales of both blocks: one aligned word; where there is no second block its half is padding that nobody writes
                const int on = kb < nkb && row < p.rows;
                cp_async4(dst + 2048 + lane * 4, on ? p.w + (long long)row * p.w_stride + p.cols + b * 2 : p.w, on ? 4 : 0);
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            for (int i = 0; i < DEPTH; ++i) fetch(turn + TEAMS * i, i);
            bool ok = true;
            Turn t;
            for (int i = 0; i < turn; ++i) t.next(slots);
            for (int kb = turn, slot = 0; kb < nkb; kb += TEAMS, slot = slot + 1 == DEPTH ? 0 : slot + 1) {
                const int s = t.at;
                const uint32_t phase = t.phase;
#pragma unroll
                for (int i = 0; i < TEAMS; ++i) t.next(slots);
                asm volatile("cp.async.wait_group %0;" ::"n"(DEPTH - 1) : "memory");
                __syncwarp();
                const uint32_t src = raw + (uint32_t)slot * RAW;
                uint4 q[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) q[c] = lds_128(src + lane * 64 + ((c ^ (lane >> 1)) & 3) * 16);
                const uint32_t sc[2] = {lds_u16(src + 2048 + lane * 4), (kb0 + kb) * 2 + 1 < nblk ? lds_u16(src + 2048 + lane * 4 + 2) : 0u};
                __syncwarp();
                fetch(kb + TEAMS * DEPTH, slot);
                ok = wait_or_abort(&empty_bar[s], phase ^ 1, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) { if (lane == 0) give_up(0x7204u); break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t at = tmem_base + ((uint32_t)quad << 21) + (uint32_t)p.n_acc * p.acc_cols + (uint32_t)s * 64;
#pragma unroll
                for (int blk = 0; blk < 2; ++blk) {
                    const __half2 d = __float2half2_rn(__half2float(__ushort_as_half((unsigned short)sc[blk])) * up);
                    const uint32_t w[8] = {q[2 * blk].x, q[2 * blk].y, q[2 * blk].z, q[2 * blk].w,
                                           q[2 * blk + 1].x, q[2 * blk + 1].y, q[2 * blk + 1].z, q[2 * blk + 1].w};
                    uint32_t hi[16], lo[16];
#pragma unroll
                    for (int c = 0; c < 8; ++c) q8_planes(w[c], d, hi + 2 * c, lo + 2 * c);
                    tmem_st16(at + blk * 16, hi);
                    tmem_st16(at + 32 + blk * 16, lo);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&full_bar[s]);
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            if (p.splits > 1) named_barrier(2, LEAVE);       // the sums below may lie where these copies went
        }
    } else {
        const int quad = warp & 3, r = quad * 32 + lane, row = m0 + r, c0 = (warp - FIRST_DRAIN) / 4 * DRAIN_COLS;
        constexpr int LOAD = F == F16_WIDE ? 32 : 16;           // columns a load: as registers allow
        float sum[DRAIN_COLS];
#pragma unroll
        for (int j = 0; j < DRAIN_COLS; ++j) sum[j] = 0.0f;
        bool ok = true;
        Turn t;
        for (int kb = 0; kb < nkb; kb += p.every, t.next(p.n_acc)) {
            const int a = t.at;
            ok = __all_sync(0xffffffffu, wait_or_abort(&full_acc[a], t.phase, abort_flag));
            if (!ok) { if (lane == 0) give_up(0x7203u); break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t at = tmem_base + ((uint32_t)quad << 21) + (uint32_t)(a * p.acc_cols + c0);
#pragma unroll
            for (int c = 0; c < DRAIN_COLS; c += LOAD)
                if (c0 + c < BN) {
                    uint32_t u[LOAD];
                    if constexpr (LOAD == 32) tmem_ld32(at + c, u);
                    else tmem_ld16(at + c, u);
#pragma unroll
                    for (int j = 0; j < LOAD; j += 2) add_pair(sum[c + j], sum[c + j + 1], __uint_as_float(u[j]), __uint_as_float(u[j + 1]));
                }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&free_acc[a]);
        }
        pdl_wait();
        for (int i = threadIdx.x - FIRST_DRAIN * 32; i < BN; i += DRAIN_WARPS * 32) xs_sh[i] = p.x_scale && n0 + i < p.n ? p.x_scale[n0 + i] : 1.0f;
        named_barrier(1, DRAIN_WARPS * 32);
        if (Q8 && p.splits > 1) named_barrier(2, LEAVE);
        const float ws = Q8 && row < p.rows ? p.w_scale[row] : 1.0f;
        const int cols = min(BN, p.n - n0);
        if (!ok) {
        } else if (p.splits > 1) {
            float *part = reinterpret_cast<float *>(ring);              // [BN][128]
#pragma unroll
            for (int c = 0; c < DRAIN_COLS; ++c)
                if (c0 + c < cols) part[(c0 + c) * WM + r] = sum[c] * ws * xs_sh[c0 + c];
        } else if (row < p.rows) {
            float *o = p.out + (long long)(n0 + c0) * p.out_ld + row;
            const float *q = p.resid ? p.resid + (long long)(n0 + c0) * p.resid_ld + row : nullptr;
#pragma unroll
            for (int c = 0; c < DRAIN_COLS; ++c)
                if (c0 + c < cols) {
                    float f = sum[c] * ws * xs_sh[c0 + c];
                    if (q) f += __ldcg(q + (long long)c * p.resid_ld);
                    o[(long long)c * p.out_ld] = f;
                }
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (p.splits > 1) {
        pdl_wait();                                                     // every thread reads and stores below
        cluster_sync();                                                 // every block's sums lie in its shared memory
        const int cols = min(BN, p.n - n0), share = (cols + p.splits - 1) / p.splits;
        const int c0 = blockIdx.z * share, c1 = min(c0 + share, cols), row = m0 + 4 * lane;
        const uint32_t part = smem_u32(ring);
        const bool vec = row + 4 <= p.rows && (p.out_ld & 3) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
        for (int c = c0 + warp; c < c1 && !*abort_flag; c += blockDim.x / 32) {
            const float4 q = sum_ranks4(part + (uint32_t)(c * WM + 4 * lane) * 4, p.splits, 0, 1);
            float v[4] = {q.x, q.y, q.z, q.w};
            float *o = p.out + (long long)(n0 + c) * p.out_ld + row;
            if (p.resid) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (row + j < p.rows) v[j] += __ldcg(p.resid + (long long)(n0 + c) * p.resid_ld + row + j);
            }
            if (vec) *reinterpret_cast<float4 *>(o) = make_float4(v[0], v[1], v[2], v[3]);
            else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (row + j < p.rows) o[j] = v[j];
            }
        }
        cluster_sync();                                                 // nobody leaves while a peer still reads
    }
    if (*abort_flag) {
        for (int i = 0; i < 200; ++i) __nanosleep(1000);                // copies in flight land before the memory is released
        __syncthreads();
    }
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)p.tmem_cols) : "memory");
    }
}

// ---- host side ---------------------------------------------------------------------------------

constexpr int SMEM_ONE = 220 * 1024, SMEM_TWO = 108 * 1024;      // one block on an SM, or two

// Blocks resident at once, one or two on an SM, in clusters of 1 .. 8 (what the occupancy calculator gives on 148 SMs: clusters
// live inside a processing cluster).
constexpr int RESIDENT[2][9] = {{0, 148, 148, 135, 132, 130, 132, 105, 120}, {0, 296, 296, 279, 284, 280, 270, 259, 264}};

struct Shape { Form form; int bn, splits, slots, two, acc_cols, n_acc, tmem; };

// Ring slots and accumulators of a tile width; false when it does not fit.
bool place_tile(Form form, int bn, int planes, bool two, Shape *o)
{
    const bool q8 = form == Q8_WIDE || form == Q8_NARROW;
    if (bn > form_bn(form) || (form == Q8_WIDE && two) || (form == Q8_NARROW && !two)) return false;
    const int raw = form == Q8_WIDE ? Shape_of<Q8_WIDE>::raw * Shape_of<Q8_WIDE>::depth : form == Q8_NARROW ? Shape_of<Q8_NARROW>::raw * Shape_of<Q8_NARROW>::depth : 0;
    const int slot = (q8 ? 0 : (int)W_TILE) + bn * KB * 2 * planes, columns = two ? 256 : 512, room = (two ? SMEM_TWO : SMEM_ONE) - raw;
    o->form = form;
    o->slots = room / slot > MAX_SLOTS ? MAX_SLOTS : room / slot;
    o->acc_cols = (bn + 31) / 32 * 32;
    if (q8) {                                                    // weight tiles live in tensor memory: 64 columns each, beside two accumulators
        const int w_slots = (columns - 2 * o->acc_cols) / 64;
        if (o->slots > w_slots) o->slots = w_slots;
        if (o->slots > 4) o->slots = 4;
    }
    const int left = columns - (q8 ? o->slots * 64 : 0);
    o->n_acc = left / o->acc_cols > MAX_ACC ? MAX_ACC : left / o->acc_cols;
    if (o->slots < 2 || o->n_acc < 2) return false;
    const int used = o->n_acc * o->acc_cols + (q8 ? o->slots * 64 : 0);
    for (o->tmem = 32; o->tmem < used;) o->tmem *= 2;
    return true;
}

// Tile width, blocks per tile and blocks per SM: the least modelled time. A step of 64 columns takes as long as the slowest of
// its products (2 clocks a column and product), its operand bytes (an SM takes in about 52 a clock) and,
// for Q8_0, making the weight tile. A block costs some 3000 clocks beside its steps and its result goes out at 8 clocks a column; in
// several waves of F16 tiles twice that with one block on an SM, and half of it with two, where one's start and end lie under the other's
// steps (a Q8_0 block has threads for a whole SM).
Shape pick_shape(bool q8, int rows, int cols, int n, int planes, int sms)
{
    const int mt = (rows + WM - 1) / WM, nkb = (cols + KB - 1) / KB;
    Shape best = {};
    double least = 1e30;
    int last_bn = 0;
    for (int nt = (n + 127) / 128; nt <= (n + 15) / 16; ++nt) {
        const int bn = ((n + nt - 1) / nt + 15) / 16 * 16;
        if (bn == last_bn) continue;
        last_bn = bn;
        if (bn < 64 && nt > 1) break;
        const int ntile = (n + bn - 1) / bn;
        const int products = q8 ? planes + 1 : planes;
        const double in = (q8 ? WM * 68.0 : (double)W_TILE) + bn * KB * 2.0 * planes;
        double step = 2.0 * bn * products;
        if (q8 && step < 300.0) step = 300.0;
        if (step < in / 52.0) step = in / 52.0;
        for (int two = 0; two <= 1; ++two) {
            Shape sh = {};
            if (!place_tile(!q8 ? (bn <= 32 ? F16_NARROW : F16_WIDE) : two ? Q8_NARROW : Q8_WIDE, bn, planes, two, &sh)) continue;
            for (int s = 1; s <= 8; ++s) {
                const int per = (nkb + s - 1) / s;
                if (s > 1 && (per < 4 || s > bn)) break;
                const long long blocks = (long long)mt * ntile * s;
                const long long place = (long long)RESIDENT[two][s] * sms / 148;
                const long long waves = (blocks + place - 1) / place;
                // two blocks share an SM's time unless the last wave leaves most SMs one block
                const double share = two ? (waves > 1 || blocks > sms * 3 / 2 ? 2.0 : blocks > sms ? 1.0 + (double)(blocks - sms) / sms : 1.0) : 1.0;
                const bool under = !q8 && two && s == 1 && waves > 1;
                const double ends = (under ? 0.5 : !q8 && waves > 1 ? 2.0 : 1.0) * (3000.0 + bn * 8.0) + (s > 1 ? 1500.0 + bn * 4.0 : 0.0);
                const double each = under && step > 2.0 * bn * products ? step * 52.0 / 56.0 : step;       // they keep the SM's port busier, too
                const double cost = waves * (share * per * each * (sh.slots < 3 && !under ? 1.1 : 1.0) + ends);
                if (cost < least) { least = cost; best = sh; best.bn = bn; best.splits = s; best.two = two; }
            }
        }
    }
    return best;
}

template <Form F>
int launch_rows(const CUtensorMap &mw, const CUtensorMap &mx, const RowsMat &a, int use_pdl, cudaStream_t st)
{
    using Of = Shape_of<F>;
    size_t smem = (size_t)((Of::q8 ? 0 : W_TILE) + a.bn * KB * 2 * a.planes) * a.slots + (size_t)Of::raw * Of::depth;
    if (a.splits > 1 && smem < (size_t)a.bn * WM * 4) smem = (size_t)a.bn * WM * 4;
    smem += 1024;
    const cudaError_t set = cudaFuncSetAttribute(rows_matmul_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_ONE + 1024);
    if (set != cudaSuccess) return (int)set;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((a.n + a.bn - 1) / a.bn, (a.rows + WM - 1) / WM, a.splits);
    cfg.blockDim = dim3(Of::threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    int n = 0;
    if (a.splits > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = 1; at[n].val.clusterDim.y = 1; at[n].val.clusterDim.z = a.splits;
        ++n;
    }
    if (use_pdl) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = at;
    cfg.numAttrs = n;
    const cudaError_t rc = cudaLaunchKernelEx(&cfg, rows_matmul_kernel<F>, mw, mx, a);
    ++g_b200_launches;
    return rc != cudaSuccess ? (int)rc : (int)cudaGetLastError();
}

// One block per weight row: the power of two that the row's scales are divided by (largest one in [2^7, 2^8)).
__global__ void __launch_bounds__(128) q8_row_scale_kernel(const uint8_t *w, long long stride, int cols, float *out)
{
    __shared__ float red[4];
    const __half *s = reinterpret_cast<const __half *>(w + (long long)blockIdx.x * stride + cols);
    float m = 0.0f;
    for (int i = threadIdx.x; i < cols / 32; i += 128) m = fmaxf(m, fabsf(__half2float(s[i])));
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        m = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
        out[blockIdx.x] = m > 0.0f && m < INFINITY ? ldexpf(1.0f, ilogbf(m) - 7) : 1.0f;
    }
}

}  // namespace

extern "C" int b200_q8_row_scale(const void *d_w, long long stride, int rows, int cols, float *d_out, void *stream)
{
    if (!d_w || !d_out || rows <= 0 || cols <= 0 || cols % 32 || (stride & 15)) return B200_E_BADARG;
    q8_row_scale_kernel<<<rows, 128, 0, (cudaStream_t)stream>>>(static_cast<const uint8_t *>(d_w), stride, cols, d_out);
    ++g_b200_launches;
    return (int)cudaGetLastError();
}

extern "C" int b200_rows_matmul(const b200_rows_matmul_args *a, void *stream)
{
    if (!a || !a->d_w || !a->d_x || !a->d_out || a->rows <= 0 || a->cols <= 0 || a->n <= 0) return B200_E_BADARG;
    if (a->wtype != B200_WT_Q8 && a->wtype != B200_WT_F16) return B200_E_UNSUPPORTED;
    const bool q8 = a->wtype == B200_WT_Q8;
    if ((a->planes != 1 && a->planes != 2) || (a->planes == 2 && a->plane_rows < a->n) || a->plane_rows < 0) return B200_E_BADARG;
    if (a->cols % (q8 ? 32 : 8) || (q8 && !a->d_w_scale) || (a->w_stride & 15) || a->x_ld < a->cols || (a->x_ld & 7)) return B200_E_BADARG;
    if (a->w_stride < (q8 ? a->cols / 32 * 34LL : a->cols * 2LL) || a->out_ld < a->rows || (a->d_resid && a->resid_ld < a->rows)) return B200_E_BADARG;
    if ((reinterpret_cast<uintptr_t>(a->d_w) & 15) || (reinterpret_cast<uintptr_t>(a->d_x) & 15)) return B200_E_BADARG;
    if ((a->rows + WM - 1) / WM > 65535) return B200_E_TOOLARGE;
    const Shape sh = pick_shape(q8, a->rows, a->cols, a->n, a->planes, tc_sm_count());
    RowsMat p = {};
    p.w = static_cast<const uint8_t *>(a->d_w); p.w_stride = a->w_stride;
    p.w_scale = a->d_w_scale; p.x_scale = a->d_x_scale;
    p.rows = a->rows; p.cols = a->cols; p.n = a->n; p.planes = a->planes; p.plane_rows = a->plane_rows;
    p.out = a->d_out; p.out_ld = a->out_ld; p.resid = a->d_resid; p.resid_ld = a->resid_ld;
    p.d_err = a->d_err;
    p.bn = sh.bn; p.slots = sh.slots; p.splits = sh.splits; p.tmem_cols = sh.tmem; p.acc_cols = sh.acc_cols; p.n_acc = sh.n_acc; p.every = a->planes == 1 ? 1 << 20 : 1;
    if (p.bn == 0) return B200_E_UNSUPPORTED;
    CUtensorMap mw, mx;
    const long long xrows = (long long)(a->planes - 1) * a->plane_rows + a->n;
    if (!tc_make_map(&mx, a->d_x, xrows, a->cols, a->x_ld * 2, KB, sh.bn, CU_TENSOR_MAP_DATA_TYPE_FLOAT16)) return B200_E_UNSUPPORTED;
    if (q8) mw = mx;                                             // not used
    else if (!tc_make_map(&mw, a->d_w, a->rows, a->cols, a->w_stride, KB, WM, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, CU_TENSOR_MAP_L2_PROMOTION_L2_256B)) return B200_E_UNSUPPORTED;
    cudaStream_t st = (cudaStream_t)stream;
    switch (sh.form) {
    case F16_WIDE: return launch_rows<F16_WIDE>(mw, mx, p, a->use_pdl, st);
    case F16_NARROW: return launch_rows<F16_NARROW>(mw, mx, p, a->use_pdl, st);
    case Q8_WIDE: return launch_rows<Q8_WIDE>(mw, mx, p, a->use_pdl, st);
    default: return launch_rows<Q8_NARROW>(mw, mx, p, a->use_pdl, st);
    }
}
