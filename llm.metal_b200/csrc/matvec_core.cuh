// Fused weight-streaming matrix-vector product for batch-1 decode (sm_100a).
//
// One block per SM slot owns a contiguous range of rows. A producer warp
// streams that range through a shared-memory ring with bulk asynchronous
// copies (TMA, cp.async.bulk + mbarrier): rows of a packed matrix are
// contiguous, so one copy instruction moves a whole stage (RB rows, 16-24 KB)
// and the ring keeps ~100 KB per block in flight without holding registers.
// Consumer threads own fixed 16-byte column slices (16 int8 quants or 8
// halves) of every row, so their slice of the input vector stays in registers
// for the whole kernel; consumer groups take stages round-robin. Warps run free of each other: a warp folds the RB rows of a stage across
// its lanes with one transposing shuffle reduction and leaves its sums in shared memory; one barrier per window of some 2000 sums (all
// rows of a block but for an LM head), then a thread per row adds the warps' sums in fixed order (reproducible run to run) and
// stores the result.
// Bound by instructions and their latencies with 4 to 5 warps on a scheduler, not by HBM: the input vector is assembled by all consumers, a barrier
// per sum, and nothing divides. A barrier and a one-warp epilogue per stage, 64-bit divisions, norms by one group: 0.28 ms a token of 41 such
// launches (2048 wide, bfloat16), 0.24 now; fp32 210 us and 175. Two blocks of half the ring on an SM, so that the next launch's
// weights arrive early: no gain (0.28), blocks of one launch then share SMs.
//
// Launched with programmatic dependent launch, a block of the NEXT kernel in
// the stream starts as soon as an SM has room for it (with the default 192 KB
// ring that is when a block of this kernel has left), fills its own ring with
// weights and only then waits for its input.
//
// The math is the reference's q8_matvec / f16_matvec
// (shaders/q8_kernels.metal:10-42, 97-127): fp32 activations, integer quants
// converted to fp32, fp32 multiply-accumulate, partial block sums scaled by
// the binary16 block scale. BF16 and F32 weights have no counterpart there. Input assembly and the epilogues fold in rms_norm
// (:133-157), residual_add (:369-375), silu_mul / gelu_mul (:337-363), the
// embedding copy (src/nn/fast_inference.c:386-392) and argmax (:469-476).
//
// This header holds the kernel and its launchers; matvec.cu instantiates them for Q8_0 and F16 weights, matvec_ext.cu
// and matvec_streams.cu for BF16 and F32 (translation units of their own: they compile side by side).
#pragma once
#include "stream_core.cuh"
#include "../../include/llmb200_kernels.h"

extern unsigned long long g_b200_launches;

namespace b200_mv {

struct Geometry {
    int T;              // threads per consumer group (a multiple of 32)
    int NG;             // consumer groups
    int nstage;         // ring slots
    unsigned slot_bytes;  // bytes per slot (RB rows, rounded up to 128)
    int base, rem;      // row units of a block, and the blocks that have one more
    int per_warp;       // 65536 / (warps of a group), rounded up: which group a warp belongs to without a division
    int win, part;      // stages per window of rows (a multiple of NG), floats of its warp sums; two windows take turns
    int xs;             // floats of the input vector in shared memory; 0: it is read as it is
};

// Sums of K values over the nC consumer threads; every thread gets them. One barrier: calls take the halves of `red` (2 x 4 x 32 floats,
// zeros where there is no warp) in turn, and between a call and the next but one lies the barrier of the one between.
template <int K>
__device__ __forceinline__ void block_sums(float (&v)[K], float *red, int &turn, int nC, int tid)
{
    float *r = red + 128 * turn;
    turn ^= 1;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        v[k] = warp_sum(v[k]);
        if ((tid & 31) == 0) r[k * 32 + (tid >> 5)] = v[k];
    }
    named_barrier(1, nC);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        float tot = 0.0f;
        for (int i = 0; i < nC >> 5; i += 4) {
            const float4 q = *reinterpret_cast<const float4 *>(r + k * 32 + i);
            tot += q.x; tot += q.y; tot += q.z; tot += q.w;
        }
        v[k] = tot;
    }
}

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void st4(float *p, float4 v) { *reinterpret_cast<float4 *>(p) = v; }
__device__ __forceinline__ float squares(float4 v, float s) { return fmaf(v.w, v.w, fmaf(v.z, v.z, fmaf(v.y, v.y, fmaf(v.x, v.x, s)))); }

// Weights of a norm for this thread's items (four elements each, nC items apart): those of the first one are fetched before the wait for the
// previous kernel, they are constants. ANY: a vector that may start on any element (the norm of slot sums of Q8_0 and F16 products takes one).
template <bool ANY = false>
struct NormWeights {
    const float *at;
    float4 first;
    __device__ __forceinline__ static float4 four(const float *p)
    {
        if (ANY && (reinterpret_cast<uintptr_t>(p) & 15)) return make_float4(p[0], p[1], p[2], p[3]);
        return ld4(p);
    }
    __device__ __forceinline__ void fetch(const float *p, int tid, int cols)
    {
        at = p;
        first = p && 4 * tid < cols ? four(p + 4 * tid) : make_float4(0, 0, 0, 0);
    }
    __device__ __forceinline__ float4 get(int it, int e) const { return it == 0 ? first : four(at + e); }
};

// The vector that a block assembles: a thread's first item (four elements) in `q`, zeros where it has none, further ones (nC items apart; more than
// 4 nC columns only) in shared memory, where the first one goes at the end. FAM_POST keeps the first one there too: a second copy of the norms by
// parts, for the register, is code that every launch fetches and few warps share (two layers of 2048, fp32, 64 ids: 12.2 ms with it, 11.4 without; layer
// norms of streams the other way round: four layers of 256, bfloat16, 40 ids 5.24 ms with the register, 5.58 without).
#define B200_ITEMS_FROM(first, it, e) for (int it = first, e = 4 * (tid + first * nC); e < cols; ++it, e += 4 * nC)
#define B200_ITEMS(it, e) B200_ITEMS_FROM(0, it, e)
#define B200_FURTHER(it, e) B200_ITEMS_FROM(HELD, it, e)             // HELD: 1 where the first one is in q

// RMS norm of the vector, `groups` equal consecutive parts of its first `dim` elements each by its own mean square; what follows them stays.
__device__ __forceinline__ void norm_parts(float *xs, const NormWeights<> &gamma, int cols, int dim, int groups, float eps, float *red, int &turn,
                                           int nC, int tid)
{
    const int len = dim / groups;
    for (int k0 = 0; k0 < groups; k0 += 4) {                             // four parts a barrier
        float ss[4] = {};
        auto squares_of = [&](const float4 &v, int e) {
            const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int lo = (k0 + k) * len, hi = k0 + k < groups ? lo + len : lo;
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (e + j >= lo && e + j < hi) ss[k] = fmaf(f[j], f[j], ss[k]);
            }
        };
        B200_ITEMS(it, e) squares_of(ld4(xs + e), e);
        block_sums<4>(ss, red, turn, nC, tid);
        // a scale to each of four lanes: the code of the divisions once (256 wide, bfloat16, 40 ids: 5.00 ms with all four in every lane, 4.84; 2048 wide
        // 5.08 and 4.85)
        const float sum = tid & 1 ? (tid & 2 ? ss[3] : ss[1]) : (tid & 2 ? ss[2] : ss[0]);
        const float scale = 1.0f / sqrtf(sum / (float)len + eps);
#pragma unroll
        for (int k = 0; k < 4; ++k) ss[k] = __shfl_sync(0xffffffffu, scale, k);
        auto normed = [&](const float4 &v, const float4 &g, int e) {
            float f[4] = {v.x, v.y, v.z, v.w};
            const float w[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int lo = (k0 + k) * len, hi = k0 + k < groups ? lo + len : lo;
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (e + j >= lo && e + j < hi) f[j] = w[j] * (f[j] * ss[k]);
            }
            return make_float4(f[0], f[1], f[2], f[3]);
        };
        B200_ITEMS(it, e) st4(xs + e, normed(ld4(xs + e), gamma.get(it, e), e));
    }
}

// Layer norm (mean taken off, variance of the deviations, weight and bias) of the first `dim` elements; the
// columns past them hold zeros before and after (their weight and bias are zero).
__device__ __forceinline__ void layer_norm(float4 &q, float *xs, const NormWeights<> &gamma, const NormWeights<> &beta, int cols, int dim, float eps, float *red,
                                           int &turn, int nC, int tid)
{
    constexpr int HELD = 1;
    float sum[1] = {(q.x + q.y) + (q.z + q.w)};
    B200_FURTHER(it, e) { const float4 v = ld4(xs + e); sum[0] += (v.x + v.y) + (v.z + v.w); }
    block_sums<1>(sum, red, turn, nC, tid);
    const float mean = sum[0] / (float)dim;
    auto centred = [&](float4 v, int e) {
        if (e < dim) v.x -= mean;
        if (e + 1 < dim) v.y -= mean;
        if (e + 2 < dim) v.z -= mean;
        if (e + 3 < dim) v.w -= mean;
        return v;
    };
    q = centred(q, 4 * tid);
    float ss[1] = {squares(q, 0.0f)};
    B200_FURTHER(it, e) { const float4 v = centred(ld4(xs + e), e); st4(xs + e, v); ss[0] = squares(v, ss[0]); }
    block_sums<1>(ss, red, turn, nC, tid);
    const float inv = 1.0f / sqrtf(ss[0] / (float)dim + eps);
    auto normed = [&](const float4 &v, const float4 &g, const float4 &b) {
        return make_float4(fmaf(g.x, v.x * inv, b.x), fmaf(g.y, v.y * inv, b.y), fmaf(g.z, v.z * inv, b.z), fmaf(g.w, v.w * inv, b.w));
    };
    q = normed(q, gamma.first, beta.first);
    B200_FURTHER(it, e) st4(xs + e, normed(ld4(xs + e), gamma.get(it, e), beta.get(it, e)));
}

// Which of the optional parts an instantiation holds (registers decide how well the row loop runs): FAM_PLAIN the parts
// every weight type has, FAM_POST post-norm inputs, gated outputs, depth sums and the logit cap, FAM_STREAMS layer
// norms, learned positions, residual streams and the squared relu.
enum { FAM_PLAIN = 0, FAM_POST = 1, FAM_STREAMS = 2 };

template <int WT, int SPT, int RB, int MAXT, int FAM>
__global__ void __launch_bounds__(MAXT)
matvec_kernel(const __grid_constant__ b200_matvec_args p, const Geometry geo)
{
    constexpr int E = (WT == B200_WT_Q8) ? 16 : (WT == B200_WT_F32) ? 4 : 8;       // elements per 16-byte slice
    constexpr bool EXT = FAM == FAM_POST, STR = FAM == FAM_STREAMS;
    constexpr int HELD = EXT ? 0 : 1;                                   // see B200_FURTHER
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int T = geo.T, NG = geo.NG, nstage = geo.nstage, nwg = T >> 5, nwgp = nwg | 1, nC = NG * T;
    unsigned char *ring = smem_raw;
    uint64_t *full = reinterpret_cast<uint64_t *>(ring + (size_t)nstage * geo.slot_bytes);
    uint64_t *empty = full + nstage;
    float *red = reinterpret_cast<float *>(ring + (size_t)nstage * geo.slot_bytes + 256);   // [2][4][32]
    float *am_v = red + 256;                                    // [32], a value per warp
    int *am_i = reinterpret_cast<int *>(am_v + 32);             // [32]
    float *xs = reinterpret_cast<float *>(am_i + 32);           // [geo.xs], the assembled input
    float *wpart = xs + geo.xs;                                 // one or two windows of [rows][nwgp] warp sums
    __shared__ int s_last;
    __shared__ float s_conn[STR ? B200_MAX_STREAMS * (B200_MAX_STREAMS + 2) : 1];     // mix, out, next read of the streams

    const int tid = threadIdx.x;
    for (int i = tid; i < 256; i += blockDim.x) red[i] = 0.0f;
    const int ralign = (p.out_mode == B200_OUT_GLU) ? 2 : 1;
    const int bid = blockIdx.x, r0 = (bid * geo.base + min(bid, geo.rem)) * ralign, r1 = r0 + (geo.base + (bid < geo.rem)) * ralign;
    const int nst = (r1 - r0 + RB - 1) / RB;

    if (tid < nstage) {
        mbar_init(&full[tid], 1); mbar_init(&empty[tid], nwg);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    // Every thread signals: the next kernel in the stream may be scheduled now and start
    // filling its own ring beside this block.
    pdl_launch_dependents();

    // ---------------- producer warp: weights depend on no earlier kernel ----------------
    if (tid >= nC) {
        if (tid == nC) {
            const unsigned char *wbase = static_cast<const unsigned char *>(p.d_w);
            for (int i = 0; i < nst; ++i) {
                const int slot = i % nstage;
                if (i >= nstage && !mbar_wait(&empty[slot], ((i / nstage) - 1) & 1)) {
                    if (p.d_err) *p.d_err = 2;
                    break;
                }
                const int row0 = r0 + i * RB;
                const int nr = min(RB, r1 - row0);
                const unsigned bytes = (unsigned)nr * (unsigned)p.row_stride;
                mbar_expect_tx(&full[slot], bytes);
                bulk_load(ring + (size_t)slot * geo.slot_bytes, wbase + (long long)row0 * p.row_stride, bytes, &full[slot]);
            }
        } else if constexpr (EXT) {
            // the producer warp's other lanes form the depth sums of this block's rows
            if (p.hist_n > 0) {
                pdl_wait();
                for (int row = r0 + (tid - nC - 1); row < r1; row += 31) {
                    float a = 0.0f;
#pragma unroll 8
                    for (int j = 0; j < p.hist_n; ++j) a = fmaf(p.d_hist_coef[j], p.d_hist[(long long)j * p.hist_stride + row], a);
                    p.d_hist_out[row] = a;
                }
            }
        }
        return;
    }

    // ---------------- consumers ----------------
    const int g = ((tid >> 5) * geo.per_warp) >> 16, t = tid - g * T, lane = t & 31, wg = t >> 5, cols = p.cols;
    const bool assemble = geo.xs > 0;            // otherwise the input is a vector that each thread reads its slices of
    int turn = 0;                                // which half of red the next sum takes

    // The norm weights are constants: their round trip is taken before the wait for the previous
    // kernel, not after it.
    NormWeights<> gm, gb;
    NormWeights<FAM == FAM_PLAIN> gp;
    gm.fetch(p.d_norm_gamma, tid, cols);
    gp.fetch(p.d_slot_norm_gamma, tid, cols);                        // of a post-norm input, of normalised slot sums, or of embeddings
    if constexpr (STR) {
        gb.fetch(p.d_norm_beta, tid, cols);
        if (p.out_mode == B200_OUT_STREAMS)                      // read after the barrier that ends the first window
            for (int i = tid; i < p.n_streams * (p.n_streams + 2); i += nC) s_conn[i] = p.d_connect[i];
    }

    pdl_wait();

    // Tensor parallel: every rank's partial vector must have landed in `slots`
    // (and, for the first kernel of a token, every rank must be done reading the
    // previous token's slots) before this block goes on.
    if (p.n_wait > 0) {
        if (tid < p.n_wait) {
            const unsigned want = (*p.d_epoch) * (unsigned)p.epoch_mul + (unsigned)p.epoch_add;
            if (!wait_flag_ge(p.d_wait_flags + tid, want, p.spin_limit > 0 ? p.spin_limit : B200_SPIN_LIMIT)) *p.d_err = 1;
        }
        named_barrier(1, nC);
    }

    // ---------------- input assembly ----------------
    // Every SM needs the whole input vector. Where it has to be assembled (slot sums, norms) all consumers of a block do it together, four
    // elements a thread: one read of the vector a block (all SMs read the same few KB of L2 at once, and every
    // extra reader queues behind the others), a barrier per sum.
    if (assemble) {
        const bool store = blockIdx.x == 0, mine = 4 * tid < cols;
        const int e0 = 4 * tid, norm_dim = p.norm_dim > 0 ? p.norm_dim : cols, groups = p.norm_groups > 1 ? p.norm_groups : 1;
        const float4 none = make_float4(0, 0, 0, 0);
        float4 q = none;
        if (p.in_mode == B200_IN_VEC || (EXT && p.in_mode == B200_IN_POSTNORM)) {
            if (HELD && mine) q = ld4(p.d_in_vec + e0);
            B200_FURTHER(it, e) st4(xs + e, ld4(p.d_in_vec + e));
            if constexpr (EXT) {
                if (p.in_mode == B200_IN_POSTNORM) {
                    const float4 mix0 = p.d_mix_in && mine ? ld4(p.d_mix_in + e0) : none;          // fetched before the norm's sums
                    const float coef = p.d_mix_in ? *p.d_mix_coef : 1.0f;
                    norm_parts(xs, gp, cols, norm_dim, groups, p.eps, red, turn, nC, tid);
                    B200_ITEMS(it, e) {
                        float4 v = ld4(xs + e);
                        if (store && p.d_post_copy) st4(p.d_post_copy + e, v);
                        if (p.d_mix_in) {
                            const float4 m = it == 0 ? mix0 : ld4(p.d_mix_in + e);
                            v = make_float4(fmaf(coef, v.x, m.x), fmaf(coef, v.y, m.y), fmaf(coef, v.z, m.z), fmaf(coef, v.w, m.w));
                            st4(xs + e, v);
                        }
                        if (store && p.d_resid_out) st4(p.d_resid_out + e, v);
                    }
                }
            }
        } else {
            if (p.in_mode == B200_IN_EMBED) {
                long long tok = p.d_tokens[*p.d_pos];
                if (tok < 0 || tok >= p.emb_rows) tok = 0;      // never index outside the table
                const float *er = p.d_emb + tok * (long long)cols;
                const float *row = STR && p.d_emb_pos ? p.d_emb_pos + (long long)min(*p.d_pos, p.emb_pos_rows - 1) * cols : nullptr;
                auto embedded = [&](int e) {
                    float4 v = ld4(er + e);
                    v.x *= p.emb_scale; v.y *= p.emb_scale; v.z *= p.emb_scale; v.w *= p.emb_scale;
                    if (row) { const float4 r = ld4(row + e); v.x += r.x; v.y += r.y; v.z += r.z; v.w += r.w; }
                    return v;
                };
                if (HELD && mine) q = embedded(e0);
                B200_FURTHER(it, e) st4(xs + e, embedded(e));
                if constexpr (STR) {
                    if (p.d_slot_norm_beta) {
                        NormWeights<> b;
                        b.fetch(p.d_slot_norm_beta, tid, cols);
                        layer_norm(q, xs, gp, b, cols, norm_dim, p.eps, red, turn, nC, tid);
                    }
                }
            } else {
                float ss[1] = {0.0f};
                auto slots = [&](int e) {
                    float4 a = none;
                    for (int k = 0; k < p.n_slots; ++k) {
                        // slots may be written by other GPUs: read them from L2, the point of coherence, never from L1
                        const float4 v = __ldcg(reinterpret_cast<const float4 *>(p.d_slots + (long long)k * p.slot_stride + e));
                        a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
                    }
                    if (FAM == FAM_PLAIN && p.d_slot_norm_gamma) ss[0] = squares(a, ss[0]);
                    else { const float4 r = ld4(p.d_resid_in + e); a.x += r.x; a.y += r.y; a.z += r.z; a.w += r.w; }
                    return a;
                };
                if (HELD && mine) q = slots(e0);
                B200_FURTHER(it, e) st4(xs + e, slots(e));
                if constexpr (FAM == FAM_PLAIN) if (p.d_slot_norm_gamma) {
                    const float4 r0 = mine ? ld4(p.d_resid_in + e0) : none;
                    block_sums<1>(ss, red, turn, nC, tid);
                    const float inv = 1.0f / sqrtf(ss[0] / (float)cols + p.eps);
                    auto added = [&](const float4 &a, const float4 &w, const float4 &r) {
                        return make_float4(r.x + w.x * a.x * inv, r.y + w.y * a.y * inv, r.z + w.z * a.z * inv, r.w + w.w * a.w * inv);
                    };
                    q = added(q, gp.first, r0);
                    B200_FURTHER(it, e) st4(xs + e, added(ld4(xs + e), gp.get(it, e), ld4(p.d_resid_in + e)));
                }
            }
            if (store && p.d_resid_out) {
                if (HELD && mine) st4(p.d_resid_out + e0, q);
                B200_FURTHER(it, e) st4(p.d_resid_out + e, ld4(xs + e));
            }
            if constexpr (STR) {
                if (p.in_mode == B200_IN_EMBED && p.d_mix_coef) {    // what the first reader takes of the streams, all equal here
                    const float c = *p.d_mix_coef;
                    q = make_float4(c * q.x, c * q.y, c * q.z, c * q.w);
                    B200_FURTHER(it, e) { const float4 v = ld4(xs + e); st4(xs + e, make_float4(c * v.x, c * v.y, c * v.z, c * v.w)); }
                }
            }
        }
        if (p.d_norm_gamma) {
            if constexpr (STR) layer_norm(q, xs, gm, gb, cols, norm_dim, p.eps, red, turn, nC, tid);
            else if constexpr (EXT) norm_parts(xs, gm, cols, norm_dim, groups, p.eps, red, turn, nC, tid);
            else {
                float ss[1] = {squares(q, 0.0f)};
                B200_FURTHER(it, e) ss[0] = squares(ld4(xs + e), ss[0]);
                block_sums<1>(ss, red, turn, nC, tid);
                const float inv = 1.0f / sqrtf(ss[0] / (float)cols + p.eps);
                auto normed = [&](const float4 &v, const float4 &w) { return make_float4(w.x * v.x * inv, w.y * v.y * inv, w.z * v.z * inv, w.w * v.w * inv); };
                q = normed(q, gm.first);
                B200_FURTHER(it, e) st4(xs + e, normed(ld4(xs + e), gm.get(it, e)));
            }
        }
        if (HELD && mine) st4(xs + e0, q);
        if (p.d_in_copy && store) B200_ITEMS(it, e) st4(p.d_in_copy + e, ld4(xs + e));
        named_barrier(1, nC);
    }
    float x[SPT][E];
    // Byte offsets of this thread's slices inside a row. Threads past the end of the row read slice 0
    // (valid memory) against a zero input slice and drop the result.
    uint32_t qoff[SPT], soff[SPT];
#pragma unroll
    for (int s = 0; s < SPT; ++s) {
        const int col = (s * T + t) * E;
        const bool on = col < cols;
#pragma unroll
        for (int e = 0; e < E; e += 4) {
            const float4 q = !on ? make_float4(0, 0, 0, 0) : ld4((assemble ? xs : p.d_in_vec) + col + e);
            x[s][e] = q.x; x[s][e + 1] = q.y; x[s][e + 2] = q.z; x[s][e + 3] = q.w;
        }
        const int c = on ? col : 0;
        qoff[s] = (uint32_t)(WT == B200_WT_Q8 ? c : WT == B200_WT_F32 ? 4 * c : 2 * c);
        soff[s] = (uint32_t)cols + (uint32_t)(c >> 5) * 2u;      // Q8: scales follow the quants of a row
    }
    if (p.d_in_copy && !assemble && blockIdx.x == 0)
        for (int e = 4 * tid; e < cols; e += 4 * nC) st4(p.d_in_copy + e, ld4(p.d_in_vec + e));

    // ---------------- consume the ring: group g takes stages g, g+NG, ... ----------------
    float best_v = -INFINITY;
    int best_i = 0x7fffffff;
    const uint32_t ring_s = smem_u32(ring), stride = (uint32_t)p.row_stride;
    int slot = g;
    unsigned phase = 0;
    for (int s0 = 0, buf = 0; s0 < nst; s0 += geo.win, buf ^= 1) {
        const int s1 = min(s0 + geo.win, nst), w0 = r0 + s0 * RB, n = min(r1 - w0, (s1 - s0) * RB);
        float *part = wpart + buf * geo.part;
        // what a gated output adds to and scales by, or the streams of the row, for the row that this thread emits first: on their way
        // while the rows are multiplied
        float o_resid = 0.0f, o_gate = 0.0f, old[STR ? B200_MAX_STREAMS : 1];
        if constexpr (EXT) {
            if (p.out_mode == B200_OUT_GATED && tid < n) {
                o_resid = p.d_out_resid[w0 + tid];
                o_gate = p.d_out_gate[w0 + tid] + p.d_out_gate_bias[w0 + tid];
            }
        }
        if constexpr (STR) {
            if (p.out_mode == B200_OUT_STREAMS) {
#pragma unroll
                for (int k = 0; k < B200_MAX_STREAMS; ++k)
                    old[k] = k < p.n_streams && tid < n ? p.d_streams_in[k * p.streams_in_stride + w0 + tid] : 0.0f;
            }
        }
        for (int i = s0 + g; i < s1; i += NG) {
            if (!mbar_wait(&full[slot], phase) && p.d_err) *p.d_err = 3;
            const uint32_t sb = ring_s + (uint32_t)slot * geo.slot_bytes;
            // Rows past the end hold stale bytes; they are computed like the others (no predicates in the
            // hot loop), stay in their own reduction lane and are never emitted.
            uint4 wq[RB][SPT];
            uint32_t ws[RB][SPT];
#pragma unroll
            for (int j = 0; j < RB; ++j)
#pragma unroll
                for (int s = 0; s < SPT; ++s) {
                    wq[j][s] = lds_128(sb + (uint32_t)j * stride + qoff[s]);
                    if (WT == B200_WT_Q8) ws[j][s] = lds_u16(sb + (uint32_t)j * stride + soff[s]);
                }
            float v[RB];
#pragma unroll
            for (int j = 0; j < RB; ++j) {
                float acc = 0.0f;
#pragma unroll
                for (int s = 0; s < SPT; ++s) {
                    float d;
                    if (WT == B200_WT_Q8) d = __half2float(__ushort_as_half((unsigned short)ws[j][s])) * dot16_q8(wq[j][s], x[s]);
                    else if (WT == B200_WT_BF16) d = dot8_bf16(wq[j][s], x[s]);
                    else if (WT == B200_WT_F32) d = dot4_f32(wq[j][s], x[s]);
                    else d = dot8_f16(wq[j][s], x[s]);
                    acc += d;                      // threads past the end of the row hold a zero input slice
                }
                v[j] = acc;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[slot]);              // this warp no longer reads the slot
            slot += NG;
            if (slot >= nstage) { slot -= nstage; phase ^= 1; }
            const float tot = reduce_rows<RB>(v, lane);
            if (lane < RB) part[((i - s0) * RB + lane) * nwgp + wg] = tot;
        }
        named_barrier(1, nC);

        // ---------------- a thread per row: the warps' sums in order, and the epilogue ----------------
        // (the next window's sums go to the other buffer, and nobody comes back to this one before the next barrier)
        auto row_sum = [&](int i) {
            float y = 0.0f;
            for (int w = 0; w < nwg; ++w) y += part[i * nwgp + w];
            return y;
        };
        if (p.out_mode == B200_OUT_GLU) {
            for (int i = 2 * tid; i < n; i += 2 * nC) {
                const float y = row_sum(i), u = row_sum(i + 1);
                const int row = w0 + i;
                if (EXT && p.glu_rows > 0 && row >= p.glu_rows) { p.d_out2[row - p.glu_rows] = y; p.d_out2[row + 1 - p.glu_rows] = u; }
                else p.d_out[0][p.out_offset + (row >> 1)] = (p.act == 0 ? act_silu(y) : act_gelu_tanh(y)) * u;
            }
            continue;
        }
        for (int i = tid; i < n; i += nC) {
            float y = row_sum(i);
            const int row = w0 + i;
            if (EXT && p.out_mode == B200_OUT_GATED) {
                if (i != tid) { o_resid = p.d_out_resid[row]; o_gate = p.d_out_gate[row] + p.d_out_gate_bias[row]; }
                p.d_out[0][p.out_offset + row] = fmaf(p.resid_alpha, o_resid, sigmoid_f32(o_gate) * y);
            } else if (STR && p.out_mode == B200_OUT_STREAMS) {
                if constexpr (STR) {
                    const int ns = p.n_streams;
                    if (i != tid) {
#pragma unroll
                        for (int k = 0; k < B200_MAX_STREAMS; ++k) old[k] = k < ns ? p.d_streams_in[k * p.streams_in_stride + row] : 0.0f;
                    }
                    float next = 0.0f;
                    for (int to = 0; to < ns; ++to) {
                        float a = s_conn[ns * ns + to] * y;
#pragma unroll
                        for (int k = 0; k < B200_MAX_STREAMS; ++k)
                            if (k < ns) a = fmaf(s_conn[k * ns + to], old[k], a);
                        p.d_streams_out[to * p.streams_out_stride + row] = a;
                        next = fmaf(s_conn[ns * ns + ns + to], a, next);
                    }
                    p.d_out[0][p.out_offset + row] = next;
                }
            } else {
                if (EXT && p.softcap > 0.0f) y = p.softcap * tanhf(y / p.softcap);
                if (STR && p.act == B200_ACT_RELU2) y = act_relu2(y);
                for (int q = 0; q < p.n_out; ++q) p.d_out[q][p.out_offset + row] = y;
                if (better(y, row, best_v, best_i)) { best_v = y; best_i = row; }
            }
        }
    }

    if (!p.d_ticket) return;

    // ---------------- last-block bookkeeping ----------------
    if (p.d_argmax_scratch) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best_v, o);
            const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
            if (better(ov, oi, best_v, best_i)) { best_v = ov; best_i = oi; }
        }
        if (lane == 0) { am_v[tid >> 5] = best_v; am_i[tid >> 5] = best_i; }
    }
    // The barrier orders every thread's stores (peers' slots included) before thread 0; its system-wide
    // fence is cumulative, so one fence per block publishes them all before the ticket is taken.
    named_barrier(1, nC);
    if (tid == 0) {
        __threadfence_system();
        if (p.d_argmax_scratch) {
            float bv = am_v[0]; int bi = am_i[0];
            for (int k = 1; k < nC / 32; ++k) if (better(am_v[k], am_i[k], bv, bi)) { bv = am_v[k]; bi = am_i[k]; }
            p.d_argmax_scratch[2 * blockIdx.x] = bv;
            reinterpret_cast<int *>(p.d_argmax_scratch)[2 * blockIdx.x + 1] = bi;
            __threadfence();
        }
        s_last = (atomicAdd(p.d_ticket, 1u) == gridDim.x - 1);
    }
    named_barrier(1, nC);
    if (!s_last || tid >= 32) return;
    __threadfence_system();
    {
        float bv = -INFINITY; int bi = 0x7fffffff;
        if (p.d_argmax_scratch) {
            for (int b = lane; b < (int)gridDim.x; b += 32) {
                const float v = *reinterpret_cast<volatile float *>(p.d_argmax_scratch + 2 * b);
                const int i = *reinterpret_cast<volatile int *>(p.d_argmax_scratch + 2 * b + 1);
                if (better(v, i, bv, bi)) { bv = v; bi = i; }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
            }
            if (bi == 0x7fffffff) bi = 0;         // nothing compared greater (all NaN): index 0, as the reference's loop
            bi += (int)p.out_offset;              // global row index of a sharded matrix
            if (lane < p.n_argmax_out) { p.d_argmax_val[lane][0] = bv; p.d_argmax_idx[lane][0] = bi; }
        }
        __syncwarp();
        if (lane == 0) {
            const int pos = p.d_pos_rw ? *p.d_pos_rw : 0;
            if (p.d_next_token && pos + 1 >= *p.d_prompt_len) p.d_next_token[pos + 1] = bi;
            if (p.advance_pos) *p.d_pos_rw = pos + 1;
            const unsigned ep = p.d_epoch ? *p.d_epoch : 0u;
            if (p.advance_epoch) *p.d_epoch_rw = ep + 1u;
            *p.d_ticket = 0u;
            if (p.n_signal > 0) {
                __threadfence_system();
                const unsigned want = ep * (unsigned)p.epoch_mul + (unsigned)p.epoch_add;
                for (int q = 0; q < p.n_signal; ++q) st_release_sys(p.d_signal_flags[q] + p.signal_index, want);
            }
        }
    }
}

// Bytes of shared memory beside the ring: barriers, sums of norms, arg-max, the input vector, the warps' sums of `part` floats.
inline size_t beside_ring(int xs, int part) { return 256 + (256 + 64 + (size_t)xs + part) * sizeof(float); }

template <int WT, int SPT, int RB, int MAXT, int FAM>
int launch(const b200_matvec_args &a, Geometry geo, int grid, cudaStream_t st)
{
    const int ralign = a.out_mode == B200_OUT_GLU ? 2 : 1;
    const int nst = ((geo.base + (geo.rem > 0)) * ralign + RB - 1) / RB;                  // of the block with the most rows
    // windows of about 2048 warp sums
    const int nwgp = (geo.T / 32) | 1, round = geo.NG * RB * nwgp;
    geo.per_warp = (65536 + geo.T / 32 - 1) / (geo.T / 32);
    geo.win = (2048 / round < 1 ? 1 : 2048 / round) * geo.NG;
    if (geo.win > nst) geo.win = (nst + geo.NG - 1) / geo.NG * geo.NG;
    geo.part = geo.win * RB * nwgp;
    const size_t smem = (size_t)geo.nstage * geo.slot_bytes + beside_ring(geo.xs, geo.part * (nst > geo.win ? 2 : 1));
    auto kern = matvec_kernel<WT, SPT, RB, MAXT, FAM>;
    if (smem > 224 * 1024) return B200_E_TOOLARGE;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(geo.NG * geo.T + 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = a.use_pdl ? 1 : 0;
    ++g_b200_launches;
    return (int)cudaLaunchKernelEx(&cfg, kern, a, geo);
}

template <int WT, int SPT, int RB, int FAM>
int launch_by_size(const b200_matvec_args &a, const Geometry &geo, int grid, cudaStream_t st)
{
    const int threads = geo.NG * geo.T + 32;
    if (threads <= 672) return launch<WT, SPT, RB, 672, FAM>(a, geo, grid, st);
    return launch<WT, SPT, RB, 1024, FAM>(a, geo, grid, st);
}

template <int WT, int SPT, int FAM = FAM_PLAIN>
int launch_by_rows(const b200_matvec_args &a, const Geometry &geo, int rb, int grid, cudaStream_t st)
{
    switch (rb) {
    case 8: return launch_by_size<WT, SPT, 8, FAM>(a, geo, grid, st);
    case 4: return launch_by_size<WT, SPT, 4, FAM>(a, geo, grid, st);
    case 2: return launch_by_size<WT, SPT, 2, FAM>(a, geo, grid, st);
    default: return launch_by_size<WT, SPT, 1, FAM>(a, geo, grid, st);
    }
}


// BF16 / F32 weights
template <int FAM>
int launch_typed(const b200_matvec_args &a, const Geometry &geo, int spt, int rb, int grid, cudaStream_t st)
{
    if (a.wtype == B200_WT_BF16)
        return spt == 1 ? launch_by_rows<B200_WT_BF16, 1, FAM>(a, geo, rb, grid, st) : launch_by_rows<B200_WT_BF16, 2, FAM>(a, geo, rb, grid, st);
    return spt == 1 ? launch_by_rows<B200_WT_F32, 1, FAM>(a, geo, rb, grid, st)
         : spt == 2 ? launch_by_rows<B200_WT_F32, 2, FAM>(a, geo, rb, grid, st) : launch_by_rows<B200_WT_F32, 4, FAM>(a, geo, rb, grid, st);
}
int launch_ext(const b200_matvec_args &a, const Geometry &geo, int spt, int rb, int grid, cudaStream_t st);        // matvec_ext.cu
int launch_ext_plain(const b200_matvec_args &a, const Geometry &geo, int spt, int rb, int grid, cudaStream_t st);  // matvec_ext_plain.cu
int launch_streams(const b200_matvec_args &a, const Geometry &geo, int spt, int rb, int grid, cudaStream_t st);    // matvec_streams.cu

} // namespace b200_mv
