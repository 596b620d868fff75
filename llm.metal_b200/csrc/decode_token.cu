// b200_token_plan, b200_token_chunks, b200_decode_token: geometry and launches of the whole-token kernel in decode_token_core.cuh.
#include "decode_token_core.cuh"

#include <stdlib.h>

int b200_tk_launch_narrow(const b200_token_args &a, cudaStream_t st);       // decode_token_narrow.cu

namespace {

constexpr int NARROW_CONSUMERS = 320;

int g_tk_sm_count = 0;

int tk_sm_count()
{
    if (!g_tk_sm_count) {
        int dev = 0, n = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
            return 0;
        g_tk_sm_count = n;
    }
    return g_tk_sm_count;
}

int plan_stage(b200_stage_geom &g, int wtype, int n_blocks, int xin_floats, int consumers)
{
    if (g.rows <= 0 || g.cols <= 0 || g.row_stride <= 0 || (g.row_stride % 16)) return B200_E_BADARG;
    if (wtype == B200_WT_Q8 ? (g.cols % 32) : (g.cols % 8)) return B200_E_BADARG;
    if (g.row_stride < (long long)b200_packed_row_stride(wtype, g.cols)) return B200_E_BADARG;
    const int ralign = g.glu ? 2 : 1;
    if (g.rows % ralign) return B200_E_BADARG;
    const int E = wtype == B200_WT_Q8 ? 16 : 8;
    const int nsl = (g.cols + E - 1) / E;
    // One 16-byte slice per thread as long as the threads suffice; two per thread beyond that, for binary16 rows only
    // (Q8_0 rows of more than 10240 columns are refused: the caller keeps its per-stage kernels).
    g.spt = nsl <= consumers ? 1 : 2;
    if (g.spt == 2 && wtype == B200_WT_Q8) return B200_E_TOOLARGE;
    g.T = (((nsl + g.spt - 1) / g.spt) + 31) / 32 * 32;
    if (g.T > consumers) return B200_E_TOOLARGE;
    g.NG = consumers / g.T;
    if (g.NG > consumers / 32) g.NG = consumers / 32;
    // a chunk (one ring slot) holds rg rows for each group: as many as fit, a power of two up to 8
    // (2 with two slices per thread: the row partials of a chunk live in registers)
    const int fit = (int)(TK_SLOT_BYTES / g.row_stride);          // rows per slot
    if (fit < ralign) return B200_E_TOOLARGE;
    while (g.NG > 1 && g.NG * ralign > fit) --g.NG;               // a slot must hold at least one row (pair) per group
    int rg = g.spt == 1 ? 8 : 2;
    while (rg > ralign && rg * g.NG > fit) rg >>= 1;
    if (rg * g.NG > fit || rg < ralign) return B200_E_TOOLARGE;
    g.rg = rg;
    g.rb = rg * g.NG;
    const int nwgp = (g.T / 32) | 1;
    int pw = TK_PART / nwgp;                           // rows whose warp partials fit one buffer
    pw -= pw % g.rb;                                   // whole chunks in a full window
    if (pw < g.rb) return B200_E_TOOLARGE;
    g.pw = pw;
    const int units = g.rows / ralign;
    g.cta_base = units / n_blocks;
    g.cta_rem = units % n_blocks;
    if (g.cols > xin_floats) return B200_E_TOOLARGE;   // the input vector is held in shared memory once per block
    g.direct_in = 0;
    return 0;
}

} // namespace

extern "C" int b200_token_plan(b200_token_args *a, int n_blocks)
{
    if (!a || a->n_layers <= 0 || a->d_model <= 0 || (a->d_model % 4)) return B200_E_BADARG;
    if (a->wtype != B200_WT_Q8 && a->wtype != B200_WT_F16) return B200_E_BADARG;
    if (a->n_kv <= 0 || a->n_q <= 0 || a->n_q % a->n_kv || (a->hd != 64 && a->hd != 128 && a->hd != 256)) return B200_E_BADARG;
    const int G = a->n_q / a->n_kv;
    if (G != 1 && G != 2 && G != 4 && G != 8) return B200_E_BADARG;
    if (a->n_ranks < 1 || a->n_ranks > B200_MAX_PEERS || a->rank < 0 || a->rank >= a->n_ranks) return B200_E_BADARG;
    if (n_blocks <= 0) n_blocks = tk_sm_count();
    if (n_blocks <= 0) return B200_E_STATE;
    // Consumer threads: half of them where every row has a thread per 16-byte slice then, and a layer is at most 96 KB of weights a block.
    // us a token of four layers, wide and narrow, by those KB: Q8_0 21 86.5 / 77.0, 32 86.9 / 79.2, 77 89.2 / 85.0; F16 40 77.6 / 68.6, 60 78.8 / 70.4,
    // 145 87.1 / 86.5; beyond, rows are what takes the time: Qwen3-4B Q8_0, 720, 156 and 180.
    // Heads in groups of eight need a warp for each; LLMB200_TK_NARROW = 0 / 1 chooses, for experiments.
    a->consumers = TK_NC;
    if (a->n_ranks == 1 && G <= 4) {
        const int E = a->wtype == B200_WT_Q8 ? 16 : 8;
        long long bytes = 0;
        bool fits = true;
        for (int k = 0; k < B200_ST_KINDS; ++k) {
            fits = fits && (a->g[k].cols + E - 1) / E <= NARROW_CONSUMERS;
            if (k != B200_ST_LM) bytes += a->g[k].rows * a->g[k].row_stride;
        }
        const char *e = getenv("LLMB200_TK_NARROW");
        if (fits && (e ? atoi(e) > 0 : bytes <= 96 * 1024LL * n_blocks)) a->consumers = NARROW_CONSUMERS;
    }
    // sequence splits: items (kv head, split) must fit the blocks; at least 32 cache rows per split at full
    // length; by default few enough that the block merging a head reads little (18, or 9 for wide heads)
    int ns = a->n_split > 0 ? a->n_split : (a->hd > 128 ? 9 : 18);
    if (ns > n_blocks / a->n_kv) ns = n_blocks / a->n_kv;
    if (ns > (a->max_seq + 31) / 32) ns = (a->max_seq + 31) / 32;
    if (ns > 32) ns = 32;
    if (ns < 1) return B200_E_TOOLARGE;                // more KV heads than blocks
    a->n_split = ns;
    // Shared memory beyond the ring and the fixed areas is one scratch area: the block-wide input vector
    // of the o and down stages, the slot sums of a normalised residual update, and the attention stage's
    // buffers with as many staged cache rows as fit.
    const Layout fixed = make_layout(a->n_layers, a->d_model, 0);
    int scratch = (232448 - 128 - fixed.total) / 4;
    scratch -= scratch % 4;
    const int att_fixed = attention_fixed_floats(G, a->hd, a->consumers == NARROW_CONSUMERS ? 256 : ATT_T);
    const int chunk_cap = (a->max_seq + ns - 1) / ns;
    int keys = scratch > att_fixed ? (scratch - att_fixed) / a->hd : 0;
    if (keys > chunk_cap) keys = chunk_cap;
    if (keys * a->hd < ns * (a->hd + 2) || keys < 1 || scratch < 2 * a->d_model) return B200_E_TOOLARGE;
    a->att_keys = keys;
    int need = att_fixed + keys * a->hd;               // what is actually used: the rest is left to L1
    if (need < 2 * a->d_model) need = 2 * a->d_model;  // slot sums and the stage's norm weights
    for (int k = 0; k < B200_ST_KINDS; ++k) {
        int rc = plan_stage(a->g[k], a->wtype, n_blocks, scratch, a->consumers);
        if (rc) return rc;
        if ((k == B200_ST_O || k == B200_ST_DOWN) && !a->g[k].direct_in && a->g[k].cols > need) need = a->g[k].cols;
    }
    scratch = (need + 3) / 4 * 4;
    if (a->l2_ahead_bytes < 0) a->l2_ahead_bytes = 0;     // default 0: measured slower than leaving the order of HBM requests to the ring
    if (a->g[B200_ST_QKV].cols != a->d_model || a->g[B200_ST_GATEUP].cols != a->d_model || !a->g[B200_ST_GATEUP].glu ||
        a->g[B200_ST_QKV].rows != (a->n_q + 2 * a->n_kv) * a->hd || a->g[B200_ST_O].cols != a->n_q * a->hd ||
        a->g[B200_ST_O].rows != a->d_model || a->g[B200_ST_DOWN].rows != a->d_model ||
        a->g[B200_ST_DOWN].cols != a->g[B200_ST_GATEUP].rows / 2 || a->g[B200_ST_QKV].glu || a->g[B200_ST_O].glu ||
        a->g[B200_ST_DOWN].glu || a->g[B200_ST_LM].cols != a->d_model || a->g[B200_ST_LM].glu)
        return B200_E_BADARG;
    a->scratch_floats = scratch;
    a->n_blocks = n_blocks;
    const Layout lo = make_layout(a->n_layers, a->d_model, scratch);
    a->smem_bytes = lo.total;
    if (a->smem_bytes > 232448) return B200_E_TOOLARGE;
    return 0;
}

extern "C" int b200_token_chunks(const b200_token_args *a, int kind, int block, int *out, int cap)
{
    if (!a || kind < 0 || kind >= B200_ST_KINDS || block < 0 || block >= a->n_blocks) return B200_E_BADARG;
    const b200_stage_geom &G = a->g[kind];
    const RowRange br = block_rows(G, block);
    int n = 0;
    for (int w0 = br.r0; w0 < br.r1; w0 += G.pw) {
        const int w1 = w0 + G.pw < br.r1 ? w0 + G.pw : br.r1;
        for (int row0 = w0; row0 < w1; row0 += G.rb) {
            if (out && n < cap) { out[3 * n] = row0; out[3 * n + 1] = min(G.rb, w1 - row0); out[3 * n + 2] = (w0 - br.r0) / G.pw; }
            ++n;
        }
    }
    return n;
}

extern "C" int b200_decode_token(const b200_token_args *ap, void *stream)
{
    if (!ap || !ap->d_layers || !ap->d_pos || !ap->d_tokens || !ap->d_prompt_len || !ap->d_epoch || !ap->d_err || !ap->d_emb ||
        !ap->d_qkv || !ap->d_attn_part || !ap->d_attn_out || !ap->d_act || !ap->d_slots_o || !ap->d_slots_dn || !ap->d_counters)
        return B200_E_BADARG;
    if (ap->n_blocks <= 0 || ap->smem_bytes <= 0 || ap->scratch_floats <= 0) return B200_E_STATE;   // b200_token_plan first
    if (ap->with_lm && (!ap->w_lm || !ap->g_final || !ap->d_logits || !ap->d_am || ap->g[B200_ST_LM].rows <= 0)) return B200_E_BADARG;
    if (ap->n_ranks > 1 && ap->with_lm && !ap->d_am_rank) return B200_E_BADARG;
    if (ap->n_tokens < 0 || (ap->n_tokens > 1 && (!ap->with_lm || ap->n_ranks > 1))) return B200_E_BADARG;
    for (int q = 0; q < ap->n_ranks; ++q)
        if (!ap->d_peer_slots_o[q] || !ap->d_peer_slots_dn[q] || !ap->d_peer_counters[q] || (ap->n_ranks > 1 && ap->with_lm && !ap->d_peer_am[q])) return B200_E_BADARG;
    if (ap->n_kv * ap->n_split > ap->n_blocks || B200_CNT_PART + ap->n_kv > 72) return B200_E_BADARG;
    const int sms = tk_sm_count();
    if (sms <= 0) return B200_E_STATE;
    if (ap->n_blocks > sms) return B200_E_TOOLARGE;    // all blocks must be resident at once
    if (ap->consumers == NARROW_CONSUMERS) { ++g_b200_launches; return b200_tk_launch_narrow(*ap, (cudaStream_t)stream); }
    void (*kern)(const b200_token_args);
    const bool multi = ap->n_ranks > 1, trace = ap->d_trace != nullptr;
#define TK_PICK(WT_) (multi ? (trace ? decode_token_kernel<WT_, true, true> : decode_token_kernel<WT_, false, true>) \
                            : (trace ? decode_token_kernel<WT_, true, false> : decode_token_kernel<WT_, false, false>))
    kern = ap->wtype == B200_WT_Q8 ? TK_PICK(B200_WT_Q8) : TK_PICK(B200_WT_F16);
#undef TK_PICK
    ++g_b200_launches;
    return launch_token(kern, *ap, (cudaStream_t)stream);
}
