/* Prompts of the Qwen3 / Gemma3 block in passes over the weights (see plain_rows.h).
 *
 * Token by token a prompt costs one read of all weights per token; here a pass of up to `cap` tokens reads them once, and the
 * products run on the tensor cores at the precision of the per-token kernels (b200_rows_matmul). Ten launches a layer:
 * norm, q/k/v product, heads and cache rows, attention, operand planes, o product, norm, gate/up product, activation, down product. */
#include "plain_rows.h"
#include "../../include/llmb200_train_kernels.h"

#include <string.h>

static const float RMS_EPS = 1e-6f;            /* hard-wired in the reference: src/nn/fast_inference.c:383 */

/* One allocation: the buffers lie in it one after the other, on 256-byte boundaries. 0, 1 when memory has no room, or -1. */
static int allocate(PlainRows *r)
{
    const size_t n = (size_t)r->cap, heads = (size_t)r->Hq * r->hd;
    size_t widest = (size_t)(r->IS > r->D ? r->IS : r->D), total = 0;
    if (heads > widest) widest = heads;
    const struct { void **at; size_t bytes; } part[] = {
        { (void **)&r->x, n * r->D * 4 }, { (void **)&r->y, n * r->D * 4 }, { (void **)&r->last, n * r->D * 4 },
        { (void **)&r->qkv, n * (heads + 2 * (size_t)r->Hkv * r->hd) * 4 }, { (void **)&r->attn, n * heads * 4 },
        { (void **)&r->gu, n * 2 * r->IS * 4 }, { (void **)&r->x_scale, n * 4 }, { (void **)&r->q_scale, n * r->Hq * 4 },
        { &r->xh, n * widest * 2 * r->planes }, { &r->q, n * heads * 2 * 2 } };
    for (size_t i = 0; i < sizeof(part) / sizeof(part[0]); ++i) total += (part[i].bytes + 255) / 256 * 256;
    const cudaError_t e = cudaMalloc(&r->block, total);
    if (e != cudaSuccess) {
        cudaGetLastError();                          /* the caller may go on without: no launch is to report this */
        r->block = NULL;
        return e == cudaErrorMemoryAllocation ? 1 : -1;
    }
    char *at = r->block;
    for (size_t i = 0; i < sizeof(part) / sizeof(part[0]); ++i) { *part[i].at = at; at += (part[i].bytes + 255) / 256 * 256; }
    return 0;
}

int llmb200_plain_rows_fit(PlainRows *r, int want, int least)
{
    if (r->cap >= want) return 0;
    CU_TRY(cudaStreamSynchronize(g_rt.stream), return -1);
    llmb200_plain_rows_free(r);
    for (int cap = want;; cap = cap / 2 > least ? cap / 2 : least) {
        r->cap = cap;
        const int rc = allocate(r);
        if (rc == 0) return 0;
        r->cap = 0;
        if (rc < 0 || cap <= least) return rc;
    }
}

void llmb200_plain_rows_free(PlainRows *r)
{
    cudaFree(r->block);
    r->block = NULL;
    r->cap = 0;
}

static b200_row_planes planes_of(const PlainRows *r, int width)
{
    b200_row_planes p = { r->xh, width, r->planes, r->cap, r->planes == 2 ? r->x_scale : NULL };
    return p;
}

int llmb200_plain_rows_product(PlainRows *r, const RowsMatrix *m, int n, float *out)
{
    if (r->planes == 1 && r->wtype == B200_WT_F16 && n > 128) {          /* plain binary16 operands: the large form, 1.7 times as fast at 2048 rows */
        b200_gemm_args g;
        memset(&g, 0, sizeof(g));
        g.A = r->xh; g.a_row = m->cols; g.a_col = 1;
        g.B = m->w; g.b_row = 1; g.b_col = m->stride / 2;
        g.C = out; g.ldc = m->rows; g.M = n; g.N = m->rows; g.K = m->cols; g.alpha = 1.0f;
        g.d_err = r->d_err;
        K_TRY(b200_gemm_f16(&g, g_rt.stream), return -1);
        return 0;
    }
    b200_rows_matmul_args a;
    memset(&a, 0, sizeof(a));
    a.wtype = r->wtype;
    a.d_w = m->w; a.w_stride = m->stride; a.rows = m->rows; a.cols = m->cols; a.d_w_scale = m->scale;
    a.d_x = r->xh; a.x_ld = m->cols; a.planes = r->planes; a.plane_rows = r->cap;
    a.d_x_scale = r->planes == 2 ? r->x_scale : NULL;
    a.n = n;
    a.d_out = out; a.out_ld = m->rows;
    a.d_err = r->d_err;
    a.use_pdl = 1;
    K_TRY(b200_rows_matmul(&a, g_rt.stream), return -1);
    return 0;
}

int llmb200_plain_rows_run(PlainRows *r, const RowsLayer *layers, int n_layers, int n_rows, int seq_len, int pos0, long long cache_seq_stride,
                           const int *index, int n_last)
{
    void *st = g_rt.stream;
    const int heads = r->Hq * r->hd;
    const b200_row_planes p_model = planes_of(r, r->D), p_heads = planes_of(r, heads), p_inter = planes_of(r, r->IS);
    for (int l = 0; l < n_layers; ++l) {
        const RowsLayer *y = &layers[l];
        const float *post = l && r->gemma ? layers[l - 1].g_post_ff : NULL;
        K_TRY(b200_rows_norm_planes(r->x, n_rows, r->D, l ? r->y : NULL, post, y->g_input, NULL, RMS_EPS, &p_model, st), return -1);
        if (llmb200_plain_rows_product(r, &y->qkv, n_rows, r->qkv)) return -1;
        b200_rows_attn_args a;
        memset(&a, 0, sizeof(a));
        a.n_q = r->Hq; a.n_kv = r->Hkv; a.hd = r->hd; a.max_seq = r->max_seq;
        a.n_rows = n_rows; a.seq_len = seq_len; a.pos0 = pos0; a.eps = RMS_EPS;
        a.d_qkv = r->qkv; a.d_q_gamma = y->g_qn; a.d_k_gamma = y->g_kn; a.d_inv_freq = y->inv_freq;
        a.d_k_cache = y->k_cache; a.d_v_cache = y->v_cache; a.cache_seq_stride = cache_seq_stride;
        a.d_q = r->q; a.d_q_scale = r->q_scale; a.d_out = r->attn;
        K_TRY(b200_rows_attn(&a, st), return -1);
        float *x = r->x, *attn = r->attn;
        if (l == n_layers - 1) {
            if (n_last == 0) return 0;
            /* attention rows go where the query planes were: as many bytes */
            K_TRY(b200_rows_gather(r->x, n_last, r->D, index, r->last, st), return -1);
            K_TRY(b200_rows_gather(r->attn, n_last, heads, index, r->q, st), return -1);
            x = r->last; attn = r->q;
            n_rows = n_last;
        }
        K_TRY(b200_rows_split_planes(attn, n_rows, heads, &p_heads, st), return -1);
        if (llmb200_plain_rows_product(r, &y->o, n_rows, r->y)) return -1;
        K_TRY(b200_rows_norm_planes(x, n_rows, r->D, r->y, r->gemma ? y->g_post_attn : NULL, r->gemma ? y->g_pre_ff : y->g_post_attn,
                                    NULL, RMS_EPS, &p_model, st), return -1);
        if (llmb200_plain_rows_product(r, &y->gateup, n_rows, r->gu)) return -1;
        K_TRY(b200_rows_glu_planes(r->gu, n_rows, r->IS, r->pairs, r->gemma, &p_inter, st), return -1);
        if (llmb200_plain_rows_product(r, &y->down, n_rows, r->y)) return -1;
    }
    return 0;
}

int llmb200_plain_rows_last(PlainRows *r, const RowsLayer *last_layer, const float *g_final, int first, int n)
{
    const b200_row_planes p = planes_of(r, r->D);
    const size_t at = (size_t)first * r->D;
    K_TRY(b200_rows_norm_planes(r->last + at, n, r->D, r->y + at, r->gemma ? last_layer->g_post_ff : NULL, g_final, NULL, RMS_EPS, &p, g_rt.stream), return -1);
    return 0;
}
