/* Prompts of the Qwen3 / Gemma3 block in passes over the weights (internal): shared by the single-sequence states
 * and the batched engine. */
#ifndef LLMB200_PLAIN_ROWS_H
#define LLMB200_PLAIN_ROWS_H

#include "internal.h"

typedef struct { const void *w; long long stride; int rows, cols; const float *scale; } RowsMatrix;   /* scale: Q8_0 only */

typedef struct {
    RowsMatrix qkv, o, gateup, down;
    const float *g_input, *g_post_attn, *g_pre_ff, *g_post_ff, *g_qn, *g_kn, *inv_freq;
    void *k_cache, *v_cache;
} RowsLayer;

/* Workspace of a pass of up to `cap` rows. planes: 2 where the per-token kernels take fp32 inputs, 1 where they take
 * binary16 ones. */
typedef struct {
    int D, Hq, Hkv, hd, IS, gemma, pairs, wtype, planes, max_seq;
    unsigned *d_err;
    int cap;
    float *x, *y, *last, *qkv, *attn, *gu, *x_scale, *q_scale;
    void *xh, *q;
    void *block;                         /* all of them */
} PlainRows;

/* A workspace for passes of `want` rows (the sizes above cap must be set), or of fewer, down to `least`, where device memory has no more:
 * r->cap says. 0, 1 when not even that could be had, -1 after a device error. What there was before is given back first. */
int llmb200_plain_rows_fit(PlainRows *r, int want, int least);
void llmb200_plain_rows_free(PlainRows *r);
/* Runs n_rows / seq_len sequences' tokens (positions pos0 on) through the layers; r->x holds the embedded rows on entry. What follows the
 * last layer's attention is formed for rows index[0..n_last) (device memory) only: nobody reads it of the others. */
int llmb200_plain_rows_run(PlainRows *r, const RowsLayer *layers, int n_layers, int n_rows, int seq_len, int pos0, long long cache_seq_stride,
                           const int *index, int n_last);
/* The LM head's operand: planes of the final norm of the index-th rows first .. first + n - 1 of the last run -> r->xh. */
int llmb200_plain_rows_last(PlainRows *r, const RowsLayer *last_layer, const float *g_final, int first, int n);
int llmb200_plain_rows_product(PlainRows *r, const RowsMatrix *m, int n, float *out);

#endif
