/* TEST INFRASTRUCTURE ONLY -- never linked into, imported by, or executed from
 * the product path (hip_llama.cpp_b200/, include/).  Allowed consumers: tests/,
 * __graft_entry__.smoke(), bench.py's cpu_baseline / --impl reference legs.
 *
 * CPU restatement (plain C, scalar, sequential sums) of the llama2 forward pass
 * that the reference runs on the host:
 *   fp32 : run.cc:196-374  (== src/seq.cpp:3-183)
 *   Q8_0 : runq.c:139-171, 317-481
 *   files: run.cc:110-161 (legacy v0), runq.c:174-251 (v2), writer train/export.py
 * Parity pinned: tests/test_oracle_vs_ref.py compares every function here
 * bit-for-bit with oracle/_ref (the reference sources compiled unmodified) and
 * with the committed fixtures in tests/golden/ (generated by the reference's own
 * train/export.py + run.cc/runq.c, see tests/golden/make_golden.py).
 *
 * Build with -ffp-contract=off: every sum below is meant to be evaluated in the
 * written order with one rounding per operation, as the -O2 reference build does.
 */
#include <fcntl.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>
#include <sys/stat.h>
#include <unistd.h>

typedef struct {
    int dim, hidden_dim, n_layers, n_heads, n_kv_heads, vocab_size, seq_len;
} orc_config;

typedef struct { const int8_t* q; const float* s; } orc_qmat;  /* runq.c:34-37 */

typedef struct {
    orc_config cfg;
    int quantized;          /* 0: legacy fp32 file, 1: version-2 Q8_0 file */
    int group_size;         /* GS, runq.c:21 */
    int shared_classifier;
    void* map; size_t map_len;
    /* fp32 tensors (both formats) */
    const float *rms_att, *rms_ffn, *rms_final;
    /* fp32 format */
    const float *tok_emb, *wq, *wk, *wv, *wo, *w1, *w2, *w3, *wcls;
    /* Q8_0 format: one (q, s) pair per layer for the layer matrices */
    orc_qmat q_tok, q_cls, *qwq, *qwk, *qwv, *qwo, *qw1, *qw2, *qw3;
    float* tok_emb_deq;     /* runq.c:205-206 dequantised embedding table */
    int act_bf16;           /* bf16 model path: every vector entering a weight matmul is rounded to bf16 first */
    int attn_bf16;          /* ... and prompt positions run the tensor-core attention rule (orc_attention_bf16_tiled) */
} orc_model;

typedef struct {
    float *x, *xb, *xb2, *hb, *hb2, *q, *att, *logits, *key_cache, *value_cache;
    int8_t *xq, *hq; float *xs, *hs;  /* quantised activations + group scales */
} orc_seq;

/* ---------------------------------------------------------------- ops ---- */

/* run.cc:196-209 / runq.c:282-295 */
void orc_rmsnorm(float* out, const float* x, const float* weight, int n) {
    float acc = 0.0f;
    for (int i = 0; i < n; i++) acc += x[i] * x[i];
    acc /= n;
    acc += 1e-5f;
    acc = 1.0f / sqrtf(acc);
    for (int i = 0; i < n; i++) out[i] = weight[i] * (acc * x[i]);
}

/* run.cc:211-229 */
void orc_softmax(float* x, int n) {
    float m = x[0];
    for (int i = 1; i < n; i++) if (x[i] > m) m = x[i];
    float denom = 0.0f;
    for (int i = 0; i < n; i++) { x[i] = expf(x[i] - m); denom += x[i]; }
    for (int i = 0; i < n; i++) x[i] /= denom;
}

/* run.cc:231-242: out[d] = W[d,n] . x[n], one sequential sum per row */
void orc_matmul_f32(float* out, const float* x, const float* w, int n, int d) {
    for (int r = 0; r < d; r++) {
        const float* row = w + (size_t)r * n;
        float acc = 0.0f;
        for (int c = 0; c < n; c++) acc += row[c] * x[c];
        out[r] = acc;
    }
}

/* run.cc:271-286: rotate consecutive pairs of q (all) and k (first kv_dim) */
void orc_rope(float* q, float* k, int dim, int kv_dim, int head_size, int pos) {
    for (int i = 0; i < dim; i += 2) {
        int j = i % head_size;
        float freq = 1.0f / powf(10000.0f, j / (float)head_size);
        float ang = pos * freq;
        float c = cosf(ang), s = sinf(ang);
        float a = q[i], b = q[i + 1];
        q[i] = a * c - b * s;
        q[i + 1] = a * s + b * c;
        if (i < kv_dim) {
            a = k[i]; b = k[i + 1];
            k[i] = a * c - b * s;
            k[i + 1] = a * s + b * c;
        }
    }
}

/* run.cc:288-326: per head scores / softmax / weighted V sum.  kc, vc point at
 * this layer's [seq_len, kv_dim] slab. */
void orc_attention(float* out, float* att, const float* q, const float* kc, const float* vc,
                   int pos, int n_heads, int kv_mul, int head_size, int kv_dim, int seq_len) {
    for (int h = 0; h < n_heads; h++) {
        const float* qh = q + h * head_size;
        float* a = att + (size_t)h * seq_len;
        int koff = (h / kv_mul) * head_size;
        for (int t = 0; t <= pos; t++) {
            const float* kt = kc + (size_t)t * kv_dim + koff;
            float sc = 0.0f;
            for (int i = 0; i < head_size; i++) sc += qh[i] * kt[i];
            sc /= sqrtf(head_size);
            a[t] = sc;
        }
        orc_softmax(a, pos + 1);
        float* o = out + h * head_size;
        memset(o, 0, head_size * sizeof(float));
        for (int t = 0; t <= pos; t++) {
            const float* vt = vc + (size_t)t * kv_dim + koff;
            float p = a[t];
            for (int i = 0; i < head_size; i++) o[i] += p * vt[i];
        }
    }
}

/* The rule of the tensor-core prompt attention of the bf16 path (hip_llama.cpp_b200/csrc/attn_prefill_tc.cu), restated:
 * the scores and sums of run.cc:288-321 with q, k, v rounded to bf16, keys visited in tiles of 128 from key 0 with an
 * online softmax; per tile p = exp(s - m_new) is rounded to bf16 for the P V product while the running sum keeps the
 * unrounded p; everything else fp32.  (Mathematically the attention of run.cc; the roundings are the tensor cores'.) */
static float orc_bf16r(float x) {
    uint32_t u; memcpy(&u, &x, 4);
    if ((u & 0x7FFFFFFFu) <= 0x7F800000u) u = (u + 0x7FFFu + ((u >> 16) & 1u)) & 0xFFFF0000u;
    memcpy(&x, &u, 4);
    return x;
}
void orc_attention_bf16_tiled(float* out, const float* q, const float* kc, const float* vc,
                              int pos, int n_heads, int kv_mul, int head_size, int kv_dim) {
    const float scale = 1.4426950408889634f / sqrtf((float)head_size);
    float sc[128], acc[256];
    for (int h = 0; h < n_heads; h++) {
        const float* qh = q + h * head_size;
        int koff = (h / kv_mul) * head_size;
        float m = -INFINITY, l = 0.0f;
        for (int i = 0; i < head_size; i++) acc[i] = 0.0f;
        for (int t0 = 0; t0 <= pos; t0 += 128) {
            int nt = pos - t0 + 1 < 128 ? pos - t0 + 1 : 128;
            float mt = -INFINITY;
            for (int j = 0; j < nt; j++) {
                const float* kt = kc + (size_t)(t0 + j) * kv_dim + koff;
                float s = 0.0f;
                for (int i = 0; i < head_size; i++) s += orc_bf16r(qh[i]) * orc_bf16r(kt[i]);
                sc[j] = s * scale;
                if (sc[j] > mt) mt = sc[j];
            }
            float mn = m > mt ? m : mt;
            float corr = exp2f(m - mn);
            float ls = 0.0f;
            for (int i = 0; i < head_size; i++) acc[i] *= corr;
            for (int j = 0; j < nt; j++) {
                float p = exp2f(sc[j] - mn);
                ls += p;
                float pb = orc_bf16r(p);
                const float* vt = vc + (size_t)(t0 + j) * kv_dim + koff;
                for (int i = 0; i < head_size; i++) acc[i] += pb * orc_bf16r(vt[i]);
            }
            l = l * corr + ls;
            m = mn;
        }
        float* o = out + h * head_size;
        float inv = 1.0f / l;
        for (int i = 0; i < head_size; i++) o[i] = acc[i] * inv;
    }
}

/* run.cc:342-349 */
void orc_swiglu(float* hb, const float* hb2, int n) {
    for (int i = 0; i < n; i++) {
        float v = hb[i];
        v *= (1.0f / (1.0f + expf(-v)));
        v *= hb2[i];
        hb[i] = v;
    }
}

/* run.cc:619-630: first maximum wins (strict >) */
int orc_argmax(const float* p, int n) {
    int best = 0; float bv = p[0];
    for (int i = 1; i < n; i++) if (p[i] > bv) { bv = p[i]; best = i; }
    return best;
}

/* runq.c:145-171.  scale = max|x| / 127 (fp32 division), q = (int8) round(x / scale)
 * with C round() = half away from zero.  An all-zero group gives scale 0 and
 * 0/0 = NaN; the C cast of NaN is undefined -- on x86-64 cvttsd2si yields
 * INT_MIN whose low byte is 0, which is what the reference binary produces,
 * and this restatement pins that case to 0. */
void orc_quantize(int8_t* q, float* s, const float* x, int n, int gs) {
    int groups = n / gs;
    for (int g = 0; g < groups; g++) {
        const float* xg = x + g * gs;
        float amax = 0.0f;
        for (int i = 0; i < gs; i++) { float v = fabsf(xg[i]); if (v > amax) amax = v; }
        float scale = amax / 127.0f;
        s[g] = scale;
        for (int i = 0; i < gs; i++) {
            float r = xg[i] / scale;
            q[g * gs + i] = (r != r) ? (int8_t)0 : (int8_t)round(r);
        }
    }
}

/* runq.c:139-143 */
void orc_dequantize(float* x, const int8_t* q, const float* s, int n, int gs) {
    for (int i = 0; i < n; i++) x[i] = q[i] * s[i / gs];
}

/* runq.c:317-342: per group int32 dot, then fp32 scale-accumulate in group order:
 * val += ((float)ival * ws) * xs */
void orc_matmul_q8(float* out, const int8_t* xq, const float* xs, const int8_t* wq,
                   const float* ws, int n, int d, int gs) {
    for (int r = 0; r < d; r++) {
        size_t base = (size_t)r * n;
        float val = 0.0f;
        for (int j = 0; j <= n - gs; j += gs) {
            int32_t iv = 0;
            for (int k = 0; k < gs; k++) iv += (int32_t)xq[j + k] * (int32_t)wq[base + j + k];
            val += ((float)iv) * ws[(base + j) / gs] * xs[j / gs];
        }
        out[r] = val;
    }
}

/* ------------------------------------------------------------ loaders ---- */

static void* map_file(const char* path, size_t* len) {
    int fd = open(path, O_RDONLY);
    if (fd < 0) return NULL;
    struct stat st;
    if (fstat(fd, &st) != 0) { close(fd); return NULL; }
    void* p = mmap(NULL, (size_t)st.st_size, PROT_READ, MAP_PRIVATE, fd, 0);
    close(fd);
    if (p == MAP_FAILED) return NULL;
    *len = (size_t)st.st_size;
    return p;
}

/* Legacy v0 file (run.cc:110-161; writer train/export.py:75-127): 7 x int32
 * Config, then fp32 tensors in the order below.  vocab_size < 0 marks an
 * unshared classifier.  Two dead RoPE tables of seq_len*head_size/2 floats sit
 * between rms_final and wcls. */
orc_model* orc_open_v0(const char* path) {
    orc_model* m = (orc_model*)calloc(1, sizeof(orc_model));
    m->map = map_file(path, &m->map_len);
    if (!m->map) { free(m); return NULL; }
    memcpy(&m->cfg, m->map, sizeof(orc_config));
    m->shared_classifier = m->cfg.vocab_size > 0;
    if (m->cfg.vocab_size < 0) m->cfg.vocab_size = -m->cfg.vocab_size;
    const orc_config* c = &m->cfg;
    size_t L = (size_t)c->n_layers, d = (size_t)c->dim, hd = (size_t)c->hidden_dim;
    size_t hs = d / c->n_heads, kvd = hs * c->n_kv_heads;
    const float* p = (const float*)((const char*)m->map + sizeof(orc_config));
    m->tok_emb = p;  p += (size_t)c->vocab_size * d;
    m->rms_att = p;  p += L * d;
    m->wq = p;       p += L * d * d;
    m->wk = p;       p += L * d * kvd;
    m->wv = p;       p += L * d * kvd;
    m->wo = p;       p += L * d * d;
    m->rms_ffn = p;  p += L * d;
    m->w1 = p;       p += L * d * hd;
    m->w2 = p;       p += L * hd * d;
    m->w3 = p;       p += L * d * hd;
    m->rms_final = p; p += d;
    p += (size_t)c->seq_len * hs / 2;
    p += (size_t)c->seq_len * hs / 2;
    m->wcls = m->shared_classifier ? m->tok_emb : p;
    return m;
}

static orc_qmat* carve_q(const char** cur, int n, size_t each, int gs) {
    orc_qmat* r = (orc_qmat*)malloc(sizeof(orc_qmat) * n);
    for (int i = 0; i < n; i++) {
        r[i].q = (const int8_t*)*cur; *cur += each;
        r[i].s = (const float*)*cur;  *cur += (each / gs) * sizeof(float);
    }
    return r;
}

/* Version-2 file (runq.c:174-251; writer train/export.py:182-260): 256-byte
 * header {u32 magic 0x616b3432, i32 version 2, Config, u8 shared_classifier,
 * i32 group_size}, fp32 norms, then per tensor int8 payload followed by its
 * fp32 group scales. */
orc_model* orc_open_v2(const char* path) {
    orc_model* m = (orc_model*)calloc(1, sizeof(orc_model));
    m->map = map_file(path, &m->map_len);
    if (!m->map) { free(m); return NULL; }
    const char* b = (const char*)m->map;
    uint32_t magic; int32_t version;
    memcpy(&magic, b, 4); memcpy(&version, b + 4, 4);
    if (magic != 0x616b3432u || version != 2) { munmap(m->map, m->map_len); free(m); return NULL; }
    memcpy(&m->cfg, b + 8, sizeof(orc_config));
    uint8_t shared; memcpy(&shared, b + 8 + sizeof(orc_config), 1);
    int32_t gs; memcpy(&gs, b + 8 + sizeof(orc_config) + 1, 4);
    m->quantized = 1; m->group_size = gs; m->shared_classifier = shared;
    const orc_config* c = &m->cfg;
    size_t d = (size_t)c->dim, hd = (size_t)c->hidden_dim;
    size_t hs = d / c->n_heads, kvd = hs * c->n_kv_heads;
    int L = c->n_layers;
    const float* f = (const float*)(b + 256);
    m->rms_att = f; f += (size_t)L * d;
    m->rms_ffn = f; f += (size_t)L * d;
    m->rms_final = f; f += d;
    const char* cur = (const char*)f;
    orc_qmat* tok = carve_q(&cur, 1, (size_t)c->vocab_size * d, gs);
    m->q_tok = tok[0]; free(tok);
    m->qwq = carve_q(&cur, L, d * d, gs);
    m->qwk = carve_q(&cur, L, d * kvd, gs);
    m->qwv = carve_q(&cur, L, d * kvd, gs);
    m->qwo = carve_q(&cur, L, d * d, gs);
    m->qw1 = carve_q(&cur, L, d * hd, gs);
    m->qw2 = carve_q(&cur, L, hd * d, gs);
    m->qw3 = carve_q(&cur, L, d * hd, gs);
    if (shared) m->q_cls = m->q_tok;
    else { orc_qmat* cl = carve_q(&cur, 1, d * (size_t)c->vocab_size, gs); m->q_cls = cl[0]; free(cl); }
    size_t ne = (size_t)c->vocab_size * d;
    m->tok_emb_deq = (float*)malloc(ne * sizeof(float));
    orc_dequantize(m->tok_emb_deq, m->q_tok.q, m->q_tok.s, (int)ne, gs);
    return m;
}

void orc_close(orc_model* m) {
    if (!m) return;
    if (m->map) munmap(m->map, m->map_len);
    free(m->qwq); free(m->qwk); free(m->qwv); free(m->qwo);
    free(m->qw1); free(m->qw2); free(m->qw3); free(m->tok_emb_deq);
    free(m);
}

void orc_get_config(const orc_model* m, int out[9]) {
    out[0] = m->cfg.dim; out[1] = m->cfg.hidden_dim; out[2] = m->cfg.n_layers;
    out[3] = m->cfg.n_heads; out[4] = m->cfg.n_kv_heads; out[5] = m->cfg.vocab_size;
    out[6] = m->cfg.seq_len; out[7] = m->group_size; out[8] = m->shared_classifier;
}

/* run.cc:76-95 / runq.c:91-115 */
orc_seq* orc_seq_new(const orc_model* m) {
    const orc_config* c = &m->cfg;
    size_t kvd = (size_t)c->dim * c->n_kv_heads / c->n_heads;
    orc_seq* s = (orc_seq*)calloc(1, sizeof(orc_seq));
    s->x = (float*)calloc(c->dim, 4);   s->xb = (float*)calloc(c->dim, 4);
    s->xb2 = (float*)calloc(c->dim, 4); s->q = (float*)calloc(c->dim, 4);
    s->hb = (float*)calloc(c->hidden_dim, 4); s->hb2 = (float*)calloc(c->hidden_dim, 4);
    s->att = (float*)calloc((size_t)c->n_heads * c->seq_len, 4);
    s->logits = (float*)calloc(c->vocab_size, 4);
    s->key_cache = (float*)calloc((size_t)c->n_layers * c->seq_len * kvd, 4);
    s->value_cache = (float*)calloc((size_t)c->n_layers * c->seq_len * kvd, 4);
    s->xq = (int8_t*)calloc(c->dim, 1); s->xs = (float*)calloc(c->dim, 4);
    s->hq = (int8_t*)calloc(c->hidden_dim, 1); s->hs = (float*)calloc(c->hidden_dim, 4);
    return s;
}

void orc_seq_free(orc_seq* s) {
    if (!s) return;
    free(s->x); free(s->xb); free(s->xb2); free(s->q); free(s->hb); free(s->hb2);
    free(s->att); free(s->logits); free(s->key_cache); free(s->value_cache);
    free(s->xq); free(s->xs); free(s->hq); free(s->hs); free(s);
}

/* which: 0 x,1 xb,2 xb2,3 hb,4 hb2,5 q,6 att,7 logits,8 key_cache,9 value_cache */
float* orc_seq_ptr(orc_seq* s, int which) {
    switch (which) {
        case 0: return s->x;   case 1: return s->xb;  case 2: return s->xb2;
        case 3: return s->hb;  case 4: return s->hb2; case 5: return s->q;
        case 6: return s->att; case 7: return s->logits;
        case 8: return s->key_cache; case 9: return s->value_cache;
    }
    return NULL;
}
int8_t* orc_seq_q(orc_seq* s, int which) { return which == 0 ? s->xq : s->hq; }
float*  orc_seq_s(orc_seq* s, int which) { return which == 0 ? s->xs : s->hs; }

/* which: 0 tok_emb,1 rms_att,2 rms_ffn,3 wq,4 wk,5 wv,6 wo,7 w1,8 w2,9 w3,10 rms_final,11 wcls */
const float* orc_weight_ptr(const orc_model* m, int which) {
    switch (which) {
        case 0: return m->quantized ? m->tok_emb_deq : m->tok_emb;
        case 1: return m->rms_att; case 2: return m->rms_ffn;
        case 3: return m->wq; case 4: return m->wk; case 5: return m->wv; case 6: return m->wo;
        case 7: return m->w1; case 8: return m->w2; case 9: return m->w3;
        case 10: return m->rms_final; case 11: return m->wcls;
    }
    return NULL;
}

/* ------------------------------------------------------------ forward ---- */

/* The bf16 model path of the B200 library (hip_llama.cpp_b200/csrc/step_bf16.cu) restated: the network of run.cc:244-374
 * on weights that are bf16-representable (the checkpoint is rounded before it is written), with every vector that enters
 * a weight matmul rounded to bf16, round to nearest even -- the operand format of the tensor cores.  Everything else
 * (RMSNorm, RoPE, attention, SwiGLU, residual stream, KV cache) stays fp32 as in run.cc. */
void orc_set_bf16_activations(orc_model* m, int on) { m->act_bf16 = on; }
void orc_set_bf16_attention(orc_model* m, int on) { m->attn_bf16 = on; }
static void round_bf16_vec(float* x, int n) {
    for (int i = 0; i < n; i++) {
        uint32_t u; memcpy(&u, &x[i], 4);
        if ((u & 0x7FFFFFFFu) <= 0x7F800000u) u = (u + 0x7FFFu + ((u >> 16) & 1u)) & 0xFFFF0000u;
        memcpy(&x[i], &u, 4);
    }
}

/* run.cc:244-374: one position of one sequence, fp32 weights */
static float* forward_f32(const orc_model* m, orc_seq* s, int token, int pos) {
    const orc_config* c = &m->cfg;
    int d = c->dim, hd = c->hidden_dim, hs = d / c->n_heads;
    int kvd = d * c->n_kv_heads / c->n_heads, kv_mul = c->n_heads / c->n_kv_heads;
    memcpy(s->x, m->tok_emb + (size_t)token * d, d * sizeof(float));
    for (int l = 0; l < c->n_layers; l++) {
        size_t loff = (size_t)l * c->seq_len * kvd;
        float* krow = s->key_cache + loff + (size_t)pos * kvd;
        float* vrow = s->value_cache + loff + (size_t)pos * kvd;
        orc_rmsnorm(s->xb, s->x, m->rms_att + (size_t)l * d, d);
        if (m->act_bf16) round_bf16_vec(s->xb, d);
        orc_matmul_f32(s->q, s->xb, m->wq + (size_t)l * d * d, d, d);
        orc_matmul_f32(krow, s->xb, m->wk + (size_t)l * d * kvd, d, kvd);
        orc_matmul_f32(vrow, s->xb, m->wv + (size_t)l * d * kvd, d, kvd);
        orc_rope(s->q, krow, d, kvd, hs, pos);
        if (m->attn_bf16 && hs <= 256)
            orc_attention_bf16_tiled(s->xb, s->q, s->key_cache + loff, s->value_cache + loff, pos, c->n_heads, kv_mul, hs, kvd);
        else
            orc_attention(s->xb, s->att, s->q, s->key_cache + loff, s->value_cache + loff,
                          pos, c->n_heads, kv_mul, hs, kvd, c->seq_len);
        if (m->act_bf16) round_bf16_vec(s->xb, d);
        orc_matmul_f32(s->xb2, s->xb, m->wo + (size_t)l * d * d, d, d);
        for (int i = 0; i < d; i++) s->x[i] += s->xb2[i];
        orc_rmsnorm(s->xb, s->x, m->rms_ffn + (size_t)l * d, d);
        if (m->act_bf16) round_bf16_vec(s->xb, d);
        orc_matmul_f32(s->hb, s->xb, m->w1 + (size_t)l * d * hd, d, hd);
        orc_matmul_f32(s->hb2, s->xb, m->w3 + (size_t)l * d * hd, d, hd);
        orc_swiglu(s->hb, s->hb2, hd);
        if (m->act_bf16) round_bf16_vec(s->hb, hd);
        orc_matmul_f32(s->xb, s->hb, m->w2 + (size_t)l * d * hd, hd, d);
        for (int i = 0; i < d; i++) s->x[i] += s->xb[i];
    }
    orc_rmsnorm(s->x, s->x, m->rms_final, d);
    if (m->act_bf16) round_bf16_vec(s->x, d);
    orc_matmul_f32(s->logits, s->x, m->wcls, d, c->vocab_size);
    return s->logits;
}

/* runq.c:344-481: same network, activations re-quantised before every matmul
 * group (:367, :437, :450, :465, :478); K and V are produced into scratch rows,
 * rotated, then copied into the cache (:389-394). */
static float* forward_q8(const orc_model* m, orc_seq* s, int token, int pos) {
    const orc_config* c = &m->cfg;
    int d = c->dim, hd = c->hidden_dim, hs = d / c->n_heads, gs = m->group_size;
    int kvd = d * c->n_kv_heads / c->n_heads, kv_mul = c->n_heads / c->n_kv_heads;
    float* kbuf = (float*)malloc(sizeof(float) * kvd);
    float* vbuf = (float*)malloc(sizeof(float) * kvd);
    memcpy(s->x, m->tok_emb_deq + (size_t)token * d, d * sizeof(float));
    for (int l = 0; l < c->n_layers; l++) {
        size_t loff = (size_t)l * c->seq_len * kvd;
        orc_rmsnorm(s->xb, s->x, m->rms_att + (size_t)l * d, d);
        orc_quantize(s->xq, s->xs, s->xb, d, gs);
        orc_matmul_q8(s->q, s->xq, s->xs, m->qwq[l].q, m->qwq[l].s, d, d, gs);
        orc_matmul_q8(kbuf, s->xq, s->xs, m->qwk[l].q, m->qwk[l].s, d, kvd, gs);
        orc_matmul_q8(vbuf, s->xq, s->xs, m->qwv[l].q, m->qwv[l].s, d, kvd, gs);
        orc_rope(s->q, kbuf, d, kvd, hs, pos);
        memcpy(s->key_cache + loff + (size_t)pos * kvd, kbuf, kvd * sizeof(float));
        memcpy(s->value_cache + loff + (size_t)pos * kvd, vbuf, kvd * sizeof(float));
        orc_attention(s->xb, s->att, s->q, s->key_cache + loff, s->value_cache + loff,
                      pos, c->n_heads, kv_mul, hs, kvd, c->seq_len);
        orc_quantize(s->xq, s->xs, s->xb, d, gs);
        orc_matmul_q8(s->xb2, s->xq, s->xs, m->qwo[l].q, m->qwo[l].s, d, d, gs);
        for (int i = 0; i < d; i++) s->x[i] += s->xb2[i];
        orc_rmsnorm(s->xb, s->x, m->rms_ffn + (size_t)l * d, d);
        orc_quantize(s->xq, s->xs, s->xb, d, gs);
        orc_matmul_q8(s->hb, s->xq, s->xs, m->qw1[l].q, m->qw1[l].s, d, hd, gs);
        orc_matmul_q8(s->hb2, s->xq, s->xs, m->qw3[l].q, m->qw3[l].s, d, hd, gs);
        orc_swiglu(s->hb, s->hb2, hd);
        orc_quantize(s->hq, s->hs, s->hb, hd, gs);
        orc_matmul_q8(s->xb, s->hq, s->hs, m->qw2[l].q, m->qw2[l].s, hd, d, gs);
        for (int i = 0; i < d; i++) s->x[i] += s->xb[i];
    }
    orc_rmsnorm(s->x, s->x, m->rms_final, d);
    orc_quantize(s->xq, s->xs, s->x, d, gs);
    orc_matmul_q8(s->logits, s->xq, s->xs, m->q_cls.q, m->q_cls.s, d, c->vocab_size, gs);
    free(kbuf); free(vbuf);
    return s->logits;
}

float* orc_forward(const orc_model* m, orc_seq* s, int token, int pos) {
    return m->quantized ? forward_q8(m, s, token, pos) : forward_f32(m, s, token, pos);
}

/* One decode step for n independent sequences (the batched semantics of
 * src/thaDNN.cpp:13-81: slot b advances at its own pos[b]); rows are
 * independent so host threads split them (compile with -fopenmp to use it). */
void orc_forward_many(const orc_model* m, orc_seq** seqs, const int* token, const int* pos,
                      int n, int n_threads) {
    (void)n_threads;
#ifdef _OPENMP
#pragma omp parallel for num_threads(n_threads > 0 ? n_threads : 1) schedule(dynamic, 1)
#endif
    for (int i = 0; i < n; i++) orc_forward(m, seqs[i], token[i], pos[i]);
}
