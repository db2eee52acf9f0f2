// One pass through the layers of a dense decoder (RMS norm, fused qkv, rotation, paged attention, gated MLP) as one call: the launches of a
// step follow one another without the caller's language in between. A step whose kernels take a few microseconds each waits for its launches
// otherwise (37 tokens through four layers of an 8B model: 40 launches, 490 us, of which the kernels 390; from here 3 us a launch).
#include <math.h>

#include "common.cuh"
#include "gemm_common.cuh"

namespace ovb {

static void fill_gemm(ovb_gemm_args* a, const ovb_llm_step* s, const ovb_llm_weight* w, const void* x, void* out, const void* residual, int T, int out_cols) {
    memset(a, 0, sizeof(*a));
    a->x = x;
    a->w = w->w;
    a->out = out;
    a->bias = w->bias;
    a->residual = residual;
    a->scales = w->scales;
    a->ws = s->gemm_ws;
    a->counters = s->gemm_counters;
    a->ws_bytes = s->gemm_ws_bytes;
    a->T = T;
    a->N = w->N;
    a->K = w->K;
    a->ldx = w->K;
    a->ldo = out_cols;
    a->ldr = residual != nullptr ? out_cols : 0;
    a->group_size = w->group_size;
    a->wmode = w->wmode;
    a->act = w->act;
    a->w_tiled = w->w_tiled;
    a->w_kb_stride = w->w_kb_stride;
}

static int64_t scratch_of(const ovb_gemm_args* a) { return is_quant(a->wmode) && a->T >= 1024 ? ovb_gemm_scratch_bytes(a) : 0; }

static int run_gemm(const ovb_llm_step* s, const ovb_llm_weight* w, const void* x, void* out, const void* residual, int T, int out_cols, ovb_stream_t stream) {
    ovb_gemm_args a;
    fill_gemm(&a, s, w, x, out, residual, T, out_cols);
    const int64_t need = scratch_of(&a);
    if (need > 0 && need <= s->scratch_bytes) {
        a.scratch = s->scratch;
        a.scratch_bytes = need;
    }
    return ovb_gemm(&a, stream);
}

// A product of normalised rows (row_idx: of those rows of h): in one launch where the kernel takes the norm in.
static int run_norm_gemm(ovb_llm_step* s, const ovb_llm_weight* w, const void* gamma, const int* row_idx, int h_rows, void* x, void* out, int T, int out_cols,
                         ovb_stream_t stream) {
    ovb_gemm_args a;
    fill_gemm(&a, s, w, s->h, out, nullptr, T, out_cols);
    if ((reinterpret_cast<uintptr_t>(gamma) & 15) == 0 && ovb_gemm_norms(&a)) {
        a.x_norm = gamma;
        a.x_eps = s->eps;
        a.x_rows = row_idx;
        a.x_count = h_rows;
        return ovb_gemm(&a, stream);
    }
    const int rc = row_idx != nullptr ? ovb_rmsnorm_rows(s->h, row_idx, gamma, x, T, w->K, s->eps, h_rows, stream)
                                      : ovb_rmsnorm(s->h, nullptr, gamma, x, nullptr, T, w->K, s->eps, stream);
    if (rc != 0) return rc;
    ++s->launches;
    return run_gemm(s, w, x, out, nullptr, T, out_cols, stream);
}

// The shapes that the buffers of the step were made for.
static int check_layer(const ovb_llm_step* s, const ovb_llm_layer* l, int i) {
    const int q = s->Hq * s->D, rows = (s->Hq + 2 * s->Hkv) * s->D;
    const bool gated = l->gate_up.act == OVB_ACT_SWIGLU;
    OVB_REQUIRE(l->qkv.N == rows && l->qkv.K == s->hidden && l->o.N == s->hidden && l->o.K == q && l->gate_up.N == 2 * s->ffn && l->gate_up.K == s->hidden &&
                    l->down.N == s->hidden && l->down.K == s->ffn,
                "ovb_llm_step: the weights of layer %d do not fit the model (hidden %d, heads %d / %d of %d, ffn %d)", i, s->hidden, s->Hq, s->Hkv, s->D, s->ffn);
    OVB_REQUIRE(gated || l->gate_up.act == OVB_ACT_NONE, "ovb_llm_step: activation %d of layer %d", l->gate_up.act, i);
    return 0;
}

}  // namespace ovb

extern "C" {

int ovb_llm_struct_bytes(int which) { return which == 0 ? (int)sizeof(ovb_llm_weight) : which == 1 ? (int)sizeof(ovb_llm_layer) : (int)sizeof(ovb_llm_step); }

int64_t ovb_llm_scratch_bytes(const ovb_llm_step* s) {
    using namespace ovb;
    int64_t most = 0;
    for (int i = 0; i < s->num_layers; ++i) {
        const ovb_llm_weight* ws[4] = {&s->layers[i].qkv, &s->layers[i].o, &s->layers[i].gate_up, &s->layers[i].down};
        for (const ovb_llm_weight* w : ws) {
            ovb_gemm_args a;
            // (addresses only count by their alignment, which all buffers of a step share)
            fill_gemm(&a, s, w, s->x, s->x, nullptr, s->T, w->act == OVB_ACT_SWIGLU ? w->N / 2 : w->N);
            const int64_t need = scratch_of(&a);
            if (need > most) most = need;
        }
    }
    return most;
}

int ovb_llm_step_run(ovb_llm_step* s, ovb_stream_t stream) {
    using namespace ovb;
    OVB_REQUIRE(s && s->layers && s->T > 0 && s->B > 0, "ovb_llm_step: empty step");
    s->launches = 0;
    const int T = s->T, B = s->B, H = s->hidden, rows = (s->Hq + 2 * s->Hkv) * s->D;
    for (int i = 0; i < s->num_layers; ++i)
        if (int rc = check_layer(s, &s->layers[i], i)) return rc;
    OVB_REQUIRE(s->head.K == H && s->head.N <= s->head_cols, "ovb_llm_step: the vocabulary projection is %d x %d", s->head.N, s->head.K);
#define OVB_STEP(call)             \
    do {                           \
        const int rc_ = (call);    \
        if (rc_ != 0) return rc_;  \
        ++s->launches;             \
    } while (0)
    OVB_STEP(ovb_embed_tokens(s->ids, s->tok_src, s->last_token, s->embed, s->h, T, H, s->vocab, stream));
    for (int i = 0; i < s->num_layers; ++i) {
        const ovb_llm_layer* l = &s->layers[i];
        OVB_STEP(run_norm_gemm(s, &l->qkv, l->norm1, nullptr, T, s->x, s->qkv, T, rows, stream));
        ovb_pa_args pa;
        memset(&pa, 0, sizeof(pa));
        pa.q = s->qkv;
        pa.out = s->attn;
        pa.k_cache = l->k_cache;
        pa.v_cache = l->v_cache;
        pa.past_lens = s->past_lens;
        pa.subsequence_begins = s->subsequence_begins;
        pa.block_indices = s->block_indices;
        pa.block_indices_begins = s->block_indices_begins;
        pa.scratch = ovb_pa_scratch_bytes(B, s->Hq, s->D, s->max_ctx) <= s->pa_scratch_bytes ? s->pa_scratch : nullptr;
        pa.B = B;
        pa.T = T;
        pa.Hq = s->Hq;
        pa.Hkv = s->Hkv;
        pa.D = s->D;
        pa.ldq = rows;
        pa.block_size = s->block_size;
        pa.max_context_len = s->max_ctx;
        pa.max_q_len = s->max_q_len;
        pa.sliding_window = s->sliding_window;
        pa.scale = (float)(1.0 / sqrt((double)s->D));
        if (s->kv_u8) {
            pa.kv_u8 = 1;
            pa.k_meta = l->k_meta;
            pa.v_meta = l->v_meta;
        }
        const bool decode = ovb_decode_attention_takes(&pa), rotates = decode && ovb_decode_attention_rotates(&pa);
        if (s->kv_u8)
            OVB_STEP(ovb_rope_kv_write_u8(s->qkv, s->positions, s->slot_map, l->k_cache, l->v_cache, l->k_meta, l->v_meta, T, s->Hq, s->Hkv, s->D, s->theta,
                                          s->block_size, stream));
        else if (!rotates)
            OVB_STEP(ovb_rope_kv_write(s->qkv, s->positions, s->slot_map, l->k_cache, l->v_cache, T, s->Hq, s->Hkv, s->D, s->theta, s->block_size, stream));
        if (decode)
            OVB_STEP(ovb_decode_attention(&pa, rotates ? s->positions : nullptr, s->slot_map, s->theta, stream));
        else
            OVB_STEP(ovb_paged_attention(&pa, stream));
        OVB_STEP(run_gemm(s, &l->o, s->attn, s->h, s->h, T, H, stream));
        if (l->gate_up.act == OVB_ACT_SWIGLU) {
            OVB_STEP(run_norm_gemm(s, &l->gate_up, l->norm2, nullptr, T, s->x, s->act, T, s->ffn, stream));
        } else {
            OVB_STEP(run_norm_gemm(s, &l->gate_up, l->norm2, nullptr, T, s->x, s->gu, T, 2 * s->ffn, stream));
            OVB_STEP(ovb_silu_mul_counted(s->gu, s->act, T, s->ffn, nullptr, stream));
        }
        OVB_STEP(run_gemm(s, &l->down, s->act, s->h, s->h, T, H, stream));
    }
    // logits only for the last token of every sequence
    OVB_STEP(run_norm_gemm(s, &s->head, s->final_norm, s->logit_idx, T, s->last_x, s->logits, B, s->head_cols, stream));
#undef OVB_STEP
    return 0;
}

}  // extern "C"
