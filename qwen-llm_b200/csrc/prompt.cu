// Many-row pass of a prompt (reference: prefill_tokens_with_multi_hidden, crates/qwen-llm/src/metal_dflash.rs:10779): up to
// PROMPT_ROWS tokens through every layer at once, each weight tile unpacked once per 128 tokens instead of once per 16.
// The layer structure, the arithmetic class (integer weights, f16 hi + lo activations, f32 sums) and the session and scratch
// state it leaves behind are those of the packed pass (model.cu: verify_core).
#include <cstring>

#include "prompt.cuh"

namespace dfl {

struct PromptWs {
    uint32_t rows = 0;   // padded rows the buffers hold
    bool tiled = false;  // attn_part for sessions with a tiled cache too
    float *x = nullptr, *xn = nullptr, *part = nullptr, *sumsq = nullptr, *q_rot = nullptr, *gate = nullptr, *o = nullptr, *attn_part = nullptr;
    float *q_n = nullptr, *k_n = nullptr, *v = nullptr, *ab = nullptr, *conv_pre = nullptr, *capture = nullptr;
    uint8_t *acts_h = nullptr, *acts_f = nullptr, *acts_v = nullptr;
    int32_t* tokens = nullptr;
    // routed experts
    float *route_logits = nullptr, *route_w = nullptr, *route_sg = nullptr, *row_scale = nullptr, *gu = nullptr, *down = nullptr;
    int32_t *route_idx = nullptr, *n_seg = nullptr, *row_of = nullptr, *pos_of = nullptr;
    int2* seg = nullptr;
    uint8_t *acts_in = nullptr, *acts_mid = nullptr;
    int32_t* pinned = nullptr;
    uint8_t* base = nullptr;
};

const float* prompt_capture(const dfl_scratch* sc) { return sc->prompt->capture; }

// Only the slots that layers were named for: what the others hold in the workspace belongs to whoever had the block before.
cudaError_t copy_captured(float* dst, const float* src, uint32_t rows, uint32_t slots, uint32_t k_layers, uint64_t hidden, cudaMemcpyKind kind,
                          cudaStream_t st) {
    const size_t pitch = (size_t)k_layers * hidden * 4;
    if (slots == k_layers) return cudaMemcpyAsync(dst, src, rows * pitch, kind, st);
    return cudaMemcpy2DAsync(dst, pitch, src, pitch, (size_t)slots * hidden * 4, rows, kind, st);
}

void prompt_ws_free(PromptWs* w) {
    if (!w) return;
    pool_free(w->base);
    pool_free(w->pinned);
    delete w;
}

static bool group_supported(const MatGroup& g) {
    for (auto& m : g.mats)
        if (!gemm_tm_supported(m)) return false;
    return true;
}

bool prompt_supported(const dfl_model* m) {
    const dfl_arch& a = m->arch;
    if (m->act_layout != ACT_TS || m->ep_world > 1) return false;
    // DFL_PROMPT_ROWS=0 keeps prompts on the packed path
    static const bool enabled = [] { const char* e = getenv("DFL_PROMPT_ROWS"); return !(e && e[0] == '0'); }();
    if (!enabled) return false;
    const bool moe = a.expert_count > 0;
    if (moe && (a.expert_count > 1024 || a.expert_used_count > 16 || a.expert_shared_feed_forward_length != a.expert_feed_forward_length)) return false;
    for (auto& L : m->layers) {
        if (!(L.is_attn ? group_supported(L.qkv) && group_supported(L.wo) : group_supported(L.in_qkv_z) && group_supported(L.w_out))) return false;
        if (moe) {
            for (const MatGroup* g : {&L.moe_gate_up, &L.moe_down, &L.moe_down_sh})
                if (g->mats.size() != 1 || !group_supported(*g)) return false;
        } else if (!group_supported(L.gate_up) || !group_supported(L.down)) return false;
    }
    return true;
}

static int tm_splits(const MatGroup& g, int tok_tiles) {
    int tiles[8];
    int n = 0;
    for (auto& m : g.mats)
        if (n < 8) tiles[n++] = m.row_tiles;
    return gemm_tm_choose_splits(tiles, n, (int)(g.n_in / TILE_K), tok_tiles);
}

static dfl_status ensure_ws(const dfl_model* m, dfl_scratch* sc, uint32_t rows, bool tiled) {
    if (sc->prompt && sc->prompt->rows >= rows && (sc->prompt->tiled || !tiled)) return DFL_OK;
    if (sc->prompt) {   // what it held, it holds on to
        rows = std::max(rows, sc->prompt->rows);
        tiled |= sc->prompt->tiled;
    }
    if (sc->prompt) cudaDeviceSynchronize();
    prompt_ws_free(sc->prompt);
    sc->prompt = nullptr;
    auto* w = new PromptWs();
    const dfl_arch& a = m->arch;
    const GdnGeom gg = m->gdn_geom();
    const uint64_t H = a.hidden_size, F = a.intermediate_size, R = rows;
    const uint64_t q_dim = (uint64_t)a.n_q_heads * a.attn_head_dim, v_dim = (uint64_t)gg.n_v * 128, wide = std::max(q_dim, v_dim);
    uint64_t part = 0;
    for (int t = 1; t <= (int)(rows / TM_TOK); ++t)
        for (auto& L : m->layers)
            for (const MatGroup* g : {&L.qkv, &L.wo, &L.in_qkv_z, &L.w_out, &L.gate_up, &L.down})   // empty where a layer has none
                if (!g->mats.empty()) part = std::max<uint64_t>(part, (uint64_t)tm_splits(*g, t) * t * TM_TOK * g->total_cols);
    // one block for all of it: sizes first, then the pointers
    uint64_t total = 0;
    auto alloc = [&](auto** p, uint64_t bytes) {
        if (w->base) *p = reinterpret_cast<std::remove_reference_t<decltype(**p)>*>(w->base + total);
        total += (bytes + 255) / 256 * 256;
    };
    for (int pass = 0; pass < 2; ++pass) {
        total = 0;
        const uint64_t tiles = rows / TM_TOK;
        alloc(&w->x, R * H * 4);
        alloc(&w->xn, R * H * 4);
        alloc(&w->part, part * 4);
        alloc(&w->sumsq, H / TILE_K * R * 4);
        alloc(&w->q_rot, R * q_dim * 4);
        alloc(&w->gate, R * q_dim * 4);
        alloc(&w->o, R * wide * 4);
        if (m->n_attn) alloc(&w->attn_part, std::max(attn_rows_partials_floats(m->attn_geom(), (int)rows, KV_F16_ROWS),
                                                   tiled ? attn_rows_partials_floats(m->attn_geom(), (int)rows, KV_F16_TILED) : 0) * 4);
        alloc(&w->q_n, R * gg.n_k * 128 * 4);
        alloc(&w->k_n, R * gg.n_k * 128 * 4);
        alloc(&w->v, R * v_dim * 4);
        alloc(&w->ab, R * 2 * gg.n_v * 4);
        alloc(&w->conv_pre, 3ull * gg.conv_dim() * 4);
        alloc(&w->capture, R * sc->k_layers * H * 4);
        alloc(&w->acts_h, tiles * (H / TILE_K) * tm_chunk(TM_TOK));
        alloc(&w->acts_f, tiles * (F / TILE_K) * tm_chunk(TM_TOK));
        alloc(&w->acts_v, tiles * (wide / TILE_K) * tm_chunk(TM_TOK));
        alloc(&w->tokens, R * 4);
        if (a.expert_count > 0) {
            const uint64_t E = a.expert_count, used = a.expert_used_count, Fe = a.expert_feed_forward_length;
            const uint64_t segs = (uint64_t)tm_moe_max_segments((int)rows, (int)E, (int)used), P = segs * TM_SEG;
            alloc(&w->route_logits, R * (E + 1) * 4);
            alloc(&w->route_w, R * E * 4);
            alloc(&w->route_sg, R * 4);
            alloc(&w->route_idx, R * used * 4);
            alloc(&w->seg, segs * 8);
            alloc(&w->n_seg, 4);
            alloc(&w->row_of, P * 4);
            alloc(&w->pos_of, R * (used + 1) * 4);
            alloc(&w->row_scale, P * 4);
            alloc(&w->gu, P * 2 * Fe * 4);
            alloc(&w->down, P * H * 4);
            alloc(&w->acts_in, segs * (H / TILE_K) * tm_chunk(TM_SEG));
            alloc(&w->acts_mid, segs * (Fe / TILE_K) * tm_chunk(TM_SEG));
        }
        if (pass == 0 && !(w->base = (uint8_t*)pool_alloc(total))) break;
    }
    w->pinned = (int32_t*)pool_alloc_host(R * 4);
    if (!w->base || !w->pinned) {
        std::string why = cudaGetErrorString(cudaGetLastError());
        prompt_ws_free(w);
        return fail(DFL_ERR_OOM, "prompt pass: allocation failed: " + why);
    }
    w->rows = rows;
    w->tiled = tiled;
    sc->prompt = w;
    return DFL_OK;
}

static int token_tiles(uint32_t n) {
    const int tile_tok = gemm_tm_tile_tok((int)n);
    return ((int)n + tile_tok - 1) / tile_tok;
}
dfl_status prompt_reserve(const dfl_model* m, const dfl_session* s, dfl_scratch* sc, uint32_t n) {
    return ensure_ws(m, sc, (uint32_t)(token_tiles(n) * TM_TOK), s->kv_mode == KV_F16_TILED);
}

dfl_status prompt_core(const dfl_model* m, dfl_session* s, dfl_scratch* sc, const uint32_t* layer_ids, uint32_t n_ids, const int32_t* tokens,
                       uint32_t n, uint32_t start, uint32_t last_rows, bool want_head) {
    const dfl_arch& a = m->arch;
    const int tile_tok = gemm_tm_tile_tok((int)n), tok_tiles = token_tiles(n), rows_pad = tok_tiles * tile_tok;
    DFL_CHECK(prompt_reserve(m, s, sc, n));
    PromptWs* w = sc->prompt;
    cudaStream_t st = s->st;
    const uint64_t H = a.hidden_size, F = a.intermediate_size, KH = sc->k_layers * H;
    const AttnGeom ag = m->attn_geom();
    const GdnGeom gg = m->gdn_geom();
    const uint64_t q_dim = (uint64_t)ag.n_q * ag.hd;
    const int n_sumsq = (int)(H / TILE_K);

    memcpy(w->pinned, tokens, n * sizeof(int32_t));
    DFL_CUDA(cudaMemcpyAsync(w->tokens, w->pinned, n * sizeof(int32_t), cudaMemcpyHostToDevice, st));
    DFL_CHECK(launch_embed_rows(st, m->embd_dtype, m->embd_ggml, H, w->tokens, (int)n, w->x, (int)H));

    auto glue_base = [&] {
        TmGlue p;
        p.n_rows = (int)n; p.rows_pad = rows_pad; p.tile_tok = tile_tok; p.err = s->err;
        return p;
    };
    const bool moe = a.expert_count > 0;
    const int n_pos = (int)a.expert_used_count + 1;
    // splits < 0: the routed experts' outputs
    auto norm_glue = [&](int splits, const float* norm_w, bool want_xn, float* capture) -> dfl_status {
        TmGlue p = glue_base();
        if (splits > 0) { p.part = w->part; p.splits = splits; p.ld_part = (int)H; }
        if (splits < 0) { p.part = w->down; p.ld_part = (int)H; p.pos_of = w->pos_of; p.n_pos = n_pos; }
        p.x = w->x; p.ld_x = (int)H;
        p.mul_w = norm_w;
        p.acts = norm_w ? w->acts_h : nullptr;
        if (want_xn) { p.xn = w->xn; p.ld_xn = (int)H; }
        p.sumsq = norm_w ? w->sumsq : nullptr;
        p.capture = capture; p.ld_capture = (int)KH;
        return launch_tm_glue(st, p, H);
    };
    // one group of matrices over the same activations, side by side into w->part; returns the split count used
    auto gemm = [&](const MatGroup& g, const uint8_t* acts, bool norm, float out_scale, int* splits) -> dfl_status {
        *splits = tm_splits(g, tok_tiles);
        for (size_t i = 0; i < g.mats.size(); ++i)
            DFL_CHECK(launch_gemm_tm(st, g.mats[i], acts, w->part + g.col_off[i], *splits, (int)n, tile_tok, norm ? w->sumsq : nullptr,
                                     norm ? n_sumsq : 0, (float)H, 1e-6f, out_scale, g.total_cols, s->err));
        return DFL_OK;
    };
    DFL_CHECK(norm_glue(0, m->layers[0].attn_norm_w, !m->layers[0].is_attn, nullptr));

    int gi = 0, ai = 0, splits = 1;
    for (uint32_t il = 0; il < a.n_layer; ++il) {
        const LayerW& L = m->layers[il];
        const bool last = il + 1 == a.n_layer;
        if (L.is_attn) {
            DFL_CHECK(gemm(L.qkv, w->acts_h, true, 1.f, &splits));
            DFL_CHECK(launch_attn_front(st, ag, true, w->part, splits, (int)L.qkv.total_cols, L.q_norm_w, L.k_norm_w, start, (int)n, s->k_cache[ai],
                                        s->v_cache[ai], s->kv_mode, w->q_rot, w->gate, nullptr, -1, rows_pad));
            if (attn_rows_supported(ag, s->kv_mode))
                DFL_CHECK(launch_attn_rows(st, ag, w->q_rot, w->gate, s->k_cache[ai], s->v_cache[ai], s->kv_mode, start, (int)n, w->attn_part, w->o, s->err,
                                           s->kv_capacity));
            else for (uint32_t r = 0; r < n; r += MAX_ROWS)
                DFL_CHECK(launch_attn_verify(st, ag, w->q_rot + r * q_dim, w->gate + r * q_dim, s->k_cache[ai], s->v_cache[ai], s->kv_mode, start + r,
                                             (int)std::min<uint32_t>(MAX_ROWS, n - r), s->attn_partials, nullptr, m->act_layout, w->o + r * q_dim, s->err,
                                             s->kv_capacity));
            TmGlue p = glue_base();
            p.mode = GLUE_COPY;
            p.x = w->o; p.ld_x = (int)q_dim;
            p.acts = w->acts_v;
            DFL_CHECK(launch_tm_glue(st, p, q_dim));
            DFL_CHECK(gemm(L.wo, w->acts_v, false, 1.f, &splits));
            ++ai;
        } else {
            TmGdn p;
            p.g = gg;
            DFL_CHECK(gemm(L.in_qkv_z, w->acts_h, true, 1.f, &splits));
            DFL_CHECK(launch_tm_small_matmul(st, L.w_ab, w->xn, (int)H, (int)n, rows_pad, H, 2 * gg.n_v, w->sumsq, n_sumsq, (float)H, 1e-6f, w->ab,
                                             2 * gg.n_v));
            const int cur = s->ssm_cur[gi];
            p.part = w->part; p.splits = splits; p.ld_part = (int)L.in_qkv_z.total_cols; p.z_col = gg.conv_dim();
            p.n_rows = (int)n; p.rows_pad = rows_pad; p.tile_tok = tile_tok; p.last_rows = (int)last_rows;
            p.conv_w = L.conv_w; p.ab = w->ab; p.dt_bias = L.dt_bias; p.a_log = L.a_log; p.norm_w = L.ssm_norm_w;
            p.conv_in = s->conv[cur][gi]; p.conv_out = s->conv[cur ^ 1][gi];
            p.state_in = s->ssm[cur][gi]; p.state_out = s->ssm[cur ^ 1][gi];
            p.q_n = w->q_n; p.k_n = w->k_n; p.v = w->v; p.o = w->o;
            p.keep_raw = sc->qkv_raw[gi]; p.keep_pre = w->conv_pre; p.keep_q = sc->q_n[gi]; p.keep_k = sc->k_n[gi]; p.keep_v = sc->v[gi];
            p.keep_ab = sc->ab[gi];
            p.acts = w->acts_v; p.err = s->err;
            DFL_CHECK(launch_tm_gdn_front(st, p));
            DFL_CHECK(launch_tm_gdn_scan(st, p));
            DFL_CHECK(launch_tm_gdn_pack(st, p));
            s->ssm_cur[gi] = cur ^ 1;
            DFL_CHECK(gemm(L.w_out, w->acts_v, false, 1.f, &splits));
            ++gi;
        }
        DFL_CHECK(norm_glue(splits, L.post_norm_w, moe, nullptr));
        if (moe) {
            // route every row, gather the rows by expert, gate | up and down over the segments (forward.rs:749-824)
            const int E = (int)a.expert_count, used = (int)a.expert_used_count, Fe = (int)a.expert_feed_forward_length, T = Fe / TILE_R;
            DFL_CHECK(launch_tm_small_matmul(st, L.router_w, w->xn, (int)H, (int)n, rows_pad, H, E + 1, w->sumsq, n_sumsq, (float)H, 1e-6f, w->route_logits,
                                             E + 1));
            DFL_CHECK(launch_moe_route(st, w->route_logits, E + 1, E, used, (int)n, w->route_w, w->route_sg, w->route_idx, s->err));
            TmMoe q;
            q.n_rows = (int)n; q.rows_pad = rows_pad; q.n_expert = E; q.n_used = used; q.f = Fe;
            q.n_shared = ((int)n + TM_SEG - 1) / TM_SEG; q.max_seg = tm_moe_max_segments((int)n, E, used);
            q.route_idx = w->route_idx; q.route_w = w->route_w; q.route_sg = w->route_sg;
            q.seg = w->seg; q.n_seg = w->n_seg; q.row_of = w->row_of; q.pos_of = w->pos_of;
            q.xn = w->xn; q.ld_xn = (int)H; q.sumsq = w->sumsq; q.n_sumsq = n_sumsq; q.norm_k = (float)H;
            q.pre_scale = 1.0f / 64.0f;
            q.row_scale = w->row_scale; q.gu = w->gu; q.acts_in = w->acts_in; q.acts_mid = w->acts_mid; q.err = s->err;
            DFL_CHECK(launch_tm_moe_segments(st, q));
            DFL_CHECK(launch_tm_moe_pack(st, q, 0, H));
            TmSegments g;
            g.seg = w->seg; g.n_seg = w->n_seg; g.n_more = q.n_shared; g.max_seg = q.max_seg;
            g.n_tiles = 2 * T; g.half_tiles = T; g.half_off = (E + 1) * T; g.tiles_per_block = T;
            g.kblocks = (int)(H / TILE_K); g.row_scale = w->row_scale;
            DFL_CHECK(launch_gemm_tm_seg(st, L.moe_gate_up.mats[0], g, w->acts_in, w->gu, 1.f, (uint32_t)(2 * Fe), s->err));
            DFL_CHECK(launch_tm_moe_pack(st, q, 1, (uint64_t)Fe));
            TmSegments d;
            d.seg = w->seg; d.n_seg = w->n_seg; d.first = q.n_shared; d.max_seg = q.max_seg - q.n_shared;
            d.n_tiles = d.half_tiles = (int)(H / TILE_R);
            d.kblocks = d.kb_per_block = Fe / TILE_K;
            DFL_CHECK(launch_gemm_tm_seg(st, L.moe_down.mats[0], d, w->acts_mid, w->down, 64.f, (uint32_t)H, s->err));
            d.n_seg = nullptr; d.first = 0; d.max_seg = q.n_shared; d.kb_per_block = 0;
            DFL_CHECK(launch_gemm_tm_seg(st, L.moe_down_sh.mats[0], d, w->acts_mid, w->down, 64.f, (uint32_t)H, s->err));
            splits = -1;
        } else {
            DFL_CHECK(gemm(L.gate_up, w->acts_h, true, 1.f, &splits));
            {
                TmGlue p = glue_base();
                p.mode = GLUE_SWIGLU;
                p.part = w->part; p.splits = splits; p.ld_part = (int)L.gate_up.total_cols;
                p.swiglu_f = (int)F;
                p.pre_scale = 1.0f / 64.0f;   // as in the packed pass: keeps silu(g) * u inside the f16 operand range
                p.acts = w->acts_f;
                DFL_CHECK(launch_tm_glue(st, p, F));
            }
            DFL_CHECK(gemm(L.down, w->acts_f, false, 64.f, &splits));
        }
        float* cap = nullptr;
        for (uint32_t k = 0; k < n_ids; ++k)
            if (layer_ids[k] == il) { cap = w->capture + (uint64_t)k * H; break; }
        DFL_CHECK(norm_glue(splits, last ? nullptr : m->layers[il + 1].attn_norm_w, !last && !m->layers[il + 1].is_attn, cap));
        bool first = true;
        for (uint32_t k = 0; k < n_ids && cap; ++k) {   // a layer listed twice: its other slots get a copy
            if (layer_ids[k] != il) continue;
            if (first) { first = false; continue; }
            DFL_CUDA(cudaMemcpy2DAsync(w->capture + (uint64_t)k * H, KH * 4, cap, KH * 4, H * 4, n, cudaMemcpyDeviceToDevice, st));
        }
    }
    if (want_head) {   // the last row alone, through the packed path's head
        GlueParams p;
        p.mode = GLUE_COPY;
        p.x = w->x + (uint64_t)(n - 1) * H; p.ld_x = (int)H;
        p.mul_w = m->out_norm_w;
        p.acts = sc->acts_h; p.bf3 = m->act_layout;
        p.sumsq = sc->sumsq;
        p.n_rows = 1; p.err = s->err;
        DFL_CHECK(launch_glue(st, p, H));
        GemmEpilogue ep;
        ep.sumsq = sc->sumsq;
        ep.n_sumsq = (int)(H / GLUE_COLS);
        ep.norm_k = (float)H;
        ep.eps = 1e-6f;
        DFL_CHECK(head_core(m, s, sc, 1, ep));
    }
    if (moe)   // the last layer's choices for the last block's rows
        DFL_CUDA(cudaMemcpyAsync(sc->route_idx, w->route_idx + (uint64_t)(n - last_rows) * a.expert_used_count, (size_t)last_rows * a.expert_used_count * 4,
                                 cudaMemcpyDeviceToDevice, st));
    // the last block's captured rows where a packed pass would have left them
    if (n_ids)
        DFL_CUDA(copy_captured(sc->capture, w->capture + (uint64_t)(n - last_rows) * KH, last_rows, n_ids, sc->k_layers, H, cudaMemcpyDeviceToDevice, st));
    s->kv_n_pos = start + n;
    sc->last_n = last_rows;
    sc->last_n_verify = last_rows;
    sc->last_start = start + n - last_rows;
    sc->have_block = true;
    return DFL_OK;
}

}  // namespace dfl
