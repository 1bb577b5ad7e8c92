// Kernels of the many-row (prompt) pass that sit between its GEMMs (prompt_ops.cu): the same steps as the 16-row kernels
// of glue.cu / gdn.cu over up to a few hundred token rows, packing activations for gemm_tm.cuh.  Rows of a pass are padded to
// whole tiles of tile_tok tokens; the packed rows beyond the pass's tokens are zeros.
#pragma once
#include "model.cuh"

namespace dfl {

#ifdef __CUDACC__
// Eight consecutive columns k8 .. k8 + 7 (k8 % 8 == 0, inside one 256-column block) of token t of a tile of `tok` tokens -> the
// hi / lo planes of the activation chunk: one 16-byte store each, eight tokens fill 128 contiguous bytes.
__device__ __forceinline__ void tm_pack_oct(uint8_t* chunk, int tok, int t, int k8, const float (&v)[8], bool& overflow) {
    uint16_t hi[8], lo[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        overflow |= (fabsf(v[e]) >= 65504.f) && (fabsf(v[e]) < INFINITY);
        const __half h = __float2half_rn(v[e]);
        hi[e] = __half_as_ushort(h);
        lo[e] = __half_as_ushort(__float2half_rn(v[e] - __half2float(h)));
    }
    // k-positions of a quad: 0, 2, 1, 3 (ts_act_kpos)
    auto quad = [](const uint16_t* h) { return make_uint2((uint32_t)h[0] | ((uint32_t)h[2] << 16), (uint32_t)h[1] | ((uint32_t)h[3] << 16)); };
    uint8_t* dst = chunk + (k8 >> 6) * tm_bstage(tok) + ((k8 >> 3) & 7) * (tok * 16) + t * 16;
    const uint2 h0 = quad(hi), h1 = quad(hi + 4), l0 = quad(lo), l1 = quad(lo + 4);
    *reinterpret_cast<uint4*>(dst) = make_uint4(h0.x, h0.y, h1.x, h1.y);
    *reinterpret_cast<uint4*>(dst + tm_bstage(tok) / 2) = make_uint4(l0.x, l0.y, l1.x, l1.y);
}
// Sum of token t's activations over 32-column sub-block j -> hi / lo planes, both k-cores.
__device__ __forceinline__ void tm_pack_sum(uint8_t* chunk, int tok, int t, int j, float sum, bool& overflow) {
    overflow |= (fabsf(sum) >= 65504.f) && (fabsf(sum) < INFINITY);
    const __half h = __float2half_rn(sum), l = __float2half_rn(sum - __half2float(h));
    uint8_t* dst = chunk + 4 * tm_bstage(tok) + t * 16 + j * 2;
    *reinterpret_cast<__half*>(dst) = h;
    *reinterpret_cast<__half*>(dst + tok * 16) = h;
    *reinterpret_cast<__half*>(dst + tm_sums(tok) / 2) = l;
    *reinterpret_cast<__half*>(dst + tm_sums(tok) / 2 + tok * 16) = l;
}
#endif

struct TmGlue {
    int mode = GLUE_RESID;          // GLUE_RESID | GLUE_SWIGLU | GLUE_COPY as in ops.cuh
    const float* part = nullptr;    // [splits][rows_pad][ld_part]
    int splits = 0, ld_part = 0;
    float* x = nullptr;
    int ld_x = 0;
    const float* mul_w = nullptr;
    float pre_scale = 1.f;
    uint8_t* acts = nullptr;
    float* xn = nullptr;            // [rows][ld_xn] f32 copy of what is packed
    int ld_xn = 0;
    float* sumsq = nullptr;         // [k / 256][rows_pad]
    float* capture = nullptr;       // capture[row * ld_capture + col]
    int ld_capture = 0;
    int swiglu_f = 0;
    const int32_t* pos_of = nullptr;   // GLUE_RESID: rows pos_of[row][0 .. n_pos) of part (-1: none) instead of `splits` slices
    int n_pos = 0;
    int n_rows = 0, rows_pad = 0, tile_tok = TM_TOK;   // rows_pad = token tiles x tile_tok
    int* err = nullptr;
};
dfl_status launch_tm_glue(cudaStream_t st, const TmGlue& p, uint64_t k);

// out [rows][ld_out] = rs[row] * xn[row] . w[j] in f32 (alpha / beta, router); k a multiple of 256
dfl_status launch_tm_small_matmul(cudaStream_t st, const float* w, const float* xn, int ld_xn, int n_rows, int rows_pad, uint64_t k, int n_out,
                                  const float* sumsq, int n_sumsq, float norm_k, float eps, float* out, int ld_out);

struct TmGdn {
    GdnGeom g{};
    const float* part = nullptr;    // [splits][rows_pad][ld_part]: qkv columns first, z columns at z_col
    int splits = 0, ld_part = 0, z_col = 0;
    int n_rows = 0, rows_pad = 0, tile_tok = TM_TOK;   // rows_pad = token tiles x tile_tok
    int last_rows = 0;              // rows of the pass's last block (what a rollback after the pass can undo); 0: none kept
    const float *conv_w = nullptr, *ab = nullptr, *dt_bias = nullptr, *a_log = nullptr, *norm_w = nullptr;
    // conv rows and state: in -> out; the `in` buffers are left holding what precedes the last block (conv rows by way of keep_pre)
    float *conv_in = nullptr, *conv_out = nullptr, *state_in = nullptr, *state_out = nullptr;
    float *q_n = nullptr, *k_n = nullptr, *v = nullptr, *o = nullptr;
    // the last block's rows for a rollback, as the 16-row pass leaves them in the scratch
    float *keep_raw = nullptr, *keep_pre = nullptr, *keep_q = nullptr, *keep_k = nullptr, *keep_v = nullptr, *keep_ab = nullptr;
    uint8_t* acts = nullptr;
    int* err = nullptr;
};
dfl_status launch_tm_gdn_front(cudaStream_t st, const TmGdn& p);
dfl_status launch_tm_gdn_scan(cudaStream_t st, const TmGdn& p);
dfl_status launch_tm_gdn_pack(cudaStream_t st, const TmGdn& p);

// Routed experts of a pass (prompt_moe.cu).
struct TmMoe {
    int n_rows = 0, rows_pad = 0, n_expert = 0, n_used = 0, f = 0;   // f: inner width of an expert and of the shared expert
    int n_shared = 0, max_seg = 0;      // segments of the shared expert; bound on all segments
    const int32_t* route_idx = nullptr; // [rows][n_used]
    const float *route_w = nullptr, *route_sg = nullptr;   // [rows][n_expert], [rows]
    int2* seg = nullptr;                // [max_seg] {expert, rows}
    int32_t *n_seg = nullptr, *row_of = nullptr, *pos_of = nullptr;   // expert segments; row of a padded row; padded rows of a row [rows][n_used + 1]
    const float *xn = nullptr, *sumsq = nullptr;
    int ld_xn = 0, n_sumsq = 0;
    float norm_k = 1.f, pre_scale = 1.f;
    float* row_scale = nullptr;         // [padded rows]
    const float* gu = nullptr;          // [padded rows][2 f]
    uint8_t *acts_in = nullptr, *acts_mid = nullptr;
    int* err = nullptr;
};
int tm_moe_max_segments(int n_rows, int n_expert, int n_used);
dfl_status launch_tm_moe_segments(cudaStream_t st, const TmMoe& p);
dfl_status launch_tm_moe_pack(cudaStream_t st, const TmMoe& p, int mode, uint64_t k);   // mode 0: gathered inputs, 1: SwiGLU

}  // namespace dfl
