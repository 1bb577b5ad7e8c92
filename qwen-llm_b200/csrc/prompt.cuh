// Kernels of the many-row (prompt) pass that sit between its GEMMs (prompt_ops.cu): the same steps as the 16-row kernels
// of glue.cu / gdn.cu over up to a few hundred token rows, packing activations for gemm_tm.cuh.  Rows of a pass are padded to
// whole tiles of tile_tok tokens; the packed rows beyond the pass's tokens are zeros.
#pragma once
#include "model.cuh"

namespace dfl {

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
    const float* gate = nullptr;    // GLUE_COPY: x * sigmoid(gate), gate [rows][ld_x]
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
    float *conv_state = nullptr, *conv_new = nullptr;
    float *state_in = nullptr, *state_out = nullptr;   // state_in is left holding the state before the last block
    float *q_n = nullptr, *k_n = nullptr, *v = nullptr, *o = nullptr;
    // the last block's rows for a rollback, as the 16-row pass leaves them in the scratch
    float *keep_raw = nullptr, *keep_pre = nullptr, *keep_q = nullptr, *keep_k = nullptr, *keep_v = nullptr, *keep_ab = nullptr;
    uint8_t* acts = nullptr;
    int* err = nullptr;
};
dfl_status launch_tm_gdn_front(cudaStream_t st, const TmGdn& p);
dfl_status launch_tm_gdn_scan(cudaStream_t st, const TmGdn& p);
dfl_status launch_tm_gdn_pack(cudaStream_t st, const TmGdn& p);

}  // namespace dfl
