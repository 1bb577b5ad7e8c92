// Element-wise kernels between two GEMMs: split-K reduction, residual add, SwiGLU, folding of
// the RMSNorm weight, hidden-state capture and packing of the next GEMM's activations, in one
// pass.  Replaces the reference's separate kernel_add_inplace_f32 / kernel_silu_mul_f32 /
// kernel_rms_norm_batched_f32 launches (kernels/elementwise.metal:89,193; rms_norm.metal:48).
//
// RMSNorm is split so that no row-wide reduction sits on the critical path: this kernel
// multiplies by the norm weight and emits per-64-column partial sums of squares; the
// consuming GEMM multiplies its result by 1/sqrt(mean(x^2) + eps) per token.
#include "ops.cuh"

namespace dfl {

// grid = (k / 64, 2), block 128: thread = (token = 8 y + tid / 16, four consecutive columns).  One float4 per split per
// thread keeps every global load of the kernel independent (one latency round); the norm weight does not depend on the
// kernel before and is fetched ahead of the dependency wait.  128 threads: the following GEMM cannot start on an SM before the glue CTAs that
// belong there have left, and its late CTAs set the end of every link of the chain (verify block 3160 -> 3132 us when 256 threads became 128).
// What bounds the kernel is latency, and a good part of it was its own code: between two of its launches GEMMs stream 100 MB and more through
// L2, so that every line of it came from far away behind the dependency wait.  Two things follow.  The slices are fetched four at a time and not eight:
// the shorter code was worth 1.3 % of a token, 0.9 % of a verify block.  And with DRY the first warp runs through it once before the wait, on a buffer
// that nobody reads (p.dry); launch_glue says where.
template <bool DRY>
__global__ void __launch_bounds__(128, 7) glue_kernel(const GlueParams p) {
    const int quad = threadIdx.x & 15;
    const float4 w = p.mul_w ? *reinterpret_cast<const float4*>(p.mul_w + blockIdx.x * GLUE_COLS + quad * 4) : make_float4(1.f, 1.f, 1.f, 1.f);
    pdl_launch_dependents();
#pragma unroll 1
    for (int pass = DRY ? 0 : 1; pass < 2; ++pass) {
        GlueParams q = p;
        int cb = blockIdx.x, n_splits = 1;
        if (pass == 0) {
            if (threadIdx.x >= 32) continue;
            float* f = reinterpret_cast<float*>(p.dry + GLUE_DRY_ACTS);
            cb &= TILE_K / GLUE_COLS - 1;
            q.acts = p.acts ? p.dry : nullptr;
            q.part = p.part ? f : nullptr; q.ld_part = q.swiglu_f = 0;
            q.x = p.x ? f : nullptr; q.ld_x = 0;
            q.xn = p.xn ? f : nullptr; q.ld_xn = 0;
            q.sumsq = p.sumsq ? f : nullptr;
            q.capture = nullptr;
            q.route_w = nullptr;
        } else {
            pdl_wait();
            // columns of an expert that no row of the block chose, where the next GEMM reads chosen experts' columns only: nothing to do (at 16
            // rows of 8 experts some 100 of 256 are chosen; packing zeros for the others wrote 5 MB a layer)
            // (the first block stands in for a list of chosen experts that is empty: its zeros are read)
            if (p.skip_unchosen && blockIdx.x >= TILE_K / GLUE_COLS && (int)blockIdx.x * GLUE_COLS < p.route_n * p.route_f) {
                const int expert = p.route_e0 + (int)blockIdx.x * GLUE_COLS / p.route_f;
                if (!__syncthreads_or(threadIdx.x < MAX_ROWS && p.route_w[threadIdx.x * p.route_e + expert] != 0.f)) return;
            }
            n_splits = p.splits_dev ? p.splits + *p.splits_dev : p.splits;
        }
        glue_quad(q, n_splits, cb, blockIdx.y * 8 + (threadIdx.x >> 4), quad, w);
    }
}

// The residual glue behind the routed experts, whose device-chosen split count can be 40 and more: grid (k / 64, 8); the four warps fetch a quarter
// of the slices each (lane = token 2 y + lane / 16, four columns) and the first adds them in order, as one thread to all slices would.  (Slices
// that a row has no part in are zeros.  Where one slice ends and the next begins follows the list of all chosen experts, though, so the other rows of a
// block do move how a row's sum is grouped, and with it the last bits.)  With a thread to all slices the
// kernel was ten rounds of loads on a third of the chip (32 x 2 CTAs): a link of the chain 12.0 -> 8.9 us, with the join it no longer waits for.
constexpr int SLICES_STAGED = 64;
__global__ void __launch_bounds__(128) glue_slices_kernel(const GlueParams p) {
    __shared__ float4 red[SLICES_STAGED][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = lane & 15, tok = 2 * blockIdx.y + (lane >> 4), cb = blockIdx.x;
    const int col0 = cb * GLUE_COLS + quad * 4;
    const float4 w = p.mul_w ? *reinterpret_cast<const float4*>(p.mul_w + col0) : make_float4(1.f, 1.f, 1.f, 1.f);
    pdl_prologue();
    const int n_splits = p.splits + *p.splits_dev;
    const bool live = tok < p.n_rows;
    float4 xv = make_float4(0.f, 0.f, 0.f, 0.f), acc = xv;
    if (live && warp == 0 && p.x) xv = __ldcg(reinterpret_cast<const float4*>(p.x + (uint64_t)tok * p.ld_x + col0));
    const float* base = p.part + (uint64_t)tok * p.ld_part + col0;
    const uint64_t stride = (uint64_t)p.part_rows * p.ld_part;
    for (int s0 = 0; s0 < n_splits; s0 += SLICES_STAGED) {
        const int n = min(SLICES_STAGED, n_splits - s0);
        if (live) {
#pragma unroll 8
            for (int s = warp; s < n; s += 4) red[s][lane] = __ldcg(reinterpret_cast<const float4*>(base + (s0 + s) * stride));
        }
        __syncthreads();
        if (live && warp == 0) {
#pragma unroll 4
            for (int s = 0; s < n; ++s) {
                const float4 a = red[s][lane];
                acc.x += a.x; acc.y += a.y; acc.z += a.z; acc.w += a.w;
            }
        }
        __syncthreads();
    }
    if (warp > 0) return;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (live) {
        v[0] = xv.x + acc.x; v[1] = xv.y + acc.y; v[2] = xv.z + acc.z; v[3] = xv.w + acc.w;
        const float4 out = make_float4(v[0], v[1], v[2], v[3]);
        if (p.x) *reinterpret_cast<float4*>(p.x + (uint64_t)tok * p.ld_x + col0) = out;
        if (p.capture) *reinterpret_cast<float4*>(p.capture + (uint64_t)tok * p.ld_capture + col0) = out;
    }
    glue_finish(p, cb, tok, quad, w, v);
}

dfl_status launch_glue(cudaStream_t st, const GlueParams& p, uint64_t k) {
    if (k == 0 || k % TILE_K) return fail(DFL_ERR_BAD_SHAPE, "glue: column count must be a positive multiple of 256");
    if (p.splits_dev && p.mode == GLUE_RESID && p.part) {
        launch_k(glue_slices_kernel, dim3((unsigned)(k / GLUE_COLS), MAX_ROWS / 2), dim3(128), 0, st, p);
        count_launch();
        DFL_CUDA(cudaGetLastError());
        return DFL_OK;
    }
    // The run before the wait is time lost unless the CTA waits anyway.  Beside a tensor-memory GEMM CTA (17 warps of 96 registers: five on one
    // scheduler leave room for no sixth) none does: CTAs start where that GEMM has ended early, at most one an SM of a residual glue, and a SwiGLU glue's
    // further ones ran it behind the GEMM (verify block of 16 rows 2791 without any, 2773 with both, 2762 us with the residual one alone).  With few
    // rows the pass proper is too short to gain (two rows 2561 without, 2588 with; five to eight 2688, 2674).  The bf16 GEMM's six warps
    // leave room for three CTAs and more (draft 716 without, 710 with the residual one, 705 us with both).
    const uint64_t n_cta = 2 * k / GLUE_COLS, n_sm = (uint64_t)sm_count();
    const bool dry = p.dry && p.n_rows > 4 && (p.bf3 == ACT_TSB ? n_cta <= 3 * n_sm : p.mode != GLUE_SWIGLU && n_cta <= n_sm);
    launch_k(dry ? glue_kernel<true> : glue_kernel<false>, dim3((unsigned)(k / GLUE_COLS), MAX_ROWS / 8), dim3(128), 0, st, p);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

__global__ void __launch_bounds__(128) glue_groups_kernel(GlueParams p) {
    const int quad = threadIdx.x & 15, g = blockIdx.z;
    const float4 w = p.mul_w ? *reinterpret_cast<const float4*>(p.mul_w + blockIdx.x * GLUE_COLS + quad * 4) : make_float4(1.f, 1.f, 1.f, 1.f);
    pdl_prologue();
    p.n_rows -= g * MAX_ROWS;
    if (p.x) p.x += (uint64_t)g * MAX_ROWS * p.ld_x;
    if (p.part) p.part += (uint64_t)g * MAX_ROWS * p.ld_part;
    if (p.acts) p.acts += (uint64_t)g * (gridDim.x * GLUE_COLS / TILE_K) * act_chunk_dev(p.bf3);
    if (p.sumsq) p.sumsq += (uint64_t)g * gridDim.x * MAX_ROWS;
    glue_quad(p, p.splits, blockIdx.x, blockIdx.y * 8 + (threadIdx.x >> 4), quad, w);
}

dfl_status launch_glue_groups(cudaStream_t st, const GlueParams& p, uint64_t k) {
    if (k == 0 || k % TILE_K || p.n_rows < 1) return fail(DFL_ERR_BAD_SHAPE, "glue groups: shape");
    if (p.splits_dev || p.xn || p.capture || p.route_w) return fail(DFL_ERR_UNSUPPORTED, "glue groups: option");
    launch_k(glue_groups_kernel, dim3((unsigned)(k / GLUE_COLS), MAX_ROWS / 8, (unsigned)((p.n_rows + MAX_ROWS - 1) / MAX_ROWS)), dim3(128), 0, st, p);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

// ---- embedding rows ---------------------------------------------------------------
__device__ __forceinline__ void embed_one(int dtype, const uint8_t* __restrict__ ggml, uint64_t h, int32_t token, float* row) {
    const uint64_t col = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= h) return;
    const uint64_t row_bytes = h / 256 * (uint64_t)ggml_bytes_per_256(dtype);
    const uint8_t* seg = ggml + (uint64_t)token * row_bytes + (col >> 8) * (uint64_t)ggml_bytes_per_256(dtype);
    row[col] = ggml_decode_elem(dtype, seg, (int)(col & 255));
}
__global__ void embed_rows_kernel(int dtype, const uint8_t* __restrict__ ggml, uint64_t h, const int32_t* tokens,
                                  float* x, int ld) {
    pdl_prologue();
    embed_one(dtype, ggml, h, tokens[blockIdx.y], x + (uint64_t)blockIdx.y * ld);
}
// A block's tokens ride in the launch itself: the copy that used to carry 64 bytes to the device cost a pass 3 us.
struct BlockTokens { int32_t id[MAX_ROWS]; };
__global__ void embed_block_kernel(int dtype, const uint8_t* __restrict__ ggml, uint64_t h, const BlockTokens tokens, float* x, int ld) {
    pdl_prologue();
    embed_one(dtype, ggml, h, tokens.id[blockIdx.y], x + (uint64_t)blockIdx.y * ld);
}

dfl_status launch_embed_rows(cudaStream_t st, int dtype, const uint8_t* ggml, uint64_t h, const int32_t* tokens, int n_rows,
                             float* x, int ld) {
    if (h % 256 || ggml_bytes_per_256(dtype) == 0) return fail(DFL_ERR_UNSUPPORTED, "embed_rows: dtype or width");
    launch_k(embed_rows_kernel, dim3(dim3((unsigned)((h + 255) / 256), (unsigned)n_rows)), dim3(256), 0, st, dtype, ggml, h, tokens, x, ld);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

dfl_status launch_embed_block(cudaStream_t st, int dtype, const uint8_t* ggml, uint64_t h, const int32_t* tokens_host, int n_rows,
                              float* x, int ld) {
    if (h % 256 || ggml_bytes_per_256(dtype) == 0) return fail(DFL_ERR_UNSUPPORTED, "embed_block: dtype or width");
    if (n_rows < 1 || n_rows > MAX_ROWS) return fail(DFL_ERR_BAD_SHAPE, "embed_block: 1 to 16 rows");
    BlockTokens t{};
    for (int i = 0; i < n_rows; ++i) t.id[i] = tokens_host[i];
    // A plain launch: it starts a pass, and what follows in the pass may read before its own dependency wait what a pass or a rollback
    // before it wrote (gdn_mix_kernel: recurrent state and conv rows).  Early launches reach back any number of
    // kernels as long as all of them fit the chip, so the chain is cut here; nothing is lost, the host has waited for the
    // pass before in every caller but the outer loop's rollback.
    embed_block_kernel<<<dim3((unsigned)((h + 255) / 256), (unsigned)n_rows), 256, 0, st>>>(dtype, ggml, h, t, x, ld);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

// ---- small f32 matrices --------------------------------------------------------------
// A CTA of 512 threads per four output columns, a thread four columns of k at a time over all rows: the rows, which every CTA reads
// from L2, are read a quarter as often as with one output per CTA (257 outputs over 2048 columns and 16 rows: 33 -> 8.5 MB,
// 11.2 -> 7 us cold), and their loads are independent.  The first weights are on their way before the dependency wait.  Sums over
// lanes, then warps, in a fixed order.
constexpr int SMALL_OUT = 4;
__global__ void __launch_bounds__(512) small_matmul_kernel(const float* __restrict__ w, const float* xn, int ld_xn,
                                                           int n_rows, uint64_t k, int n_out, const float* sumsq, int n_sumsq,
                                                           float norm_k, float eps, float out_scale, float* out,
                                                           int ld_out) {
    const int o0 = blockIdx.x * SMALL_OUT, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float* wr[SMALL_OUT];   // outputs beyond the last read its row and are not stored
#pragma unroll
    for (int j = 0; j < SMALL_OUT; ++j) wr[j] = w + (uint64_t)min(o0 + j, n_out - 1) * k;
    float4 wv[SMALL_OUT];
    uint64_t c = (uint64_t)threadIdx.x * 4;
    if (c < k) {
#pragma unroll
        for (int j = 0; j < SMALL_OUT; ++j) wv[j] = *reinterpret_cast<const float4*>(wr[j] + c);
    }
    __shared__ float scale_s[MAX_ROWS];
    __shared__ float red[16][MAX_ROWS * SMALL_OUT];
    pdl_prologue();
    float acc[MAX_ROWS * SMALL_OUT];   // [row][output]
#pragma unroll
    for (int i = 0; i < MAX_ROWS * SMALL_OUT; ++i) acc[i] = 0.f;
    while (c < k) {
#pragma unroll
        for (int r = 0; r < MAX_ROWS; ++r) {
            if (r < n_rows) {
                const float4 xv = *reinterpret_cast<const float4*>(xn + (uint64_t)r * ld_xn + c);
#pragma unroll
                for (int j = 0; j < SMALL_OUT; ++j)
                    acc[SMALL_OUT * r + j] = fmaf(wv[j].w, xv.w, fmaf(wv[j].z, xv.z, fmaf(wv[j].y, xv.y, fmaf(wv[j].x, xv.x, acc[SMALL_OUT * r + j]))));
            }
        }
        c += 512 * 4;
        if (c < k) {
#pragma unroll
            for (int j = 0; j < SMALL_OUT; ++j) wv[j] = *reinterpret_cast<const float4*>(wr[j] + c);
        }
    }
    // per-token output scale (16 threads per token, fixed tree)
    if (threadIdx.x < 256) {
        const int tok = threadIdx.x >> 4, part = threadIdx.x & 15;
        float ss = 0.f;
        if (sumsq)
            for (int i = part; i < n_sumsq; i += 16) ss += sumsq[i * MAX_ROWS + tok];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (part == 0) scale_s[tok] = sumsq ? out_scale * (1.0f / sqrtf(ss / norm_k + eps)) : out_scale;
    }
#pragma unroll
    for (int n = 32; n >= 2; n >>= 1) {   // lane l ends with values 2 l, 2 l + 1
        const bool up = lane & (n >> 1);
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float give = up ? acc[i] : acc[i + n], keep = up ? acc[i + n] : acc[i];
            acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, n >> 1);
        }
    }
    *reinterpret_cast<float2*>(&red[warp][2 * lane]) = make_float2(acc[0], acc[1]);
    __syncthreads();
    if (threadIdx.x < MAX_ROWS * SMALL_OUT) {
        const int r = threadIdx.x / SMALL_OUT, j = threadIdx.x % SMALL_OUT;
        float s = 0.f;
#pragma unroll
        for (int wi = 0; wi < 16; ++wi) s += red[wi][threadIdx.x];
        if (r < n_rows && o0 + j < n_out) out[(uint64_t)r * ld_out + o0 + j] = s * scale_s[r];
    }
}

dfl_status launch_small_matmul(cudaStream_t st, const float* w, const float* xn, int ld_xn, int n_rows, uint64_t k, int n_out,
                               const GemmEpilogue& ep, float* out, int ld_out) {
    if (k % 4) return fail(DFL_ERR_BAD_SHAPE, "small_matmul: k must be a multiple of 4");
    launch_k(small_matmul_kernel, dim3((n_out + SMALL_OUT - 1) / SMALL_OUT), dim3(512), 0, st, w, xn, ld_xn, n_rows, k, n_out, ep.sumsq, ep.n_sumsq, ep.norm_k, ep.eps, ep.out_scale, out,
                                               ld_out);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

}  // namespace dfl
