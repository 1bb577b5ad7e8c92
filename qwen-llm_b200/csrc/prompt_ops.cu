// Element-wise, convolution and recurrence kernels of the many-row prompt pass (see prompt.cuh).
#include <cooperative_groups.h>

#include <mutex>

#include "prompt.cuh"

namespace dfl {

namespace cg = cooperative_groups;

// Threads of the packing kernels: CTA = 8 tokens x one 256-column block; lane = (token lane & 7, core lane >> 3), a warp covers
// the 32 columns of one sub-block, so reads are 128-byte runs of a token's row and stores 128-byte runs of a k-core.
// The modes are compiled apart: in one body they took 72 registers, three CTAs an SM (512 rows: 14.6 -> 14.0 us a residual
// step, 23.9 -> 19.6 a SwiGLU, cold).
template <bool SWIGLU>
__global__ void __launch_bounds__(256, SWIGLU ? 4 : 6) tm_glue_kernel(const TmGlue p) {
    pdl_prologue();
    __shared__ float ss_s[8][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tk = lane & 7, k8 = warp * 32 + (lane >> 3) * 8;
    const int row = blockIdx.y * 8 + tk, col = blockIdx.x * 256 + k8;
    const bool live = row < p.n_rows;
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = 0.f;
    auto add8 = [](float (&a)[8], const float* src) {
        const float4 x = __ldcg(reinterpret_cast<const float4*>(src)), y = __ldcg(reinterpret_cast<const float4*>(src) + 1);
        a[0] += x.x; a[1] += x.y; a[2] += x.z; a[3] += x.w;
        a[4] += y.x; a[5] += y.y; a[6] += y.z; a[7] += y.w;
    };
    auto store8 = [](float* dst, const float (&a)[8]) {
        reinterpret_cast<float4*>(dst)[0] = make_float4(a[0], a[1], a[2], a[3]);
        reinterpret_cast<float4*>(dst)[1] = make_float4(a[4], a[5], a[6], a[7]);
    };
    if (live) {
        const uint64_t stride = (uint64_t)p.rows_pad * p.ld_part;
        const float* base = p.part ? p.part + (uint64_t)row * p.ld_part + col : nullptr;
        if (SWIGLU) {
            float g[8] = {}, u[8] = {};
            for (int s = 0; s < p.splits; ++s) {
                add8(g, base + s * stride);
                add8(u, base + s * stride + p.swiglu_f);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = silu_f(g[e]) * u[e];
        } else {
            if (p.pos_of) {   // the routed experts' outputs of this row: shared expert first, then its choices in order
                for (int j = 0; j < p.n_pos; ++j) {
                    const int pos = p.pos_of[row * p.n_pos + j];
                    if (pos >= 0) add8(v, p.part + (uint64_t)pos * p.ld_part + col);
                }
            } else if (base)
                for (int s = 0; s < p.splits; ++s) add8(v, base + s * stride);
            if (p.x) {
                float xv[8] = {};
                add8(xv, p.x + (uint64_t)row * p.ld_x + col);
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = xv[e] + v[e];
                if (p.part) store8(p.x + (uint64_t)row * p.ld_x + col, v);
            }
        }
        if (!SWIGLU && p.capture) store8(p.capture + (uint64_t)row * p.ld_capture + col, v);
    }
    if (!SWIGLU && p.sumsq) {
        float ss = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) ss = fmaf(v[e], v[e], ss);
        ss += __shfl_xor_sync(0xffffffffu, ss, 8);
        ss += __shfl_xor_sync(0xffffffffu, ss, 16);
        if (lane < 8) ss_s[warp][lane] = ss;
        __syncthreads();
        if (threadIdx.x < 8) {
            float t = 0.f;
#pragma unroll
            for (int w = 0; w < 8; ++w) t += ss_s[w][threadIdx.x];
            p.sumsq[(uint64_t)blockIdx.x * p.rows_pad + blockIdx.y * 8 + threadIdx.x] = t;
        }
    }
    if (!SWIGLU && p.mul_w) {
        float w[8] = {};
        add8(w, p.mul_w + col);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] *= w[e];
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] *= p.pre_scale;
    if (!SWIGLU && p.xn && live) store8(p.xn + (uint64_t)row * p.ld_xn + col, v);
    if (p.acts) {
        uint8_t* chunk = p.acts + ((uint64_t)(row / p.tile_tok) * gridDim.x + blockIdx.x) * tm_chunk(p.tile_tok);
        bool over = false;
        tm_pack_oct(chunk, p.tile_tok, row % p.tile_tok, k8, v, over);
        float sum = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
        sum += __shfl_xor_sync(0xffffffffu, sum, 8);
        sum += __shfl_xor_sync(0xffffffffu, sum, 16);
        if (lane < 8) tm_pack_sum(chunk, p.tile_tok, row % p.tile_tok, warp, sum, over);
        if (over) atomicCAS(p.err, 0, DEV_ERR_OVERFLOW);
    }
}

dfl_status launch_tm_glue(cudaStream_t st, const TmGlue& p, uint64_t k) {
    if (k == 0 || k % TILE_K || p.rows_pad % p.tile_tok) return fail(DFL_ERR_BAD_SHAPE, "tm_glue: shape");
    launch_k(p.mode == GLUE_SWIGLU ? tm_glue_kernel<true> : tm_glue_kernel<false>, dim3((unsigned)(k / TILE_K), (unsigned)(p.rows_pad / 8)), dim3(256), 0, st, p);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

// ---- small f32 projections ----------------------------------------------------------------------
// Cluster of four CTAs = 32 rows x 32 outputs, a quarter of k each; 256 threads = sixteen 8 x 8 tiles (4 row groups x 4 output
// groups) of sixteen k-lanes.  64 columns of the 32 + 32 rows travel with cp.async, three stages deep (read straight through L1
// the rows, a multiple of 4 KiB apart, evict one another: 71 us at 77 rows x 64 outputs); an 8 x 8 tile then reads 16 bytes
// per 64 multiply-adds, which keeps the load unit and the multiply-add pipe about even.  Lanes, then the four quarters, are
// added in a fixed order.
constexpr int SMM_PITCH = 68, SMM_STAGE = 64 * SMM_PITCH, SMM_STAGES = 3;
__global__ void __cluster_dims__(1, 1, 4) __launch_bounds__(256)
tm_small_matmul_kernel(const float* __restrict__ w, const float* xn, int ld_xn, int n_rows, int rows_pad, int k, int n_out, const float* sumsq,
                       int n_sumsq, float norm_k, float eps, float* out, int ld_out) {
    extern __shared__ __align__(16) float smm[];   // [stage][32 x rows, 32 w rows][64 columns]
    __shared__ float part[32][33];
    cg::cluster_group cluster = cg::this_cluster();
    pdl_prologue();
    const int r0 = blockIdx.x * 32, o0 = blockIdx.y * 32, kq = k / 4, k0 = blockIdx.z * kq;
    const int rg = (threadIdx.x >> 6) * 8, og = ((threadIdx.x >> 4) & 3) * 8, kl = threadIdx.x & 15;
    float acc[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) acc[i] = 0.f;
    const int n_steps = kq / 64;
    auto fetch = [&](int step) {   // thread = (row of 64, a quarter of its 256 bytes)
        if (step < n_steps) {
            const int r = threadIdx.x >> 2, q = (threadIdx.x & 3) * 16;
            const float* src = (r < 32 ? xn + (uint64_t)min(r0 + r, n_rows - 1) * ld_xn : w + (uint64_t)min(o0 + r - 32, n_out - 1) * k) + k0 + step * 64 + q;
            float* dst = smm + (step % SMM_STAGES) * SMM_STAGE + r * SMM_PITCH + q;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst + 4 * i)), "l"(src + 4 * i) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0);
    fetch(1);
    for (int st = 0; st < n_steps; ++st) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();   // step st has landed for everyone; stage (st + 2) % 3 was consumed in step st - 1
        fetch(st + 2);
        const float* xs = smm + (st % SMM_STAGES) * SMM_STAGE + rg * SMM_PITCH + kl * 4;
        const float* ws = smm + (st % SMM_STAGES) * SMM_STAGE + (32 + og) * SMM_PITCH + kl * 4;
        float4 xv[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) xv[i] = *reinterpret_cast<const float4*>(xs + i * SMM_PITCH);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float4 wv = *reinterpret_cast<const float4*>(ws + j * SMM_PITCH);
#pragma unroll
            for (int i = 0; i < 8; ++i)
                acc[8 * i + j] = fmaf(wv.w, xv[i].w, fmaf(wv.z, xv[i].z, fmaf(wv.y, xv[i].y, fmaf(wv.x, xv[i].x, acc[8 * i + j]))));
        }
    }
    // lane kl keeps entries 4 kl .. 4 kl + 3 of the tile
#pragma unroll
    for (int n = 32; n >= 4; n >>= 1) {
        const bool up = kl & (n / 4);
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float give = up ? acc[i] : acc[i + n], keep = up ? acc[i + n] : acc[i];
            acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, n / 4);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) part[rg + ((4 * kl + i) >> 3)][og + ((4 * kl + i) & 7)] = acc[i];
    cluster.sync();
    {
        const int r = 8 * (int)cluster.block_rank() + (threadIdx.x >> 5), o = threadIdx.x & 31, row = r0 + r;
        float v = 0.f;
#pragma unroll
        for (unsigned q = 0; q < 4; ++q) v += *cluster.map_shared_rank(&part[r][o], q);
        if (row < n_rows && o0 + o < n_out) {
            float ss = 0.f;
            for (int q = 0; q < n_sumsq; ++q) ss += sumsq[(uint64_t)q * rows_pad + row];
            out[(uint64_t)row * ld_out + o0 + o] = v * (1.0f / sqrtf(ss / norm_k + eps));
        }
    }
    cluster.sync();   // nobody leaves while its part is being read
}

dfl_status launch_tm_small_matmul(cudaStream_t st, const float* w, const float* xn, int ld_xn, int n_rows, int rows_pad, uint64_t k, int n_out,
                                  const float* sumsq, int n_sumsq, float norm_k, float eps, float* out, int ld_out) {
    if (k % 256) return fail(DFL_ERR_BAD_SHAPE, "tm_small_matmul: k must be a multiple of 256");
    constexpr size_t SMEM = (size_t)SMM_STAGES * SMM_STAGE * sizeof(float);
    static std::once_flag once[16];
    int dev = 0;
    DFL_CUDA(cudaGetDevice(&dev));
    cudaError_t attr = cudaSuccess;
    std::call_once(once[dev & 15], [&] { attr = cudaFuncSetAttribute(tm_small_matmul_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM); });
    DFL_CUDA(attr);
    launch_k(tm_small_matmul_kernel, dim3((unsigned)((n_rows + 31) / 32), (unsigned)((n_out + 31) / 32), 4), dim3(256), SMEM, st, w, xn, ld_xn, n_rows,
             rows_pad, (int)k, n_out, sumsq, n_sumsq, norm_k, eps, out, ld_out);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

// ---- gated delta net: conv + SiLU + L2 norms over all rows of the pass ---------------------------
// grid (heads of 128 channels, rows / 16), four warps of four rows each, lane = four channels; the three rows before a warp's own come
// from the pass's projection output again (or from the session's conv rows for the first ones).
__global__ void __launch_bounds__(128) tm_gdn_front_kernel(const TmGdn p) {
    pdl_prologue();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, head = blockIdx.x;
    const int conv_dim = p.g.conv_dim(), i0 = blockIdx.y * 16 + 4 * w, c = head * 128 + 4 * lane;
    if (i0 >= p.n_rows) return;
    float4 xv[7];
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        const int row = i0 - 3 + k;
        xv[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < 0) xv[k] = *reinterpret_cast<const float4*>(p.conv_in + (row + 3) * conv_dim + c);
        else if (row < p.n_rows) {
            for (int s = 0; s < p.splits; ++s) {
                const float4 a = __ldcg(reinterpret_cast<const float4*>(p.part + ((uint64_t)s * p.rows_pad + row) * p.ld_part + c));
                xv[k].x += a.x; xv[k].y += a.y; xv[k].z += a.z; xv[k].w += a.w;
            }
        }
    }
    float4 tap[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) tap[e] = *reinterpret_cast<const float4*>(p.conv_w + (uint64_t)(c + e) * 4);
    float y[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float in[4][4] = {{xv[j].x, xv[j + 1].x, xv[j + 2].x, xv[j + 3].x}, {xv[j].y, xv[j + 1].y, xv[j + 2].y, xv[j + 3].y},
                                {xv[j].z, xv[j + 1].z, xv[j + 2].z, xv[j + 3].z}, {xv[j].w, xv[j + 1].w, xv[j + 2].w, xv[j + 3].w}};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float s = 0.f;
            s += tap[e].x * in[e][0];
            s += tap[e].y * in[e][1];
            s += tap[e].z * in[e][2];
            s += tap[e].w * in[e][3];
            y[j][e] = silu_f(s);
        }
    }
    const bool is_v = head >= 2 * p.g.n_k, is_q = head < p.g.n_k;
    if (!is_v) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float sq = warp_sum((y[j][0] * y[j][0] + y[j][1] * y[j][1]) + (y[j][2] * y[j][2] + y[j][3] * y[j][3]));
            const float inv = 1.0f / fmaxf(sqrtf(sq), 1e-6f);
#pragma unroll
            for (int e = 0; e < 4; ++e) y[j][e] *= inv;
        }
    }
    const int h = is_v ? head - 2 * p.g.n_k : is_q ? head : head - p.g.n_k;
    const int ld = (is_v ? p.g.n_v : p.g.n_k) * 128;
    float* dst = (is_v ? p.v : is_q ? p.q_n : p.k_n) + h * 128 + 4 * lane;
    float* keep = (is_v ? p.keep_v : is_q ? p.keep_q : p.keep_k) + h * 128 + 4 * lane;
    const int keep0 = p.n_rows - p.last_rows;   // first row of the last block
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int row = i0 + j;
        if (row >= p.n_rows) break;
        const float4 o = make_float4(y[j][0], y[j][1], y[j][2], y[j][3]);
        *reinterpret_cast<float4*>(dst + (uint64_t)row * ld) = o;
        if (p.last_rows && row >= keep0) {
            *reinterpret_cast<float4*>(keep + (uint64_t)(row - keep0) * ld) = o;
            *reinterpret_cast<float4*>(p.keep_raw + (uint64_t)(row - keep0) * conv_dim + c) = xv[j + 3];
        }
    }
    // row r of the sequence {state rows -3 .. -1, rows 0 ..} is xv[r - i0 + 3]; every row has one owner (rows below 0: the first warp)
    auto mine = [&](int r) { return (r >= i0 && r < i0 + 4) || (r < 0 && i0 == 0); };
#pragma unroll
    for (int k = 0; k < 7; ++k) {
        const int r = i0 - 3 + k;
        if (!mine(r)) continue;
        const int tn = r - (p.n_rows - 3), tp = r - (keep0 - 3);   // index in the new state / in the state before the last block
        if (tn >= 0 && tn < 3) *reinterpret_cast<float4*>(p.conv_out + tn * conv_dim + c) = xv[k];
        if (p.last_rows && tp >= 0 && tp < 3) *reinterpret_cast<float4*>(p.keep_pre + tp * conv_dim + c) = xv[k];
    }
}

dfl_status launch_tm_gdn_front(cudaStream_t st, const TmGdn& p) {
    launch_k(tm_gdn_front_kernel, dim3((unsigned)(p.g.conv_dim() / 128), (unsigned)((p.n_rows + 15) / 16)), dim3(128), 0, st, p);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

// ---- gated delta net: the recurrence -------------------------------------------------------------
// Sixteen tokens at a time.  With S0 the state before a block, u_i = S0 k_i, w_i = S0 q_i and D_ij = g_{j+1} .. g_i the decay
// between two tokens of the block (G_i from its start), the token recurrence
//     c_i = beta_i (v_i - g_i S_{i-1} k_i),  S_i = g_i S_{i-1} + c_i k_i^T,  o_i = S_i q_i
// is, row by row of S (a row = one value channel),
//     (I + L) c = b,  L_ij = beta_i D_ij (k_j . k_i) for j < i,  b_i = beta_i (v_i - G_i u_i),
//     o_i = G_i w_i + sum_{j <= i} D_ij (k_j . q_i) c_j,   S = G_15 S0 + sum_j D_15,j c_j k_j^T,
// all in f32 and without a division.  A token-by-token scan waits twice per token for a three-level shuffle sum (512 tokens:
// 242 us a layer); here a block's 32 sums are in flight together and only the 16-step substitution is serial, in registers.
// grid (n_v, 4 quarters of the value channels), 256 threads; state, k and q rows lie in shared memory, rows 132 floats apart so that eight
// neighbouring ones start in different 16-byte bank groups.  Per block, a barrier behind each:
//   A  dots: warp = 32 key channels x the k or the q rows, lane = four state rows x four tokens, sums in registers;
//   B  the four channel ranges added, L and M from the Gram matrices and decays; the rows after next are requested;
//   C  warp 0: substitution, lane = state row, 16 steps of one multiply-add; warps 4 - 7: the Gram matrices of the next block (they do not
//      depend on the state); warp 1: its gates and decays;
//   D  outputs (lane = state row) and the state.
// No sum crosses lanes.  Before, a warp owned four rows and summed 64 + 64 values over its lanes per block (124 exchanges a warp) with the
// Gram matrices in front: 148 us a layer for 512 tokens, now 135; what is left is
// shared-memory bandwidth (4500 wavefronts a block of 16 tokens) and the substitution.
constexpr int SCAN_BLK = 16, SCAN_GS = 132, SCAN_RS = 36, SCAN_BUFS = 3;
struct ScanSmem {
    float s[32][SCAN_GS];                  // state rows of the CTA
    float kq[SCAN_BUFS][32][SCAN_GS];      // a block's k rows, then its q rows
    float vs[SCAN_BUFS][SCAN_BLK][32];
    float red[4][32 * SCAN_RS];            // [channel range][state row][k, q row]
    float gram[4][SCAN_BLK * SCAN_RS];     // [channel range][k row][k, q row]
    float a[32][33];                       // S0 k_i, S0 q_i: [vector][state row]
    float L[SCAN_BLK][SCAN_BLK], M[SCAN_BLK][SCAN_BLK];   // [j][i]
    float C[SCAN_BLK][32];                 // c_j of every state row
    float gs[2][SCAN_BLK], bs[2][SCAN_BLK], G[2][SCAN_BLK], D[2][SCAN_BLK];
};
__global__ void __launch_bounds__(256, 1) tm_gdn_scan_kernel(const TmGdn p) {
    extern __shared__ __align__(16) uint8_t scan_smem[];
    ScanSmem& sm = *reinterpret_cast<ScanSmem*>(scan_smem);
    const GdnGeom& g = p.g;
    const int h = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, hk = h % g.n_k, dv_cta = blockIdx.y * 32;
    const int rg = lane >> 2, vg = lane & 3, c0 = (warp & 3) * 32;
    const float dtb = p.dt_bias[h], alog = p.a_log[h];
    pdl_prologue();
    const uint64_t s_off = ((uint64_t)h * 128 + dv_cta) * 128;
    for (int i = threadIdx.x; i < 32 * 32; i += 256)
        *reinterpret_cast<float4*>(&sm.s[i >> 5][4 * (i & 31)]) = __ldcg(reinterpret_cast<const float4*>(p.state_in + s_off) + i);
    auto cp16 = [](void* dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory"); };
    // block boundaries: multiples of 16 from the start, and the first row of the part a rollback may undo
    const int ckpt = p.last_rows ? p.n_rows - p.last_rows : 0;
    auto next_of = [&](int r0) { return min(r0 < ckpt && r0 + SCAN_BLK > ckpt ? ckpt : r0 + SCAN_BLK, p.n_rows); };
    auto fetch = [&](int r0, int buf) {   // rows beyond the block's are zeros: they add nothing and decay nothing
        const int n = r0 < p.n_rows ? next_of(r0) - r0 : 0;
        for (int i = threadIdx.x; i < 32 * 32; i += 256) {
            const int v = i >> 5, r = v & 15, d = (i & 31) * 4;
            if (r < n) cp16(&sm.kq[buf][v][d], (v < 16 ? p.k_n : p.q_n) + ((uint64_t)(r0 + r) * g.n_k + hk) * 128 + d);
            else *reinterpret_cast<float4*>(&sm.kq[buf][v][d]) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (threadIdx.x < SCAN_BLK * 8) {
            const int r = threadIdx.x >> 3, d = (threadIdx.x & 7) * 4;
            if (r < n) cp16(&sm.vs[buf][r][d], p.v + ((uint64_t)(r0 + r) * g.n_v + h) * 128 + dv_cta + d);
            else *reinterpret_cast<float4*>(&sm.vs[buf][r][d]) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // a block's gate inputs are loaded a block ahead by sixteen lanes of warp 1, which turn them into gates and decays
    float ga = 0.f, gb = 0.f;
    auto gate_load = [&](int r0) {
        if (warp == 1 && lane < SCAN_BLK && r0 + lane < p.n_rows) {
            const float* a = p.ab + (uint64_t)(r0 + lane) * (2 * g.n_v) + h;
            ga = __ldcg(a);
            gb = __ldcg(a + g.n_v);
        }
    };
    auto gate_store = [&](int r0, int par) {
        if (warp != 1) return;
        const int n = next_of(r0) - r0;
        if (lane < SCAN_BLK) {
            sm.gs[par][lane] = lane < n ? expf(softplus_f(ga + dtb) * alog) : 1.f;
            sm.bs[par][lane] = lane < n ? sigmoid_f(gb) : 0.f;
            const int kr = r0 + lane - ckpt;
            if (p.last_rows && kr >= 0 && lane < n && blockIdx.y == 0) {
                p.keep_ab[(uint64_t)kr * (2 * g.n_v) + h] = ga;
                p.keep_ab[(uint64_t)kr * (2 * g.n_v) + g.n_v + h] = gb;
            }
        }
        __syncwarp();
        const int i = lane & 15;   // G_i and D_15,i
        float v = 1.f;
#pragma unroll
        for (int t = 0; t < SCAN_BLK; ++t)
            if (lane < 16 ? t <= i : t > i) v *= sm.gs[par][t];
        (lane < 16 ? sm.G : sm.D)[par][i] = v;
    };
    // k_j . k_i and k_j . q_i of a block: warp 4 + x = channels 32 x .., lane = two rows j x eight vectors
    auto gram = [&](int buf) {
        if (warp < 4) return;
        float acc[2][8];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int n = 0; n < 8; ++n) acc[i][n] = 0.f;
#pragma unroll 2
        for (int kk = 0; kk < 32; kk += 4) {
            float4 r[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) r[i] = *reinterpret_cast<const float4*>(&sm.kq[buf][rg + 8 * i][c0 + kk]);
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                const float4 x = *reinterpret_cast<const float4*>(&sm.kq[buf][vg + 4 * n][c0 + kk]);
#pragma unroll
                for (int i = 0; i < 2; ++i) acc[i][n] = fmaf(r[i].w, x.w, fmaf(r[i].z, x.z, fmaf(r[i].y, x.y, fmaf(r[i].x, x.x, acc[i][n]))));
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int n = 0; n < 8; ++n) sm.gram[warp & 3][(rg + 8 * i) * SCAN_RS + vg + 4 * n] = acc[i][n];
    };
    // the conv rows before the last block replace the pass's first ones, which the front kernel has read; one slice per CTA
    if (p.last_rows) {
        const int n = 3 * g.conv_dim() / 4, per = (n + gridDim.x * gridDim.y - 1) / (gridDim.x * gridDim.y);
        const int first = (blockIdx.y * gridDim.x + blockIdx.x) * per;
        for (int i = first + threadIdx.x; i < min(n, first + per); i += 256)
            reinterpret_cast<float4*>(p.conv_in)[i] = __ldcg(reinterpret_cast<const float4*>(p.keep_pre) + i);
    }
    fetch(0, 0);
    gate_load(0);
    fetch(next_of(0), 1);
    gate_store(0, 0);
    gate_load(next_of(0));
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    gram(0);
    int buf = 0, par = 0;
    for (int r0 = 0; r0 < p.n_rows;) {
        const int r1 = next_of(r0), n = r1 - r0, nbuf = buf == SCAN_BUFS - 1 ? 0 : buf + 1, fbuf = nbuf == SCAN_BUFS - 1 ? 0 : nbuf + 1;
        // ---- A: u = S0 k, w = S0 q
        {
            const int v0 = (warp >> 2) * 16;
            float acc[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int m = 0; m < 4; ++m) acc[i][m] = 0.f;
#pragma unroll 4
            for (int kk = 0; kk < 32; kk += 4) {
                float4 r[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) r[i] = *reinterpret_cast<const float4*>(&sm.s[rg + 8 * i][c0 + kk]);
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const float4 x = *reinterpret_cast<const float4*>(&sm.kq[buf][v0 + vg + 4 * m][c0 + kk]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[i][m] = fmaf(r[i].w, x.w, fmaf(r[i].z, x.z, fmaf(r[i].y, x.y, fmaf(r[i].x, x.x, acc[i][m]))));
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int m = 0; m < 4; ++m) sm.red[warp & 3][(rg + 8 * i) * SCAN_RS + v0 + vg + 4 * m] = acc[i][m];
        }
        __syncthreads();   // also: gram and gates of this block
        // ---- B: lane = vector
        if (r1 < p.n_rows) fetch(next_of(r1), fbuf);   // its last reader was phase D of the block before
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const int at = (warp + 8 * m) * SCAN_RS + lane;
            sm.a[lane][warp + 8 * m] = (sm.red[0][at] + sm.red[1][at]) + (sm.red[2][at] + sm.red[3][at]);
        }
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const int j = warp + 8 * m, i = lane & 15, at = j * SCAN_RS + lane;
            float d = 1.f;   // D_ij
#pragma unroll
            for (int t = 1; t < SCAN_BLK; ++t)
                if (t > j && t <= i) d *= sm.gs[par][t];
            const float dot = (sm.gram[0][at] + sm.gram[1][at]) + (sm.gram[2][at] + sm.gram[3][at]);
            if (lane < 16) sm.L[j][i] = i > j ? sm.bs[par][i] * d * dot : 0.f;
            else sm.M[j][i] = i >= j ? d * dot : 0.f;
        }
        if (r1 < p.n_rows) asm volatile("cp.async.wait_group 1;" ::: "memory");   // the next block's rows
        __syncthreads();
        // ---- C
        if (warp == 0) {   // lane = state row
            float u[SCAN_BLK];
#pragma unroll
            for (int i = 0; i < SCAN_BLK; ++i) u[i] = sm.bs[par][i] * (sm.vs[buf][i][lane] - sm.G[par][i] * sm.a[i][lane]);
#pragma unroll
            for (int j = 0; j < SCAN_BLK; ++j) {
                sm.C[j][lane] = u[j];
#pragma unroll
                for (int i4 = (j + 1) / 4; i4 < 4; ++i4) {
                    const float4 l = *reinterpret_cast<const float4*>(&sm.L[j][4 * i4]);
                    if (4 * i4 > j) u[4 * i4] = fmaf(-l.x, u[j], u[4 * i4]);
                    if (4 * i4 + 1 > j) u[4 * i4 + 1] = fmaf(-l.y, u[j], u[4 * i4 + 1]);
                    if (4 * i4 + 2 > j) u[4 * i4 + 2] = fmaf(-l.z, u[j], u[4 * i4 + 2]);
                    if (4 * i4 + 3 > j) u[4 * i4 + 3] = fmaf(-l.w, u[j], u[4 * i4 + 3]);
                }
            }
        } else if (r1 < p.n_rows) {
            if (warp == 1) {
                gate_store(r1, par ^ 1);
                gate_load(next_of(r1));
            }
            gram(nbuf);
        }
        __syncthreads();
        // ---- D: outputs of tokens warp, warp + 8 (lane = state row); state rows 4 warp .. + 3 (lane = four channels)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int i = warp + 8 * half;
            float o0 = sm.G[par][i] * sm.a[16 + i][lane], o1 = 0.f;
#pragma unroll
            for (int j = 0; j < SCAN_BLK; j += 2) {   // M is zero for j > i
                o0 = fmaf(sm.M[j][i], sm.C[j][lane], o0);
                o1 = fmaf(sm.M[j + 1][i], sm.C[j + 1][lane], o1);
            }
            if (i < n) p.o[((uint64_t)(r0 + i) * g.n_v + h) * 128 + dv_cta + lane] = o0 + o1;
        }
        {
            const float Gend = sm.G[par][SCAN_BLK - 1];
            float4 s4[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                s4[r] = *reinterpret_cast<const float4*>(&sm.s[4 * warp + r][4 * lane]);
                s4[r].x *= Gend; s4[r].y *= Gend; s4[r].z *= Gend; s4[r].w *= Gend;
            }
#pragma unroll
            for (int j = 0; j < SCAN_BLK; ++j) {
                const float4 k = *reinterpret_cast<const float4*>(&sm.kq[buf][j][4 * lane]), c4 = *reinterpret_cast<const float4*>(&sm.C[j][4 * warp]);
                const float d = sm.D[par][j], c[4] = {d * c4.x, d * c4.y, d * c4.z, d * c4.w};
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    s4[r].x = fmaf(c[r], k.x, s4[r].x); s4[r].y = fmaf(c[r], k.y, s4[r].y);
                    s4[r].z = fmaf(c[r], k.z, s4[r].z); s4[r].w = fmaf(c[r], k.w, s4[r].w);
                }
            }
            float* out = r1 == p.n_rows ? p.state_out : p.last_rows && r1 == ckpt ? p.state_in : nullptr;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                *reinterpret_cast<float4*>(&sm.s[4 * warp + r][4 * lane]) = s4[r];
                if (out) *reinterpret_cast<float4*>(out + s_off + (4 * warp + r) * 128 + 4 * lane) = s4[r];
            }
        }
        __syncthreads();
        r0 = r1; buf = nbuf; par ^= 1;
    }
}

dfl_status launch_tm_gdn_scan(cudaStream_t st, const TmGdn& p) {
    static std::once_flag once[16];
    int dev = 0;
    cudaGetDevice(&dev);
    cudaError_t e = cudaSuccess;
    auto allow = [&] { e = cudaFuncSetAttribute(tm_gdn_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ScanSmem)); };
    if (dev >= 0 && dev < 16) std::call_once(once[dev], allow);
    else allow();
    DFL_CUDA(e);
    launch_k(tm_gdn_scan_kernel, dim3((unsigned)p.g.n_v, 4), dim3(256), sizeof(ScanSmem), st, p);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

// ---- gated delta net: y = rmsnorm(o; eps * 128) * w * silu(z), packed ------------------------------
// CTA = 8 tokens x two heads (256 channels), threads as in tm_glue_kernel
__global__ void __launch_bounds__(256) tm_gdn_pack_kernel(const TmGdn p) {
    pdl_prologue();
    __shared__ float ss_s[8][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tk = lane & 7, k8 = warp * 32 + (lane >> 3) * 8;
    const int row = blockIdx.y * 8 + tk, col = blockIdx.x * 256 + k8;
    const bool live = row < p.n_rows;
    float v[8] = {}, z[8] = {};
    auto add8 = [](float (&a)[8], const float* src) {
        const float4 x = __ldcg(reinterpret_cast<const float4*>(src)), y = __ldcg(reinterpret_cast<const float4*>(src) + 1);
        a[0] += x.x; a[1] += x.y; a[2] += x.z; a[3] += x.w;
        a[4] += y.x; a[5] += y.y; a[6] += y.z; a[7] += y.w;
    };
    if (live) {
        add8(v, p.o + (uint64_t)row * p.g.n_v * 128 + col);
        for (int s = 0; s < p.splits; ++s) add8(z, p.part + ((uint64_t)s * p.rows_pad + row) * p.ld_part + p.z_col + col);
    }
    float ss = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) ss = fmaf(v[e], v[e], ss);
    ss += __shfl_xor_sync(0xffffffffu, ss, 8);
    ss += __shfl_xor_sync(0xffffffffu, ss, 16);
    if (lane < 8) ss_s[warp][lane] = ss;
    __syncthreads();
    const int w0 = warp & 4;   // the four warps of this head
    const float tot = ((ss_s[w0][tk] + ss_s[w0 + 1][tk]) + ss_s[w0 + 2][tk]) + ss_s[w0 + 3][tk];
    const float sc = 1.0f / sqrtf(tot / 128.f + 1e-6f * 128.f);
    float nw[8] = {};
    add8(nw, p.norm_w + (k8 & 127));
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = live ? v[e] * sc * nw[e] * silu_f(z[e]) : 0.f;
    uint8_t* chunk = p.acts + ((uint64_t)(row / p.tile_tok) * gridDim.x + blockIdx.x) * tm_chunk(p.tile_tok);
    bool over = false;
    tm_pack_oct(chunk, p.tile_tok, row % p.tile_tok, k8, v, over);
    float sum = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
    sum += __shfl_xor_sync(0xffffffffu, sum, 8);
    sum += __shfl_xor_sync(0xffffffffu, sum, 16);
    if (lane < 8) tm_pack_sum(chunk, p.tile_tok, row % p.tile_tok, warp, sum, over);
    if (over) atomicCAS(p.err, 0, DEV_ERR_OVERFLOW);
}

dfl_status launch_tm_gdn_pack(cudaStream_t st, const TmGdn& p) {
    launch_k(tm_gdn_pack_kernel, dim3((unsigned)(p.g.n_v * 128 / 256), (unsigned)(p.rows_pad / 8)), dim3(256), 0, st, p);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

}  // namespace dfl
