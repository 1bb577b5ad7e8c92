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
// grid (n_v, 4 quarters of the value channels), 256 threads: a warp owns four state rows and a lane four key channels of each,
// so that one 16-byte load of a k or q row serves all four (with eight lanes a row the kernel was bound by shared-memory
// bandwidth at the token scan's time).  The sums over the lanes halve the values they carry at every step; a lane keeps its
// rows and tokens in an order rotated by its own number, so that what it passes on is always the upper half and no
// select is needed.  Lane 8 r + l ends up with tokens 2 l, 2 l + 1 of row r.  The next block's rows travel with cp.async.
constexpr int SCAN_BLK = 16;
struct ScanSmem {
    float qs[2][SCAN_BLK][128], ks[2][SCAN_BLK][128], vs[2][SCAN_BLK][32];
    float L[SCAN_BLK][SCAN_BLK + 4], M[SCAN_BLK][SCAN_BLK + 4];   // L[j][i] (column major: one step of the substitution reads a column), M[i][j]
    float C[32][SCAN_BLK + 4];   // c_j D_15,j of every state row
    float gs[2][SCAN_BLK], bs[2][SCAN_BLK], G[SCAN_BLK], D[SCAN_BLK];
};
__global__ void __launch_bounds__(256, 1) tm_gdn_scan_kernel(const TmGdn p) {
    extern __shared__ __align__(16) uint8_t scan_smem[];
    ScanSmem& sm = *reinterpret_cast<ScanSmem*>(scan_smem);
    const GdnGeom& g = p.g;
    const int h = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rr = lane >> 3, lg = lane & 7, hk = h % g.n_k;
    const int dv_cta = blockIdx.y * 32, dv_l = warp * 4 + rr, dv = dv_cta + dv_l;   // the row whose tokens this lane finishes
    const float dtb = p.dt_bias[h], alog = p.a_log[h];
    pdl_prologue();
    float S[4][4];   // S[r]: row r ^ rr of the warp's four, key channels 4 lane .. + 3
    const uint64_t s_off = ((uint64_t)h * 128 + dv_cta + warp * 4) * 128 + 4 * lane;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const float4 s4 = __ldcg(reinterpret_cast<const float4*>(p.state_in + s_off + (r ^ rr) * 128));
        S[r][0] = s4.x; S[r][1] = s4.y; S[r][2] = s4.z; S[r][3] = s4.w;
    }
    auto cp16 = [](void* dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory"); };
    // block boundaries: multiples of 16 from the start, and the first row of the part a rollback may undo
    const int ckpt = p.last_rows ? p.n_rows - p.last_rows : 0;
    auto next_of = [&](int r0) { return min(r0 < ckpt && r0 + SCAN_BLK > ckpt ? ckpt : r0 + SCAN_BLK, p.n_rows); };
    auto fetch = [&](int r0, int buf) {   // rows beyond the block's are zeros: they add nothing and decay nothing
        const int n = next_of(r0) - r0;
        for (int i = threadIdx.x; i < SCAN_BLK * 32; i += 256) {
            const int r = i >> 5, d = (i & 31) * 4;
            if (r < n) {
                cp16(&sm.qs[buf][r][d], p.q_n + ((uint64_t)(r0 + r) * g.n_k + hk) * 128 + d);
                cp16(&sm.ks[buf][r][d], p.k_n + ((uint64_t)(r0 + r) * g.n_k + hk) * 128 + d);
            } else {
                *reinterpret_cast<float4*>(&sm.qs[buf][r][d]) = make_float4(0.f, 0.f, 0.f, 0.f);
                *reinterpret_cast<float4*>(&sm.ks[buf][r][d]) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        if (threadIdx.x < SCAN_BLK * 8) {
            const int r = threadIdx.x >> 3, d = (threadIdx.x & 7) * 4;
            if (r < n) cp16(&sm.vs[buf][r][d], p.v + ((uint64_t)(r0 + r) * g.n_v + h) * 128 + dv_cta + d);
            else *reinterpret_cast<float4*>(&sm.vs[buf][r][d]) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // gate inputs of a block: loaded a block ahead by 16 threads, turned into gates when the block starts
    float ga = 0.f, gb = 0.f;
    auto gate_load = [&](int r0) {
        if (threadIdx.x < SCAN_BLK && r0 + (int)threadIdx.x < p.n_rows) {
            const float* a = p.ab + (uint64_t)(r0 + threadIdx.x) * (2 * g.n_v) + h;
            ga = __ldcg(a);
            gb = __ldcg(a + g.n_v);
        }
    };
    auto gate_store = [&](int r0, int buf) {
        if (threadIdx.x >= SCAN_BLK) return;
        const int n = next_of(r0) - r0, i = threadIdx.x;
        sm.gs[buf][i] = i < n ? expf(softplus_f(ga + dtb) * alog) : 1.f;
        sm.bs[buf][i] = i < n ? sigmoid_f(gb) : 0.f;
        const int kr = r0 + i - ckpt;
        if (p.last_rows && kr >= 0 && i < n && blockIdx.y == 0) {
            p.keep_ab[(uint64_t)kr * (2 * g.n_v) + h] = ga;
            p.keep_ab[(uint64_t)kr * (2 * g.n_v) + g.n_v + h] = gb;
        }
    };
    auto put = [&](float* dst) {
#pragma unroll
        for (int r = 0; r < 4; ++r) *reinterpret_cast<float4*>(dst + s_off + (r ^ rr) * 128) = make_float4(S[r][0], S[r][1], S[r][2], S[r][3]);
    };
    // dot products of the four rows with the block's sixteen rows of `src`, summed over the lanes: tokens 2 lg and 2 lg + 1 of row rr
    auto dots = [&](const float (*src)[128], float& d0, float& d1) {
        float v[64];   // [row slot][token slot]; token slot t is token t ^ 2 lg
#pragma unroll
        for (int t = 0; t < SCAN_BLK; ++t) {
            const float4 x = *reinterpret_cast<const float4*>(&src[t ^ (2 * lg)][4 * lane]);
#pragma unroll
            for (int r = 0; r < 4; ++r) v[16 * r + t] = fmaf(S[r][3], x.w, fmaf(S[r][2], x.z, fmaf(S[r][1], x.y, S[r][0] * x.x)));
        }
#pragma unroll
        for (int n = 32; n >= 2; n >>= 1) {
#pragma unroll
            for (int i = 0; i < n; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i + n], n / 2);
        }
        d0 = v[0]; d1 = v[1];
    };
    // the conv rows before the last block replace the pass's first ones, which the front kernel has read; one slice per CTA
    if (p.last_rows) {
        const int n = 3 * g.conv_dim() / 4, per = (n + gridDim.x * gridDim.y - 1) / (gridDim.x * gridDim.y);
        const int c0 = (blockIdx.y * gridDim.x + blockIdx.x) * per;
        for (int i = c0 + threadIdx.x; i < min(n, c0 + per); i += 256)
            reinterpret_cast<float4*>(p.conv_in)[i] = __ldcg(reinterpret_cast<const float4*>(p.keep_pre) + i);
    }
    fetch(0, 0);
    gate_load(0);
    int buf = 0;
    for (int r0 = 0; r0 < p.n_rows; buf ^= 1) {
        const int r1 = next_of(r0), n = r1 - r0;
        gate_store(r0, buf);
        if (r1 < p.n_rows) {
            fetch(r1, buf ^ 1);
            gate_load(r1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        // ---- the block's Gram matrices and decays: a thread computes a 4 x 4 tile of K K^T or Q K^T over sixteen of the 128 channels,
        // eight lanes share a tile (the eight warps: 2 matrices x 16 tiles)
        {
            const int tile = threadIdx.x >> 3, i0 = ((tile >> 2) & 3) * 4, j0 = (tile & 3) * 4;
            const bool is_m = tile >= 16;
            if (j0 <= i0) {   // uniform over the tile's eight lanes
                const float(*ri)[128] = is_m ? sm.qs[buf] : sm.ks[buf];
                float acc[16];
#pragma unroll
                for (int x = 0; x < 16; ++x) acc[x] = 0.f;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float4 a[4], b[4];
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        a[x] = *reinterpret_cast<const float4*>(&ri[i0 + x][32 * c + 4 * lg]);
                        b[x] = *reinterpret_cast<const float4*>(&sm.ks[buf][j0 + x][32 * c + 4 * lg]);
                    }
#pragma unroll
                    for (int x = 0; x < 4; ++x)
#pragma unroll
                        for (int y = 0; y < 4; ++y)
                            acc[4 * x + y] = fmaf(a[x].w, b[y].w, fmaf(a[x].z, b[y].z, fmaf(a[x].y, b[y].y, fmaf(a[x].x, b[y].x, acc[4 * x + y]))));
                }
                const uint32_t mask = 0xffu << (lane & 24);
#pragma unroll
                for (int n = 8; n >= 2; n >>= 1) {   // lane lg keeps entries 2 lg, 2 lg + 1
                    const bool up = lg & (n / 2);
#pragma unroll
                    for (int x = 0; x < n; ++x) {
                        const float give = up ? acc[x] : acc[x + n], keep = up ? acc[x + n] : acc[x];
                        acc[x] = keep + __shfl_xor_sync(mask, give, n / 2);
                    }
                }
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const int e = 2 * lg + x, i = i0 + (e >> 2), j = j0 + (e & 3);
                    float dec = 1.f;   // D_ij
#pragma unroll
                    for (int t = 1; t < SCAN_BLK; ++t) dec *= (t > j && t <= i) ? sm.gs[buf][t] : 1.f;
                    if (is_m) sm.M[i][j] = j <= i ? dec * acc[x] : 0.f;
                    else sm.L[j][i] = j < i ? sm.bs[buf][i] * dec * acc[x] : 0.f;
                }
            } else if (is_m) {   // above the diagonal
                sm.M[i0 + (lg >> 1)][j0 + 2 * (lg & 1)] = 0.f;
                sm.M[i0 + (lg >> 1)][j0 + 2 * (lg & 1) + 1] = 0.f;
            }
            if (threadIdx.x >= 256 - 32) {   // G_i and D_15,i
                const int i = lane & 15;
                float v = 1.f;
#pragma unroll
                for (int t = 0; t < SCAN_BLK; ++t) v *= (lane < 16 ? t <= i : t > i) ? sm.gs[buf][t] : 1.f;
                (lane < 16 ? sm.G : sm.D)[i] = v;
            }
        }
        // ---- u = S0 k, w = S0 q
        float u01[2], w01[2];
        dots(sm.ks[buf], u01[0], u01[1]);
        dots(sm.qs[buf], w01[0], w01[1]);
        __syncthreads();   // L, M, G, D
        // ---- substitution, by all eight lanes of a row alike: u becomes c
        float u[SCAN_BLK];
#pragma unroll
        for (int i = 0; i < SCAN_BLK; ++i) u[i] = __shfl_sync(0xffffffffu, u01[i & 1], 8 * rr + (i >> 1));
#pragma unroll
        for (int i = 0; i < SCAN_BLK; ++i) u[i] = sm.bs[buf][i] * (sm.vs[buf][i][dv_l] - sm.G[i] * u[i]);
#pragma unroll
        for (int j = 0; j < SCAN_BLK - 1; ++j) {
#pragma unroll
            for (int i4 = (j + 1) / 4; i4 < 4; ++i4) {
                const float4 l = *reinterpret_cast<const float4*>(&sm.L[j][4 * i4]);
                if (4 * i4 > j) u[4 * i4] = fmaf(-l.x, u[j], u[4 * i4]);
                if (4 * i4 + 1 > j) u[4 * i4 + 1] = fmaf(-l.y, u[j], u[4 * i4 + 1]);
                if (4 * i4 + 2 > j) u[4 * i4 + 2] = fmaf(-l.z, u[j], u[4 * i4 + 2]);
                if (4 * i4 + 3 > j) u[4 * i4 + 3] = fmaf(-l.w, u[j], u[4 * i4 + 3]);
            }
        }
        // ---- outputs of tokens 2 lg, 2 lg + 1; c for the state
        float* o_row = p.o + (uint64_t)r0 * g.n_v * 128 + h * 128 + dv;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int i = 2 * lg + t;
            float o0 = sm.G[i] * w01[t], o1 = 0.f;
#pragma unroll
            for (int j4 = 0; j4 < 4; ++j4) {
                const float4 m = *reinterpret_cast<const float4*>(&sm.M[i][4 * j4]);
                o0 = fmaf(m.x, u[4 * j4], o0); o1 = fmaf(m.y, u[4 * j4 + 1], o1);
                o0 = fmaf(m.z, u[4 * j4 + 2], o0); o1 = fmaf(m.w, u[4 * j4 + 3], o1);
            }
            if (i < n) o_row[(uint64_t)i * g.n_v * 128] = o0 + o1;
        }
        if (lg == 0) {
#pragma unroll
            for (int j4 = 0; j4 < 4; ++j4) {
                const float4 d = *reinterpret_cast<const float4*>(&sm.D[4 * j4]);
                *reinterpret_cast<float4*>(&sm.C[dv_l][4 * j4]) = make_float4(u[4 * j4] * d.x, u[4 * j4 + 1] * d.y, u[4 * j4 + 2] * d.z, u[4 * j4 + 3] * d.w);
            }
        }
        __syncwarp();
        // ---- state
        const float Gend = sm.G[SCAN_BLK - 1];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[r][e] *= Gend;
#pragma unroll
        for (int i4 = 0; i4 < 4; ++i4) {
            float4 k4[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) k4[t] = *reinterpret_cast<const float4*>(&sm.ks[buf][4 * i4 + t][4 * lane]);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float4 c4 = *reinterpret_cast<const float4*>(&sm.C[warp * 4 + (r ^ rr)][4 * i4]);
                const float c[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    S[r][0] = fmaf(c[t], k4[t].x, S[r][0]); S[r][1] = fmaf(c[t], k4[t].y, S[r][1]);
                    S[r][2] = fmaf(c[t], k4[t].z, S[r][2]); S[r][3] = fmaf(c[t], k4[t].w, S[r][3]);
                }
            }
        }
        r0 = r1;
        if (p.last_rows && r0 == ckpt) put(p.state_in);
        __syncthreads();   // this block's buffers, L, M, G and D are free
    }
    put(p.state_out);
}

dfl_status launch_tm_gdn_scan(cudaStream_t st, const TmGdn& p) {
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
