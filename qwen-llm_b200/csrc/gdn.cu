// Gated-delta-net block of the verify pass (oracle: Forward::gdn_step,
// crates/qwen-llm/src/forward.rs:940-1107; reference GPU path metal_dflash.rs:9421-9777,
// kernels/ssm_conv.metal:225-277,305-346, kernels/gated_delta_net.metal:382-470).
//
// Rollback design: the recurrence reads the state from one buffer and writes the advanced
// state to another, and the block's raw qkv rows and gate inputs stay in the scratch.  A full
// accept just swaps the two buffers; a partial accept re-runs the same scan device code for
// the first n_keep tokens from the untouched pre-block state, which reproduces the sequential
// state bit for bit without the reference's per-token state checkpoints
// (metal_dflash.rs:5863-5896: n_gdn x N x state bytes written every verify).
#include <cooperative_groups.h>

#include "ops.cuh"

namespace dfl {

namespace cg = cooperative_groups;

__global__ void gdn_conv_restore_kernel(int conv_dim, const float* conv_pre, const float* qkv_raw, int n_keep,
                                        float* conv_state) {
    pdl_prologue();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= conv_dim) return;
    // rows of the virtual sequence {pre[0], pre[1], pre[2], raw[0], ..., raw[n_keep-1]}; keep the last three
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        const int idx = n_keep + t;  // index into the virtual sequence
        conv_state[t * conv_dim + c] = idx < 3 ? conv_pre[idx * conv_dim + c] : qkv_raw[(uint64_t)(idx - 3) * conv_dim + c];
    }
}
dfl_status launch_gdn_conv_restore(cudaStream_t st, const GdnGeom& g, const float* conv_pre, const float* qkv_raw, int n_keep,
                                   float* conv_state) {
    const int cd = g.conv_dim();
    launch_k(gdn_conv_restore_kernel, dim3((cd + 255) / 256), dim3(256), 0, st, cd, conv_pre, qkv_raw, n_keep, conv_state);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

// ---- alpha and beta projections ----------------------------------------------------------------------
// A CTA of 128 threads per four outputs and 512 columns, a thread four columns, rows four at a time.  Its 72 registers a thread find no room beside a
// GEMM CTA: the CTAs start where the last projection has ended early, next to each other, and fill its uneven end.  (As sixteen CTAs behind the z
// projection, each reading all rows, the projections held up the mixer for 7 us.)  Behind a GEMM launched with trigger_late it acquires that launch's mark instead of waiting, and the
// dependency wait at its end makes its own completion say that the GEMM's outputs are there too, which the kernels behind rely on.
constexpr int AB_OUT = 4;
static_assert(AB_COLS == 128 * 4, "four columns a thread");
__global__ void __launch_bounds__(128, 7) ab_proj_kernel(const float* __restrict__ w, const float* xn, int ld_xn, int n_rows, int k, int n_out,
                                                         float* ab_part, LateMark late) {
    __shared__ float red[4][MAX_ROWS * AB_OUT];
    const int o0 = blockIdx.x * AB_OUT, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = blockIdx.y * AB_COLS + threadIdx.x * 4;
    const uint32_t late_seen = late.word ? late_peek(late.word) : 0u;
    float4 wv[AB_OUT];   // outputs beyond the last read its row and are not stored
#pragma unroll
    for (int j = 0; j < AB_OUT; ++j)
        wv[j] = c < k ? *reinterpret_cast<const float4*>(w + (uint64_t)min(o0 + j, n_out - 1) * k + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    pdl_launch_dependents();
    if (late.word) late_acquire(late.word, late.value, late_seen);
    else pdl_wait();
    float4 x[4];
    auto fetch = [&](int t0) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            x[i] = t0 + i < n_rows && c < k ? __ldcg(reinterpret_cast<const float4*>(xn + (uint64_t)(t0 + i) * ld_xn + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    fetch(0);
#pragma unroll 1
    for (int t0 = 0; t0 < MAX_ROWS; t0 += 4) {
        float v[16];   // [token - t0][output]
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < AB_OUT; ++j) v[4 * i + j] = fmaf(wv[j].w, x[i].w, fmaf(wv[j].z, x[i].z, fmaf(wv[j].y, x[i].y, wv[j].x * x[i].x)));
        if (t0 + 4 < MAX_ROWS) fetch(t0 + 4);
#pragma unroll
        for (int n = 8; n >= 1; n >>= 1) {   // lanes 2 l, 2 l + 1 end with half the sum of value l each
            const bool up = lane & (2 * n);
#pragma unroll
            for (int i = 0; i < n; ++i) {
                const float give = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * n);
            }
        }
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
        if (!(lane & 1)) red[warp][t0 * AB_OUT + (lane >> 1)] = v[0];
    }
    __syncthreads();
    if (threadIdx.x < MAX_ROWS * AB_OUT) {
        const int tok = threadIdx.x / AB_OUT, o = o0 + threadIdx.x % AB_OUT;
        const float t = (red[0][threadIdx.x] + red[1][threadIdx.x]) + (red[2][threadIdx.x] + red[3][threadIdx.x]);
        if (tok < n_rows && o < n_out) ab_part[((uint64_t)blockIdx.y * MAX_ROWS + tok) * n_out + o] = t;
    }
    if (late.word) pdl_wait();
}

dfl_status launch_ab_proj(cudaStream_t st, const float* w, const float* xn, int ld_xn, int n_rows, uint64_t k, int n_out, float* ab_part,
                          LateMark late) {
    if (k % 4) return fail(DFL_ERR_BAD_SHAPE, "ab_proj: k must be a multiple of 4");
    launch_k(ab_proj_kernel, dim3((unsigned)((n_out + AB_OUT - 1) / AB_OUT), (unsigned)ab_slices(k)), dim3(128), 0, st, w, xn, ld_xn, n_rows, (int)k,
             n_out, ab_part, late);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

// The recurrent state of eight value channels (rows) in a warp: eight lanes (cg = lane % 8) share two rows, a lane owns the sixteen key channels
// (columns) 4 cg + 32 m .. + 3 of both, as pairs.  What bounds a token is the chain through the sums over lanes: three exchanges here and one to
// pass the coefficient on (with four columns of four rows a lane there were five and one, and 16 tokens took 5.3 us; with eight lanes a row and one
// row each, reading the k and q rows from shared memory was the limit, 32 lanes x 128 bytes a warp and token as here for half the rows).
struct GdnRows {
    uint64_t s[2][8];
    using Vec = uint64_t[8];   // this lane's sixteen columns of a k or q row
    __device__ static __forceinline__ void fetch(Vec& v, const float* row, int cg) {
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(row + 32 * m + 4 * cg);
            v[2 * m] = t.x; v[2 * m + 1] = t.y;
        }
    }
    __device__ __forceinline__ void load(const float* base, int cg) {   // base: the lane's first row
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const float4 t = __ldcg(reinterpret_cast<const float4*>(base + r * 128 + 32 * m + 4 * cg));
                s[r][2 * m] = pack2(t.x, t.y); s[r][2 * m + 1] = pack2(t.z, t.w);
            }
    }
    __device__ __forceinline__ void store(float* base, int cg) const {
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int m = 0; m < 4; ++m) *reinterpret_cast<ulonglong2*>(base + r * 128 + 32 * m + 4 * cg) = make_ulonglong2(s[r][2 * m], s[r][2 * m + 1]);
    }
    // Sums over the lanes of S k (lanes with bit 2 clear) and S q (bit 2 set), of the first row (bit 1 clear) or the second.  The two travel
    // together: a token's output needs the state after its update, which is the state the next token's S k needs, so one
    // pass over the lanes per token serves both and the output never waits in the chain.
    __device__ __forceinline__ float dots(const Vec& k, const Vec& q, int lane) const {
        auto dot = [&](const uint64_t(&a)[8], const Vec& x) {
            uint64_t t0 = mul2(a[0], x[0]), t1 = mul2(a[1], x[1]);
#pragma unroll
            for (int i = 2; i < 8; i += 2) { t0 = fma2(a[i], x[i], t0); t1 = fma2(a[i + 1], x[i + 1], t1); }
            float lo, hi;
            unpack2(add2(t0, t1), lo, hi);
            return lo + hi;
        };
        const float k0 = dot(s[0], k), k1 = dot(s[1], k), q0 = dot(s[0], q), q1 = dot(s[1], q);
        const bool second = lane & 4, up = lane & 2;
        const float a0 = (second ? q0 : k0) + __shfl_xor_sync(0xffffffffu, second ? k0 : q0, 4);
        const float a1 = (second ? q1 : k1) + __shfl_xor_sync(0xffffffffu, second ? k1 : q1, 4);
        const float v = (up ? a1 : a0) + __shfl_xor_sync(0xffffffffu, up ? a0 : a1, 2);
        return v + __shfl_xor_sync(0xffffffffu, v, 1);
    }
    // S = g S + c k^T with c = beta (v - g S k); sk and v: of the lane's row as dots() gives it, meaningful in lanes with bit 2 clear
    __device__ __forceinline__ void update(const Vec& k, float sk, float v, float gexp, float beta, int lane) {
        const float coeff = beta * (v - gexp * sk);
        const float c[2] = {__shfl_sync(0xffffffffu, coeff, lane & 24), __shfl_sync(0xffffffffu, coeff, (lane & 24) + 2)};
        const uint64_t g2 = pack2(gexp, gexp);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint64_t c2 = pack2(c[r], c[r]);
#pragma unroll
            for (int i = 0; i < 8; ++i) s[r][i] = add2(mul2(g2, s[r][i]), mul2(c2, k[i]));
        }
    }
};

// ---- state alone (partial accept) -----------------------------------------------------------------
// grid (n_v, 4 quarters of a head's 128 value channels), block 128: a warp owns 8 state rows (GdnRows); the block's rows and
// gate inputs are staged in shared memory, so the serial part touches no global memory.
__device__ __forceinline__ float gdn_gate(float alpha, float dt_bias, float a_log) { return expf(softplus_f(alpha + dt_bias) * a_log); }

__global__ void __launch_bounds__(128) gdn_rescan_kernel(GdnGeom g, const float* state_in, float* state_out, const float* k_n,
                                                         const float* v, const float* ab, const float* __restrict__ dt_bias,
                                                         const float* __restrict__ a_log, int n_rows) {
    __shared__ __align__(16) float ks[MAX_ROWS][128];
    __shared__ float vs[MAX_ROWS][32], gs[MAX_ROWS], bs[MAX_ROWS];
    pdl_prologue();
    const int h = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cg = lane & 7, hk = h % g.n_k, dv_cta = blockIdx.y * 32, row = warp * 8 + 2 * (lane >> 3);
    const uint64_t s_off = ((uint64_t)h * 128 + dv_cta + row) * 128;
    GdnRows S;
    S.load(state_in + s_off, cg);
    for (int idx = threadIdx.x; idx < n_rows * 32; idx += 128) {
        const int i = idx >> 5, d4 = (idx & 31) * 4;
        *reinterpret_cast<float4*>(&ks[i][d4]) = *reinterpret_cast<const float4*>(k_n + ((uint64_t)i * g.n_k + hk) * 128 + d4);
        vs[i][idx & 31] = v[((uint64_t)i * g.n_v + h) * 128 + dv_cta + (idx & 31)];
    }
    if (threadIdx.x < n_rows) {
        const float* a = ab + (uint64_t)threadIdx.x * (2 * g.n_v) + h;
        gs[threadIdx.x] = gdn_gate(a[0], dt_bias[h], a_log[h]);
        bs[threadIdx.x] = sigmoid_f(a[g.n_v]);
    }
    __syncthreads();
    for (int i = 0; i < n_rows; ++i) {
        GdnRows::Vec k;
        GdnRows::fetch(k, ks[i], cg);
        S.update(k, S.dots(k, k, lane), vs[i][row + ((lane >> 1) & 1)], gs[i], bs[i], lane);
    }
    S.store(state_out + s_off, cg);
}

dfl_status launch_gdn_rescan(cudaStream_t st, const GdnGeom& g, const float* state_in, float* state_out, const float* k_n,
                             const float* v, const float* ab, const float* dt_bias, const float* a_log, int n_rows) {
    launch_k(gdn_rescan_kernel, dim3((unsigned)g.n_v, 4), dim3(128), 0, st, g, state_in, state_out, k_n, v, ab, dt_bias, a_log, n_rows);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

// ---- the whole mixer of a block -------------------------------------------------------------------
// Convolution + SiLU, L2 norms of q and k, delta-rule scan, gated RMSNorm and activation packing in one kernel.  What bounds it is
// latency: every kernel boundary and every cross-stream join would be microseconds of waiting, and inside it every exchange is.
// grid (n_v, 4) in clusters of four along y: CTA = one v head x a quarter (32) of its value channels, 288 threads.
//   * convolution: thread = four channels x four rows; the CTA takes all 128 q and 128 k channels of the head's k head and its own
//     32 v channels (each CTA of the cluster the same q and k: reading 64 KB of partial sums more from L2 costs less than passing
//     the rows around the cluster, which took two cluster barriers before the first token).  What does not come from the kernels before
//     - state, filter taps, old conv rows, weights - is fetched before the dependency wait (earlier passes or a rollback wrote the state and
//     the conv rows, and a pass begins with a plain launch, launch_embed_block, which waits for all of that);
//   * recurrence: four warps own 8 state rows each (GdnRows); everything it reads is in shared memory;
//   * y = rmsnorm(o; eps * 128) * w * silu(z): every CTA writes its quarter's share of a token's sum of squares to all four,
//     one cluster barrier, rank-ordered sum, then packs its 32 columns (one sub-block) of the output projection's activations.
// Loops stay loops: the kernel runs once a layer between kernels that fill the instruction caches, and straight code is fetched once per pass.
// (Three warps running through the code once before the wait, as the glue does, took longer than the 1 - 5 us there are: verify block 2747 -> 2953 us.)
// A row's result does not depend on how many rows the block has.  Measured (9B-class widths, 16 rows, end of the projections to end of the
// mixer): 20.9 -> 13.4 us, 2.4 of them the alpha / beta kernel, which the mixer waited for before.
constexpr int MIX_THREADS = 288;
__global__ void __cluster_dims__(1, 4, 1) __launch_bounds__(MIX_THREADS) gdn_mix_kernel(const GdnMixParams p) {
    __shared__ __align__(16) float raw[(MAX_ROWS + 3) * 288];   // input rows of the convolution behind the three old ones
    __shared__ __align__(16) float qs[MAX_ROWS][128], ks[MAX_ROWS][128], vs[MAX_ROWS][32];
    float(*os)[32] = reinterpret_cast<float(*)[32]>(raw);   // outputs, once the convolution is done
    __shared__ float gs[MAX_ROWS], bs[MAX_ROWS];
    __shared__ float ssp[16][MAX_ROWS];     // partial sums of a row's squares (its RMS norm)
    __shared__ float ss_all[4][MAX_ROWS];   // [cluster rank][token]: sums of squares of the outputs
    cg::cluster_group cluster = cg::this_cluster();
    cluster.barrier_arrive();   // matched by the wait before the write into another CTA's shared memory
    const GdnGeom& g = p.g;
    const int h = blockIdx.x, rank = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int hk = h % g.n_k, conv_dim = g.conv_dim(), dv_cta = rank * 32;
    const bool owner = h < g.n_k;   // of several v heads on one k head, the one that writes the k head's rows
    const int cg = lane & 7, srow = (warp & 3) * 8 + 2 * (lane >> 3);   // state rows of warps 0 - 3 (GdnRows)
    const uint64_t s_off = ((uint64_t)h * 128 + dv_cta + srow) * 128;
    // -- before the dependency wait --
    GdnRows S;
    if (warp < 4) S.load(p.state_in + s_off, cg);
    const int quad = threadIdx.x % 72, rg = threadIdx.x / 72;   // this thread's four channels and rows 4 rg .. + 3
    const int sec = quad < 32 ? 0 : quad < 64 ? 1 : 2;          // q, k, v
    const int c = (sec == 0 ? hk * 128 : sec == 1 ? (g.n_k + hk) * 128 - 128 : (2 * g.n_k + h) * 128 + dv_cta - 256) + 4 * quad;
    float4 tap[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) tap[e] = *reinterpret_cast<const float4*>(p.conv_w + (uint64_t)(c + e) * 4);
    if (rg < 3) *reinterpret_cast<float4*>(&raw[rg * 288 + 4 * quad]) = __ldcg(reinterpret_cast<const float4*>(p.conv_in + rg * conv_dim + c));
    const float dtb = p.dt_bias[h], alog = p.a_log[h];
    const bool finishing = warp >= 4 && warp < 8;                       // 128 threads: (token, four channels)
    const int ftok = (threadIdx.x >> 3) & 15, fquad = threadIdx.x & 7;
    const float4 nw = *reinterpret_cast<const float4*>(p.norm_w + dv_cta + fquad * 4);
    if (p.prefetch_bytes && threadIdx.x == 0) {   // the output projection's weights on their way to L2: its CTAs cannot start beside this kernel's
        const uint64_t n_cta = (uint64_t)gridDim.x * gridDim.y, per = (p.prefetch_bytes / n_cta + 15) & ~15ull;
        const uint64_t at = per * (blockIdx.y * gridDim.x + blockIdx.x);
        if (at < p.prefetch_bytes) bulk_prefetch_l2(p.prefetch + at, (uint32_t)(at + per <= p.prefetch_bytes ? per : p.prefetch_bytes - at));
    }
    pdl_prologue();
    // -- input rows: the split-K slices of the projections --
    {
        float4 xv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) xv[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        const float* base = p.part + (uint64_t)(4 * rg) * p.ld_part + c;
#pragma unroll 4
        for (int s = 0; s < p.splits; ++s, base += (uint64_t)MAX_ROWS * p.ld_part) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (4 * rg + j < p.n_rows) {
                    const float4 t = __ldcg(reinterpret_cast<const float4*>(base + (uint64_t)j * p.ld_part));
                    xv[j].x += t.x; xv[j].y += t.y; xv[j].z += t.z; xv[j].w += t.w;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) *reinterpret_cast<float4*>(&raw[(3 + 4 * rg + j) * 288 + 4 * quad]) = xv[j];
    }
    // slices of alpha and beta (warp 8: lane = 2 token + which) and of the rows' sums of squares (warps 0 - 7: 16 threads a row)
    float ab = 0.f;
    if (warp == 8) {
        if ((lane >> 1) < p.n_rows) {
            const float* src = p.ab_part + (uint64_t)(lane >> 1) * 2 * g.n_v + (lane & 1) * g.n_v + h;
#pragma unroll 8
            for (int s = 0; s < p.slices; ++s) ab += __ldcg(src + (uint64_t)s * MAX_ROWS * 2 * g.n_v);
        }
    } else {
        const int tok = threadIdx.x & 15, part = threadIdx.x >> 4;
        float ss = 0.f;
#pragma unroll 4
        for (int s = part; s < p.n_sumsq; s += 16) ss += __ldcg(p.sumsq + s * MAX_ROWS + tok);
        ssp[part][tok] = ss;
    }
    // the finishing threads fetch their z values now and use them at the end
    float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (finishing && ftok < p.n_rows) {
        const float* zp = p.part + (uint64_t)ftok * p.ld_part + p.z_col + h * 128 + dv_cta + fquad * 4;
#pragma unroll 4
        for (int s = 0; s < p.splits; ++s) {
            const float4 t = __ldcg(reinterpret_cast<const float4*>(zp + (uint64_t)s * MAX_ROWS * p.ld_part));
            z4.x += t.x; z4.y += t.y; z4.z += t.z; z4.w += t.w;
        }
    }
    __syncthreads();
    // -- convolution, SiLU --
    const bool keeper = sec == 2 || (owner && rank == 0);   // writes the channels' rows for a rollback, and the new conv rows
    {
        const float* at = raw + (uint64_t)(4 * rg) * 288 + 4 * quad;
        float4 x0 = *reinterpret_cast<const float4*>(at), x1 = *reinterpret_cast<const float4*>(at + 288), x2 = *reinterpret_cast<const float4*>(at + 576);
        float* dst = sec == 0 ? &qs[4 * rg][4 * quad] : sec == 1 ? &ks[4 * rg][4 * quad - 128] : &vs[4 * rg][4 * quad - 256];
        const int ld = sec == 2 ? 32 : 128;
#pragma unroll 1
        for (int row = 4 * rg; row < 4 * rg + 4; ++row, dst += ld) {
            at += 288;
            const float4 x3 = *reinterpret_cast<const float4*>(at + 576);
            // s = sum_k w[k] * window[k], k ascending (forward.rs:1000-1010)
            auto conv = [](const float4& w, float a, float b, float c, float d) {
                float sacc = 0.f;
                sacc += w.x * a;
                sacc += w.y * b;
                sacc += w.z * c;
                sacc += w.w * d;
                return silu_f(sacc);
            };
            float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
            if (row < p.n_rows) {
                y = make_float4(conv(tap[0], x0.x, x1.x, x2.x, x3.x), conv(tap[1], x0.y, x1.y, x2.y, x3.y), conv(tap[2], x0.z, x1.z, x2.z, x3.z),
                                conv(tap[3], x0.w, x1.w, x2.w, x3.w));
                if (sec == 2) *reinterpret_cast<float4*>(p.v + ((uint64_t)row * g.n_v + h) * 128 + dv_cta + 4 * quad - 256) = y;
                if (keeper) *reinterpret_cast<float4*>(p.qkv_raw + (uint64_t)row * conv_dim + c) = x3;
            }
            *reinterpret_cast<float4*>(dst) = y;
            x0 = x1; x1 = x2; x2 = x3;
        }
    }
    if (keeper && rg < 3)   // new conv state = rows n_rows .. n_rows + 2 of {three old rows, the block's rows}
        *reinterpret_cast<float4*>(p.conv_out + rg * conv_dim + c) = *reinterpret_cast<const float4*>(&raw[(p.n_rows + rg) * 288 + 4 * quad]);
    __syncthreads();
    // -- L2 norms of the k and q rows (forward.rs:1269-1275): warp = a row at a time; gates: warp 8 --
    if (warp < 8) {
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            const int row = warp + 8 * (n & 1);
            float* at = n < 2 ? &ks[row][4 * lane] : &qs[row][4 * lane];
            float4 x = *reinterpret_cast<const float4*>(at);
            const float inv = 1.0f / fmaxf(sqrtf(warp_sum((x.x * x.x + x.y * x.y) + (x.z * x.z + x.w * x.w))), 1e-6f);
            x.x *= inv; x.y *= inv; x.z *= inv; x.w *= inv;
            *reinterpret_cast<float4*>(at) = x;
            if (owner && (row & 3) == rank && row < p.n_rows)   // for a rollback
                *reinterpret_cast<float4*>((n < 2 ? p.k_n : p.q_n) + ((uint64_t)row * g.n_k + hk) * 128 + 4 * lane) = x;
        }
    } else {
        const int tok = lane >> 1, which = lane & 1;
        float ss = 0.f;
#pragma unroll
        for (int q = 0; q < 16; ++q) ss += ssp[q][tok];
        ab *= 1.0f / sqrtf(ss / p.norm_k + p.eps);
        if (tok < p.n_rows) {
            if (which == 0) gs[tok] = gdn_gate(ab, dtb, alog);
            else bs[tok] = sigmoid_f(ab);
            if (rank == 0) p.ab[(uint64_t)tok * (2 * g.n_v) + which * g.n_v + h] = ab;
        }
    }
    __syncthreads();
    // -- per token (forward.rs:1054-1091): sk = S k (state before decay), coeff = beta (v - g sk), S = g S + coeff k, o = S q --
    if (warp < 4) {
        const int vrow = srow + ((lane >> 1) & 1);   // the row whose sums this lane ends with
        GdnRows::Vec k, q;   // q: of the token before (none yet)
        GdnRows::fetch(k, ks[0], cg);
        GdnRows::fetch(q, ks[0], cg);
        float vi = vs[0][vrow], gi = gs[0], bi = bs[0];
#pragma unroll 2
        for (int i = 0; i < p.n_rows; ++i) {   // the next token's operands are fetched while this one's sums travel
            const int in = i + 1 < p.n_rows ? i + 1 : i;
            GdnRows::Vec qn, kn;
            const float sk = S.dots(k, q, lane);
            GdnRows::fetch(qn, qs[i], cg);
            GdnRows::fetch(kn, ks[in], cg);
            const float vn = vs[in][vrow], gn = gs[in], bn = bs[in];
            if (i > 0 && (lane & 5) == 4) os[i - 1][vrow] = sk;
            S.update(k, sk, vi, gi, bi, lane);
#pragma unroll
            for (int x = 0; x < 8; ++x) { k[x] = kn[x]; q[x] = qn[x]; }
            vi = vn; gi = gn; bi = bn;
        }
        const float o = S.dots(q, q, lane);
        if ((lane & 5) == 4) os[p.n_rows - 1][vrow] = o;
    }
    cluster.barrier_wait();   // every CTA of the cluster has started: its shared memory may be written
    __syncthreads();
    if (warp < 8) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int i = warp + 8 * half;
            const float x = i < p.n_rows ? os[i][lane] : 0.f;
            const float sq = warp_sum(x * x);
            if (lane < 4) *cluster.map_shared_rank(&ss_all[rank][i], (unsigned)lane) = sq;
        }
    }
    cluster.sync();   // all shares have arrived; nothing is written into another CTA after this point
    if (warp < 4) S.store(p.state_out + s_off, cg);
    if (finishing) {
        const int tok = ftok, quad = fquad, col0 = h * 128 + dv_cta + quad * 4;
        float o[4] = {0.f, 0.f, 0.f, 0.f};
        if (tok < p.n_rows) {
            const float tot = ((ss_all[0][tok] + ss_all[1][tok]) + ss_all[2][tok]) + ss_all[3][tok];   // rank order: the same sum in all four CTAs
            const float sc = 1.0f / sqrtf(tot / 128.f + 1e-6f * 128.f);   // eps = RMS_EPS * head_dim (forward.rs:1098)
            o[0] = os[tok][quad * 4 + 0] * sc * nw.x * silu_f(z4.x);
            o[1] = os[tok][quad * 4 + 1] * sc * nw.y * silu_f(z4.y);
            o[2] = os[tok][quad * 4 + 2] * sc * nw.z * silu_f(z4.z);
            o[3] = os[tok][quad * 4 + 3] * sc * nw.w * silu_f(z4.w);
        }
        uint8_t* chunk = p.acts + (uint64_t)(col0 >> 8) * act_chunk_dev(p.layout);
        bool over = false;
        pack_quad_any(chunk, p.layout, tok, col0 & 255, o, over);
        if (p.layout == ACT_F16 || p.layout == ACT_TS) {
            float sum = o[0] + o[1] + o[2] + o[3];   // the CTA's 32 channels are one 32-column sub-block: eight neighbouring threads
#pragma unroll
            for (int of = 4; of > 0; of >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, of);
            if (quad == 0) store_subsum(chunk, p.layout, tok, (col0 & 255) >> 5, sum, over);
        }
        if (over) atomicCAS(p.err, 0, DEV_ERR_OVERFLOW);
    }
}

dfl_status launch_gdn_mix(cudaStream_t st, const GdnMixParams& p) {
    if (p.g.hd != 128 || p.g.conv_k != 4) return fail(DFL_ERR_UNSUPPORTED, "gdn: head_dim must be 128 and conv kernel 4");
    launch_k(gdn_mix_kernel, dim3((unsigned)p.g.n_v, 4), dim3(MIX_THREADS), 0, st, p);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

}  // namespace dfl
