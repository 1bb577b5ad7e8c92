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

// The recurrent state of four value channels (rows) in a warp: a lane owns four key channels (columns 4 lane .. + 3) of every
// row, so that one 16-byte load of a k or q row serves all four (with eight lanes a row each warp read every k and q row
// sixteen bytes at a time per row group, and the 16-token loop was bound by shared-memory bandwidth: 530 clocks a token).
// Slot r of lane l holds row r ^ (l / 8): the first two steps of a sum over the lanes then always pass on the upper slots, and
// lane group l / 8 ends with the sum of row l / 8.
struct GdnRows {
    float4 s[4];
    __device__ __forceinline__ void load(const float* base, int rr) {   // base: row 0, this lane's columns
#pragma unroll
        for (int r = 0; r < 4; ++r) s[r] = __ldcg(reinterpret_cast<const float4*>(base + (r ^ rr) * 128));
    }
    __device__ __forceinline__ void store(float* base, int rr) const {
#pragma unroll
        for (int r = 0; r < 4; ++r) *reinterpret_cast<float4*>(base + (r ^ rr) * 128) = s[r];
    }
    // Sums over the lanes of S k and S q: row l / 8 of S k in lanes with bit 2 clear, of S q in the others.  The two travel
    // together: a token's output needs the state after its update, which is the state the next token's S k needs, so one
    // pass over the lanes per token serves both and the output never waits in the chain.
    __device__ __forceinline__ float dots(const float4 k, const float4 q, int lane) const {
        float pk[4], pq[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            pk[r] = fmaf(s[r].w, k.w, fmaf(s[r].z, k.z, fmaf(s[r].y, k.y, s[r].x * k.x)));
            pq[r] = fmaf(s[r].w, q.w, fmaf(s[r].z, q.z, fmaf(s[r].y, q.y, s[r].x * q.x)));
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            pk[r] += __shfl_xor_sync(0xffffffffu, pk[r + 2], 16);
            pq[r] += __shfl_xor_sync(0xffffffffu, pq[r + 2], 16);
        }
        pk[0] += __shfl_xor_sync(0xffffffffu, pk[1], 8);
        pq[0] += __shfl_xor_sync(0xffffffffu, pq[1], 8);
        const bool up = lane & 4;
        float v = (up ? pq[0] : pk[0]) + __shfl_xor_sync(0xffffffffu, up ? pk[0] : pq[0], 4);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        return v;
    }
    // S = g S + c k^T with c = beta (v - g S k); sk and v: of row l / 8, meaningful in lanes with bit 2 clear
    __device__ __forceinline__ void update(const float4 k, float sk, float v, float gexp, float beta, int rr) {
        const float coeff = beta * (v - gexp * sk);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float c = __shfl_sync(0xffffffffu, coeff, (r ^ rr) * 8);
            s[r].x = __fadd_rn(__fmul_rn(gexp, s[r].x), __fmul_rn(c, k.x));
            s[r].y = __fadd_rn(__fmul_rn(gexp, s[r].y), __fmul_rn(c, k.y));
            s[r].z = __fadd_rn(__fmul_rn(gexp, s[r].z), __fmul_rn(c, k.z));
            s[r].w = __fadd_rn(__fmul_rn(gexp, s[r].w), __fmul_rn(c, k.w));
        }
    }
};

// ---- state alone (partial accept) -----------------------------------------------------------------
// grid (n_v, 4 quarters of a head's 128 value channels), block 256: a warp owns 4 state rows (GdnRows); the block's rows and
// gate inputs are staged in shared memory, so the serial part touches no global memory.
__device__ __forceinline__ float gdn_gate(float alpha, float dt_bias, float a_log) { return expf(softplus_f(alpha + dt_bias) * a_log); }

__global__ void __launch_bounds__(256) gdn_rescan_kernel(GdnGeom g, const float* state_in, float* state_out, const float* k_n,
                                                         const float* v, const float* ab, const float* __restrict__ dt_bias,
                                                         const float* __restrict__ a_log, int n_rows) {
    __shared__ __align__(16) float ks[MAX_ROWS][128];
    __shared__ float vs[MAX_ROWS][32], gs[MAX_ROWS], bs[MAX_ROWS];
    pdl_prologue();
    const int h = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rr = lane >> 3, hk = h % g.n_k, dv_cta = blockIdx.y * 32;
    const uint64_t s_off = ((uint64_t)h * 128 + dv_cta + warp * 4) * 128 + 4 * lane;
    GdnRows S;
    S.load(state_in + s_off, rr);
    for (int idx = threadIdx.x; idx < n_rows * 32; idx += 256) {
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
        const float4 k = *reinterpret_cast<const float4*>(&ks[i][4 * lane]);
        S.update(k, S.dots(k, k, lane), vs[i][warp * 4 + rr], gs[i], bs[i], rr);
    }
    S.store(state_out + s_off, rr);
}

dfl_status launch_gdn_rescan(cudaStream_t st, const GdnGeom& g, const float* state_in, float* state_out, const float* k_n,
                             const float* v, const float* ab, const float* dt_bias, const float* a_log, int n_rows) {
    launch_k(gdn_rescan_kernel, dim3((unsigned)g.n_v, 4), dim3(256), 0, st, g, state_in, state_out, k_n, v, ab, dt_bias, a_log, n_rows);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

// ---- the whole mixer of a block -------------------------------------------------------------------
// Convolution + SiLU, L2 norms of q and k, delta-rule scan, gated RMSNorm and activation packing in one
// kernel.  What bounds it is latency: as four kernels (two of them on side streams) the 16 rows took 28 us between the end of
// the input projections (alpha / beta ride on CTAs behind the last of them) and the start of the output projection, of which 1.8 us is the recurrence; every kernel boundary
// and every cross-stream join is several us of waiting.
// grid (n_v, 4) in clusters of four along y: CTA = one v head x a quarter (32) of its value channels, 256 threads.
//   * convolution: warp = two rows, lane = four channels of the CTA's share: 32 q and 32 k channels of the head's k head and
//     its own 32 v channels.  The q and k shares travel to the other three CTAs through distributed shared memory together
//     with their sums of squares, so that each CTA holds the full 16 x 128 q and k rows and normalises them itself;
//   * recurrence: a warp owns 4 state rows (GdnRows); everything it reads is in shared memory.  State, filter taps and old conv
//     rows are fetched before the dependency wait (earlier passes or a rollback wrote them, and a pass begins with a plain
//     launch, launch_embed_block, which waits for all of that), the z rows are requested before the token loop;
//   * y = rmsnorm(o; eps * 128) * w * silu(z): every CTA writes its quarter's share of a token's sum of squares to all four,
//     one cluster barrier, rank-ordered sum, then packs its 32 columns (one sub-block) of the output projection's activations.
// A row's result does not depend on how many rows the block has.
__global__ void __cluster_dims__(1, 4, 1) __launch_bounds__(256) gdn_mix_kernel(const GdnMixParams p) {
    __shared__ __align__(16) float qs[MAX_ROWS][128], ks[MAX_ROWS][128], vs[MAX_ROWS][32];
    __shared__ float os[MAX_ROWS][32], gs[MAX_ROWS], bs[MAX_ROWS];
    __shared__ float inv[2][MAX_ROWS];
    __shared__ float nrm[4][2][MAX_ROWS];   // [cluster rank][q, k][row]: sums of squares over the rank's 32 channels
    __shared__ float ss_all[4][MAX_ROWS];   // [cluster rank][token]: sums of squares of the outputs
    cg::cluster_group cluster = cg::this_cluster();
    cluster.barrier_arrive();   // matched by the wait before the first write into another CTA's shared memory
    const GdnGeom& g = p.g;
    const int h = blockIdx.x, rank = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int hk = h % g.n_k, conv_dim = g.conv_dim(), dv_cta = rank * 32;
    const bool owner = h < g.n_k;   // of several v heads on one k head, the one that writes the k head's rows
    const int rr = lane >> 3, lg = lane & 7;
    const uint64_t s_off = ((uint64_t)h * 128 + dv_cta + warp * 4) * 128 + 4 * lane;
    // -- before the dependency wait --
    GdnRows S;
    S.load(p.state_in + s_off, rr);
    const int sec = lane >> 3;   // 0 q, 1 k, 2 v, 3 idle
    const int c = (sec == 0 ? hk : sec == 1 ? g.n_k + hk : 2 * g.n_k + h) * 128 + dv_cta + 4 * lg;   // this lane's four channels
    float4 tap[4], old[3];
#pragma unroll
    for (int e = 0; e < 4; ++e) tap[e] = sec < 3 ? *reinterpret_cast<const float4*>(p.conv_w + (uint64_t)(c + e) * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int t = 0; t < 3; ++t)
        old[t] = sec < 3 && warp < 2 ? __ldcg(reinterpret_cast<const float4*>(p.conv_in + t * conv_dim + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float dtb = p.dt_bias[h], alog = p.a_log[h];
    pdl_prologue();
    // -- convolution: rows 2 warp, 2 warp + 1; xv[k] = input at row 2 warp - 3 + k --
    const int i0 = 2 * warp;
    float4 xv[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) xv[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (warp == 0) { xv[0] = old[0]; xv[1] = old[1]; xv[2] = old[2]; }
    if (warp == 1) xv[0] = old[2];
    if (sec < 3) {
#pragma unroll 4
        for (int s = 0; s < p.splits; ++s) {
            const float* base = p.part + (uint64_t)s * MAX_ROWS * p.ld_part + c;
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                const int row = i0 - 3 + k;
                if (row >= 0 && row < p.n_rows) {
                    const float4 a = __ldcg(reinterpret_cast<const float4*>(base + (uint64_t)row * p.ld_part));
                    xv[k].x += a.x; xv[k].y += a.y; xv[k].z += a.z; xv[k].w += a.w;
                }
            }
        }
    }
    float alpha = 0.f, beta = 0.f;
    if (threadIdx.x < p.n_rows) {
        alpha = __ldcg(p.ab + (uint64_t)threadIdx.x * (2 * g.n_v) + h);
        beta = __ldcg(p.ab + (uint64_t)threadIdx.x * (2 * g.n_v) + g.n_v + h);
    }
    // the finishing threads (token, four channels) fetch their z values now and use them after the token loop
    const int ftok = threadIdx.x >> 3, fquad = threadIdx.x & 7;
    float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (threadIdx.x < 128 && ftok < p.n_rows) {
        const float* zp = p.part + (uint64_t)ftok * p.ld_part + p.z_col + h * 128 + dv_cta + fquad * 4;
#pragma unroll 4
        for (int s = 0; s < p.splits; ++s) {
            const float4 t = __ldcg(reinterpret_cast<const float4*>(zp + (uint64_t)s * MAX_ROWS * p.ld_part));
            z4.x += t.x; z4.y += t.y; z4.z += t.z; z4.w += t.w;
        }
    }
    // -- convolution output, SiLU; q and k rows to every CTA of the cluster --
    float y[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const float in[4][4] = {{xv[j].x, xv[j + 1].x, xv[j + 2].x, xv[j + 3].x}, {xv[j].y, xv[j + 1].y, xv[j + 2].y, xv[j + 3].y},
                                {xv[j].z, xv[j + 1].z, xv[j + 2].z, xv[j + 3].z}, {xv[j].w, xv[j + 1].w, xv[j + 2].w, xv[j + 3].w}};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            // s = sum_k w[k] * window[k], k ascending (forward.rs:1000-1010)
            float sacc = 0.f;
            sacc += tap[e].x * in[e][0];
            sacc += tap[e].y * in[e][1];
            sacc += tap[e].z * in[e][2];
            sacc += tap[e].w * in[e][3];
            y[j][e] = i0 + j < p.n_rows ? silu_f(sacc) : 0.f;
        }
    }
    cluster.barrier_wait();   // every CTA of the cluster has started: its shared memory may be written
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int row = i0 + j;
        const float4 y4 = make_float4(y[j][0], y[j][1], y[j][2], y[j][3]);
        float sq = (y4.x * y4.x + y4.y * y4.y) + (y4.z * y4.z + y4.w * y4.w);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if (sec < 2) {
            float* dst = sec == 0 ? &qs[row][dv_cta + 4 * lg] : &ks[row][dv_cta + 4 * lg];
#pragma unroll
            for (unsigned r = 0; r < 4; ++r) {
                *reinterpret_cast<float4*>(cluster.map_shared_rank(dst, r)) = y4;
                if (lg == 0) *cluster.map_shared_rank(&nrm[rank][sec][row], r) = sq;
            }
        } else if (sec == 2) {
            *reinterpret_cast<float4*>(&vs[row][4 * lg]) = y4;
            if (row < p.n_rows) *reinterpret_cast<float4*>(p.v + ((uint64_t)row * g.n_v + h) * 128 + dv_cta + 4 * lg) = y4;
        }
        if (row < p.n_rows && (sec == 2 || (sec < 2 && owner))) *reinterpret_cast<float4*>(p.qkv_raw + (uint64_t)row * conv_dim + c) = xv[j + 3];
    }
    if (sec == 2 || (sec < 2 && owner)) {
        // new conv state = rows n_rows .. n_rows + 2 of {three old rows, the block's rows}
#pragma unroll
        for (int t = 0; t < 3; ++t) {
            const int r = p.n_rows + t - 3;   // row of the block, or below zero an old row
            if (r < 0) {
                if (warp == 0) *reinterpret_cast<float4*>(p.conv_out + t * conv_dim + c) = r == -2 ? old[1] : old[2];   // n_rows >= 1: never old[0]
            } else if (r == i0 || r == i0 + 1) {
                *reinterpret_cast<float4*>(p.conv_out + t * conv_dim + c) = r == i0 ? xv[3] : xv[4];
            }
        }
    }
    cluster.sync();
    if (threadIdx.x >= 64 && threadIdx.x < 96) {   // 1 / max(||y||, eps) of the q and k rows (forward.rs:1269-1275)
        const int row = lane & 15, sel = lane >> 4;
        inv[sel][row] = 1.0f / fmaxf(sqrtf(((nrm[0][sel][row] + nrm[1][sel][row]) + nrm[2][sel][row]) + nrm[3][sel][row]), 1e-6f);
    }
    if (threadIdx.x < p.n_rows) {
        gs[threadIdx.x] = gdn_gate(alpha, dtb, alog);
        bs[threadIdx.x] = sigmoid_f(beta);
    }
    __syncthreads();
    // -- per token (forward.rs:1054-1091): sk = S k (state before decay), coeff = beta (v - g sk), S = g S + coeff k, o = S q --
    auto row4 = [&](const float(*rows)[128], int sel, int i) {
        float4 x = *reinterpret_cast<const float4*>(&rows[i][4 * lane]);
        const float f = inv[sel][i];
        x.x *= f; x.y *= f; x.z *= f; x.w *= f;
        return x;
    };
    float4 k4 = row4(ks, 1, 0), q4 = k4;   // q of the token before (none yet)
    float vi = vs[0][warp * 4 + rr], gi = gs[0], bi = bs[0];
#pragma unroll 2
    for (int i = 0; i < p.n_rows; ++i) {   // the next token's operands are fetched while this one's sums travel
        const int in = i + 1 < p.n_rows ? i + 1 : i;
        const float4 qn = row4(qs, 0, i), kn = row4(ks, 1, in);
        const float vn = vs[in][warp * 4 + rr], gn = gs[in], bn = bs[in];
        const float sk = S.dots(k4, q4, lane);
        if (i > 0 && lg == 4) os[i - 1][warp * 4 + rr] = sk;
        S.update(k4, sk, vi, gi, bi, rr);
        k4 = kn; q4 = qn; vi = vn; gi = gn; bi = bn;
    }
    {
        const float o = S.dots(q4, q4, lane);
        if (lg == 4) os[p.n_rows - 1][warp * 4 + rr] = o;
    }
    S.store(p.state_out + s_off, rr);
    if (owner)   // the normalised rows of this CTA's share, for a rollback
        for (int idx = threadIdx.x; idx < p.n_rows * 16; idx += 256) {
            const int row = idx >> 4, sel = (idx >> 3) & 1, d = dv_cta + (idx & 7) * 4;
            float4 x = *reinterpret_cast<const float4*>(sel ? &ks[row][d] : &qs[row][d]);
            const float f = inv[sel][row];
            x.x *= f; x.y *= f; x.z *= f; x.w *= f;
            *reinterpret_cast<float4*>((sel ? p.k_n : p.q_n) + ((uint64_t)row * g.n_k + hk) * 128 + d) = x;
        }
    __syncthreads();
    for (int i = warp; i < MAX_ROWS; i += 8) {
        const float x = i < p.n_rows ? os[i][lane] : 0.f;
        const float sq = warp_sum(x * x);
        if (lane < 4) *cluster.map_shared_rank(&ss_all[rank][i], (unsigned)lane) = sq;
    }
    cluster.sync();   // all shares have arrived; nothing is written into another CTA after this point
    if (threadIdx.x < 128) {
        const int tok = ftok, quad = fquad, col0 = h * 128 + dv_cta + quad * 4;
        float o[4] = {0.f, 0.f, 0.f, 0.f};
        if (tok < p.n_rows) {
            const float tot = ((ss_all[0][tok] + ss_all[1][tok]) + ss_all[2][tok]) + ss_all[3][tok];   // rank order: the same sum in all four CTAs
            const float sc = 1.0f / sqrtf(tot / 128.f + 1e-6f * 128.f);   // eps = RMS_EPS * head_dim (forward.rs:1098)
            const float4 nw = *reinterpret_cast<const float4*>(p.norm_w + dv_cta + quad * 4);
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
    launch_k(gdn_mix_kernel, dim3((unsigned)p.g.n_v, 4), dim3(256), 0, st, p);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

}  // namespace dfl
