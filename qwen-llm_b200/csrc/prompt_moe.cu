// Routed experts of the many-row prompt pass: the pass's (row, expert) pairs are gathered by expert into segments of at most
// TM_SEG rows, so that every chosen expert's weights are streamed and unpacked once per segment whatever rows chose it (a
// 16-row block streams two fifths of a layer's 256 experts for its own sixteen rows).
// Padded row = segment * TM_SEG + position.  Segments 0 .. n_shared - 1 hold all rows in order for the shared expert.
#include <mutex>

#include "prompt.cuh"

namespace dfl {

// One CTA, thread e = expert e.  The rows that chose an expert are one bit each (a row chooses an expert at most once), so a
// pair's rank inside its expert is a count of bits before its row: row order, whatever the timing, and no scan over the pairs.
__global__ void __launch_bounds__(1024) tm_moe_segments_kernel(const TmMoe p) {
    pdl_prologue();
    extern __shared__ uint32_t mask[];   // [expert][words]
    __shared__ int warp_sum[32], first_s[1024];
    const int words = (p.n_rows + 31) / 32, n_pairs = p.n_rows * p.n_used, e = threadIdx.x, lane = e & 31, warp = e >> 5;
    for (int i = e; i < p.n_expert * words; i += 1024) mask[i] = 0u;
    __syncthreads();
    for (int i = e; i < n_pairs; i += 1024) {
        const int x = p.route_idx[i], row = i / p.n_used;
        if (x >= 0) atomicOr(&mask[x * words + (row >> 5)], 1u << (row & 31));
    }
    __syncthreads();
    int cnt = 0;
    if (e < p.n_expert)
        for (int w = 0; w < words; ++w) cnt += __popc(mask[e * words + w]);
    const int n_seg = (cnt + TM_SEG - 1) / TM_SEG;
    int incl = n_seg;   // inclusive prefix sum over the experts
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    int before = 0;
    for (int w = 0; w < warp; ++w) before += warp_sum[w];
    const int first = p.n_shared + before + incl - n_seg;
    first_s[e] = first;
    if (e == 1023) *p.n_seg = before + incl;   // expert segments
    for (int j = 0; j < n_seg; ++j) p.seg[first + j] = make_int2(e, min(TM_SEG, cnt - j * TM_SEG));
    __syncthreads();
    for (int i = e; i < n_pairs; i += 1024) {
        const int x = p.route_idx[i], row = i / p.n_used, j = i % p.n_used;
        int at = -1;   // a row that routes nowhere
        if (x >= 0) {
            const uint32_t* mx = mask + x * words;
            int rank = __popc(mx[row >> 5] & ((1u << (row & 31)) - 1u));
            for (int w = 0; w < (row >> 5); ++w) rank += __popc(mx[w]);
            at = first_s[x] * TM_SEG + rank;
            p.row_of[at] = row;
        }
        p.pos_of[row * (p.n_used + 1) + 1 + j] = at;
    }
    for (int r = e; r < p.n_rows; r += 1024) {   // the shared expert's segments
        p.row_of[r] = r;
        p.pos_of[r * (p.n_used + 1)] = r;
    }
    for (int j = e; j < p.n_shared; j += 1024) p.seg[j] = make_int2(p.n_expert, min(TM_SEG, p.n_rows - j * TM_SEG));
}

// Pack kernels: CTA = 8 padded rows x one 256-column block, threads as in tm_glue_kernel.  MODE 0: the rows' normalised inputs,
// gathered; MODE 1: silu(gate) * up * route weight from the gate | up output.
template <int MODE>
__global__ void __launch_bounds__(256) tm_moe_pack_kernel(const TmMoe p) {
    pdl_prologue();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k8 = warp * 32 + (lane >> 3) * 8, col = blockIdx.x * 256 + k8;
    const int pos = blockIdx.y * 8 + (lane & 7), si = pos / TM_SEG, t = pos % TM_SEG;
    if (si >= p.n_shared + *p.n_seg) return;   // uniform over the CTA
    const int2 seg = p.seg[si];
    if ((int)(blockIdx.y * 8) % TM_SEG >= (seg.y + 7) / 8 * 8) return;
    const bool live = t < seg.y;
    float v[8] = {};
    if (live) {
        const int row = p.row_of[pos];
        if (MODE == 0) {
            const float4* src = reinterpret_cast<const float4*>(p.xn + (uint64_t)row * p.ld_xn + col);
            const float4 a = src[0], b = src[1];
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
            if (blockIdx.x == 0 && k8 == 0) {
                float ss = 0.f;
                for (int q = 0; q < p.n_sumsq; ++q) ss += p.sumsq[(uint64_t)q * p.rows_pad + row];
                p.row_scale[pos] = 1.0f / sqrtf(ss / p.norm_k + 1e-6f);
            }
        } else {
            const float w = seg.x < p.n_expert ? p.route_w[(uint64_t)row * p.n_expert + seg.x] : p.route_sg[row];
            const float* src = p.gu + (uint64_t)pos * 2 * p.f + col;
            const float4 ga = __ldcg(reinterpret_cast<const float4*>(src)), gb = __ldcg(reinterpret_cast<const float4*>(src) + 1);
            const float4 ua = __ldcg(reinterpret_cast<const float4*>(src + p.f)), ub = __ldcg(reinterpret_cast<const float4*>(src + p.f) + 1);
            const float g[8] = {ga.x, ga.y, ga.z, ga.w, gb.x, gb.y, gb.z, gb.w}, u[8] = {ua.x, ua.y, ua.z, ua.w, ub.x, ub.y, ub.z, ub.w};
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = silu_f(g[e]) * u[e] * w * p.pre_scale;
        }
    }
    uint8_t* chunk = (MODE == 0 ? p.acts_in : p.acts_mid) + ((uint64_t)si * gridDim.x + blockIdx.x) * tm_chunk(TM_SEG);
    bool over = false;
    tm_pack_oct(chunk, tm_seg_tok(seg.y), t, k8, v, over);
    float sum = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
    sum += __shfl_xor_sync(0xffffffffu, sum, 8);
    sum += __shfl_xor_sync(0xffffffffu, sum, 16);
    if (lane < 8) tm_pack_sum(chunk, tm_seg_tok(seg.y), t, warp, sum, over);
    if (over) atomicCAS(p.err, 0, DEV_ERR_OVERFLOW);
}

int tm_moe_max_segments(int n_rows, int n_expert, int n_used) {
    const int pairs = n_rows * n_used;
    // an expert with c > 0 rows has at most 1 + (c - 1) / TM_SEG segments
    return (n_rows + TM_SEG - 1) / TM_SEG + (pairs < n_expert ? pairs : n_expert) + pairs / TM_SEG;
}

dfl_status launch_tm_moe_segments(cudaStream_t st, const TmMoe& p) {
    if (p.n_expert > 1024) return fail(DFL_ERR_UNSUPPORTED, "tm_moe: expert count");
    const size_t smem = (size_t)p.n_expert * ((p.n_rows + 31) / 32) * 4;
    if (smem > 64 * 1024) return fail(DFL_ERR_UNSUPPORTED, "tm_moe: experts x rows");
    static std::once_flag once[16];
    int dev = 0;
    DFL_CUDA(cudaGetDevice(&dev));
    cudaError_t attr = cudaSuccess;
    std::call_once(once[dev & 15], [&] { attr = cudaFuncSetAttribute(tm_moe_segments_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024); });
    DFL_CUDA(attr);
    launch_k(tm_moe_segments_kernel, dim3(1), dim3(1024), smem, st, p);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}
dfl_status launch_tm_moe_pack(cudaStream_t st, const TmMoe& p, int mode, uint64_t k) {
    const dim3 grid((unsigned)(k / TILE_K), (unsigned)(p.max_seg * TM_SEG / 8));
    if (mode == 0) launch_k(tm_moe_pack_kernel<0>, grid, dim3(256), 0, st, p);
    else launch_k(tm_moe_pack_kernel<1>, grid, dim3(256), 0, st, p);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

}  // namespace dfl
