// Routed-expert FFN, routing stage (reference: moe.metal:995-1089 kernels, metal_forward/moe.rs:349-751 host,
// CPU oracle forward.rs:749-824; the selection rule followed here is the CPU oracle's).
//
// One warp per token: softmax over all experts, the k experts with the largest probability
// (ties -> lower expert id) found with warp shuffles, weights re-normalised by their own sum
// (floored at 2^-14), written as one dense row route_w[token][expert] with zeros for the experts
// that were not chosen.  The expert GEMMs then run over all experts of the layer as two large
// few-row GEMMs (gate|up with n_out = E * F', down with n_in = E * F'), the SwiGLU glue multiplies
// each expert's inner columns by the token's route weight, so experts that were not chosen
// contribute exact zeros.  The shared expert's sigmoid gate comes from one extra router row.
#include "ops.cuh"

namespace dfl {

// Probabilities live in a warp's registers: 8 a lane up to ROUTE_NARROW experts, 32 beyond: four times the compares and registers of a choice
// (300 rows of 256 experts, routing kernel alone: 6.9 us with 32, 4.7 with 8).
constexpr int MOE_MAX_EXPERTS = 1024, ROUTE_NARROW = 256;

// Routing of one row by one warp, probabilities in registers (PER a lane).  fetch(v, gate): the row's logits lane + 32 k and the shared expert's gate
// logit, every load under way before the first is used;
// mark(expert): called for each expert with a weight.  `real` false: the same instructions on zeros, nothing read or written in global memory.
template <int PER, class Fetch, class Mark>
__device__ __forceinline__ void moe_route_row(int tok, int lane, int n_expert, int n_used, int n_rows, float* route_w, float* shared_gate,
                                              int32_t* route_idx, int* err, bool real, Fetch fetch, Mark mark) {
    float* wrow = route_w + (uint64_t)tok * n_expert;
    float v[PER], gate, mx = -INFINITY;
    if (tok < n_rows) fetch(v, gate);
    if (real)
        for (int i = lane; i < n_expert; i += 32) wrow[i] = 0.f;
    if (tok >= n_rows) {
        if (!real) return;
        if (lane == 0) shared_gate[tok] = 0.f;
        for (int j = lane; j < n_used; j += 32) route_idx[tok * n_used + j] = -1;
        return;
    }
    bool bad = !isfinite(gate);
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        if (lane + 32 * k >= n_expert) continue;
        bad |= !isfinite(v[k]);
        mx = fmaxf(mx, v[k]);
    }
    if (__any_sync(0xffffffffu, bad)) {
        // route status NONFINITE (kernels/moe.metal:355-360): the row routes nowhere and the error word poisons the session
        if (lane == 0) {
            atomicCAS(err, 0, DEV_ERR_NONFINITE);
            shared_gate[tok] = 0.f;
        }
        for (int j = lane; j < n_used; j += 32) route_idx[tok * n_used + j] = -1;
        return;
    }
    mx = warp_max(mx);
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        if (lane + 32 * k >= n_expert) continue;
        v[k] = expf(v[k] - mx);
        sum += v[k];
    }
    sum = warp_sum(sum);
    const float inv = 1.0f / sum;
#pragma unroll
    for (int k = 0; k < PER; ++k) v[k] = lane + 32 * k < n_expert ? v[k] * inv : -2.f;   // below zero: not there, or taken
    float chosen_p = 0.f;   // lane j keeps the j-th choice
    int chosen_i = -1;
    const int picks = real ? n_used : 1;
#pragma unroll 1
    for (int j = 0; j < picks; ++j) {
        float best = -1.f;
        int at = 0;
#pragma unroll
        for (int k = 0; k < PER; ++k)
            if (v[k] > best) { best = v[k]; at = k; }
        // the largest probability, then the lowest expert that has it (probabilities are not negative, so their bits are in order; a lane
        // without one left has the key 0)
        const uint32_t key = best < 0.f ? 0u : __float_as_uint(best) + 1u, top = __reduce_max_sync(0xffffffffu, key);
        const int bi = (int)__reduce_min_sync(0xffffffffu, key == top ? (uint32_t)(lane + 32 * at) : 0x7fffffffu);
        if (lane == (j & 31)) { chosen_p = __uint_as_float(top - 1u); chosen_i = bi; }
#pragma unroll
        for (int k = 0; k < PER; ++k)
            if (lane + 32 * k == bi) v[k] = -2.f;
    }
    // sum of the chosen probabilities in choice order (the oracle's order)
    float wsum = 0.f;
    for (int j = 0; j < picks && j < 32; ++j) wsum += __shfl_sync(0xffffffffu, chosen_p, j);
    wsum = fmaxf(wsum, 6.103515625e-05f);
    const float w = chosen_p / wsum;
    if (lane < picks && chosen_i >= 0) {
        if (real) {
            wrow[chosen_i] = w;
            route_idx[tok * n_used + lane] = chosen_i;
        }
        if (w != 0.f) mark(chosen_i);
    }
    if (real && lane == 0) shared_gate[tok] = sigmoid_f(gate);
}

template <int PER>
__global__ void __launch_bounds__(32) moe_route_kernel(const float* logits, int ld, int n_expert, int n_used, int n_rows,
                                                       float* route_w, float* shared_gate,
                                                       int32_t* route_idx, int* err) {
    pdl_prologue();
    const float* x = logits + (uint64_t)blockIdx.x * ld;
    moe_route_row<PER>(blockIdx.x, threadIdx.x, n_expert, n_used, n_rows, route_w, shared_gate, route_idx, err, true,
                       [&](float(&v)[PER], float& gate) {
                           gate = x[n_expert];
#pragma unroll
                           for (int k = 0; k < PER; ++k)
                               if ((int)threadIdx.x + 32 * k < n_expert) v[k] = x[threadIdx.x + 32 * k];
                       },
                       [](int) {});
}

dfl_status launch_moe_route(cudaStream_t st, const float* logits, int ld, int n_expert, int n_used, int n_rows, float* route_w,
                            float* shared_gate, int32_t* route_idx, int* err) {
    if (n_expert < 1 || n_expert > MOE_MAX_EXPERTS || n_used < 1 || n_used > 32 || n_used > n_expert)
        return fail(DFL_ERR_UNSUPPORTED, "moe_route: expert_count must be in [1, 1024] and expert_used_count in [1, 32]");
    launch_k(n_expert <= ROUTE_NARROW ? moe_route_kernel<ROUTE_NARROW / 32> : moe_route_kernel<MOE_MAX_EXPERTS / 32>, dim3((unsigned)(n_rows > MAX_ROWS ? n_rows : MAX_ROWS)), dim3(32), 0, st, logits, ld, n_expert, n_used, n_rows, route_w, shared_gate, route_idx, err);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

// ---- the row tiles of the gate|up matrix that belong to chosen experts ------------------------------------------------
// The gate|up matrix of a layer is [gate of every local expert | shared gate | up of every local expert | shared up],
// T row tiles per expert and Ts per shared block.  An expert is active when any row of the block routes to it; the
// list holds the tiles of the active experts and of the shared expert, so the GEMM streams only those.  It is padded
// by repetition up to min_tiles (a repeated tile is computed twice with the same result), which keeps every CTA of the
// fixed launch geometry busy with at least one tile.
struct MoeListArgs {
    int n_expert, e0, n_local, T, Ts, min_tiles;
    int32_t *tile_map, *n_tiles;
    int KB, min_kb;
    int32_t *kb_map, *n_kb;
    int kc, down_tiles, max_splits, n_sm;
};
// active: this thread's local expert (thread = expert).  `real` false: nothing written to global memory.
__device__ __forceinline__ void moe_build_lists(bool active, const MoeListArgs a, bool real) {
    const int n_local = a.n_local, T = a.T, Ts = a.Ts, min_tiles = a.min_tiles, KB = a.KB, min_kb = a.min_kb;
    const int kc = a.kc, down_tiles = a.down_tiles, max_splits = a.max_splits, n_sm = a.n_sm;
    int32_t *tile_map = a.tile_map, *n_tiles = a.n_tiles, *kb_map = a.kb_map, *n_kb = a.n_kb;
    __shared__ int warp_count[MOE_MAX_EXPERTS / 32];
    __shared__ int total_sh;
    const int e = threadIdx.x, warp = e >> 5, lane = e & 31;
    const uint32_t bal = __ballot_sync(0xffffffffu, active);
    if (lane == 0) warp_count[warp] = __popc(bal);
    __syncthreads();
    if (warp == 0) {   // counts -> ranks of the warps' first experts
        const int own = warp_count[lane];
        int run = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int below = __shfl_up_sync(0xffffffffu, run, o);
            if (lane >= o) run += below;
        }
        warp_count[lane] = run - own;
        if (lane == 31) total_sh = run;
    }
    __syncthreads();
    const int n_act = total_sh, rank = warp_count[warp] + __popc(bal & ((1u << lane) - 1u));
    const int up_base = n_local * T + Ts, up_list = n_act * T + Ts, n = 2 * up_list;
    if (active && real)
        for (int j = 0; j < T; ++j) {
            tile_map[rank * T + j] = e * T + j;
            tile_map[up_list + rank * T + j] = up_base + e * T + j;
        }
    if (e < Ts && real) {
        tile_map[n_act * T + e] = n_local * T + e;
        tile_map[up_list + n_act * T + e] = up_base + n_local * T + e;
    }
    __syncthreads();
    for (int i = n + e; i < min_tiles && real; i += MOE_MAX_EXPERTS) tile_map[i] = n > 0 ? tile_map[i % n] : i;
    if (e == 0 && real) *n_tiles = n > min_tiles ? n : min_tiles;
    // column blocks of the down matrix (KB per expert): the active experts' blocks first, then the others, whose
    // activations are zero - the list is cut after the active ones, but never below min_kb entries
    if (kb_map && e < n_local && real) {
        const int pos = active ? rank : n_act + (e - rank);
        for (int j = 0; j < KB; ++j) kb_map[pos * KB + j] = e * KB + j;
    }
    if (kb_map && e == 0) {
        const int want = n_act * KB, all = n_local * KB;
        const int len = want > min_kb ? want : (min_kb < all ? min_kb : all);
        // split geometry for this list length: enough splits to keep a CTA's blocks resident and to give every SM
        // work, as many CTAs per split as fit beside them; 0 = the launch's own geometry
        int s = 0, cps = 0;
        if (max_splits > 0) {
            s = (len + kc - 1) / kc;
            const int fill = (n_sm + down_tiles - 1) / down_tiles;
            if (s < fill) s = fill;
            if (s > max_splits) s = max_splits;
            if (s > len) s = len;
            cps = n_sm / s < down_tiles ? n_sm / s : down_tiles;
        }
        if (real) {
            n_kb[0] = len;
            n_kb[1] = s;
            n_kb[2] = cps;
        }
    }
}

// Routing of the block's rows (warps 0-15, one row each) and the lists in one launch.  One CTA with little to do, so what it took was
// latency, and most of that its code coming from far away (the GEMMs between two launches stream everything else out of L2): it runs through
// itself once before the dependency wait, which it reaches 10 us early, without writing anything.  Choices by warp reductions instead of
// five exchanges, the chosen experts passed on in shared memory: a link of the chain 11.2 -> 6.9 us
// (the logits into shared memory 1.2 us, softmax and choice 2.7, lists 1.5).
template <int PER>
__global__ void __launch_bounds__(MOE_MAX_EXPERTS) moe_route_lists_kernel(const RouterLogits x, int n_used, int n_rows, float* route_w,
                                                                          float* shared_gate, int32_t* route_idx, int* err, const MoeListArgs a) {
    extern __shared__ __align__(16) float logits[];   // [16][n_expert + 1]
    __shared__ float scale[MAX_ROWS];
    __shared__ bool chosen[MOE_MAX_EXPERTS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, e = threadIdx.x, n_col = a.n_expert + 1;
    pdl_launch_dependents();
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
        const bool real = pass;
        if (real) pdl_wait();
        // the slices of all rows (sixteen rows of any length are whole 16-byte pieces), a thread's loads under way together; the rows' scales by
        // warps 16 - 31
        const int n4 = MAX_ROWS * n_col / 4;
        float ss = 0.f;
        if (warp >= MAX_ROWS)
            for (int i = lane; i < x.n_sumsq; i += 32) ss += real ? __ldcg(x.sumsq + i * MAX_ROWS + warp - MAX_ROWS) : 1.f;
#pragma unroll 1
        for (int i = e; i < n4; i += MOE_MAX_EXPERTS) {
            float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
            for (int s = 0; s < x.slices; ++s) {
                if (!real) continue;
                const float4 v = __ldcg(reinterpret_cast<const float4*>(x.part) + (uint64_t)s * n4 + i);
                t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w;
            }
            reinterpret_cast<float4*>(logits)[i] = t;
        }
        if (warp >= MAX_ROWS) {
            ss = warp_sum(ss);
            if (lane == 0) scale[warp - MAX_ROWS] = 1.0f / sqrtf(ss / x.norm_k + x.eps);
        }
        chosen[e] = false;
        __syncthreads();
        if (warp < MAX_ROWS)
            moe_route_row<PER>(warp, lane, a.n_expert, n_used, n_rows, route_w, shared_gate, route_idx, err, real,
                               [&](float(&v)[PER], float& gate) {
                                   const float* row = logits + warp * n_col;
                                   const float f = scale[warp];
                                   gate = row[a.n_expert] * f;
#pragma unroll
                                   for (int k = 0; k < PER; ++k)
                                       if (lane + 32 * k < a.n_expert) v[k] = row[lane + 32 * k] * f;
                               },
                               [&](int i) { chosen[i] = true; });
        __syncthreads();
        moe_build_lists(e < a.n_local && chosen[a.e0 + e], a, real);
        __syncthreads();
    }
}

static MoeListArgs moe_list_args(int n_expert, int e0, int n_local, int tiles_per_expert, int shared_tiles, int min_tiles, int32_t* tile_map,
                                 int32_t* n_tiles, int kb_per_expert, int min_kb, int32_t* kb_map, int32_t* n_kb, int kc, int down_tiles,
                                 int max_splits) {
    return MoeListArgs{n_expert, e0, n_local, tiles_per_expert, shared_tiles, min_tiles, tile_map, n_tiles, kb_per_expert, min_kb, kb_map, n_kb,
                       kc, down_tiles, max_splits, sm_count()};
}

dfl_status launch_moe_route_lists(cudaStream_t st, const RouterLogits& x, int n_expert, int n_used, int n_rows, float* route_w,
                                  float* shared_gate, int32_t* route_idx, int e0, int n_local, int tiles_per_expert, int shared_tiles,
                                  int min_tiles, int32_t* tile_map, int32_t* n_tiles, int kb_per_expert, int min_kb, int32_t* kb_map,
                                  int32_t* n_kb, int kc, int down_tiles, int max_splits, int* err) {
    if (n_expert < 1 || n_expert > MOE_MAX_EXPERTS || n_used < 1 || n_used > 32 || n_used > n_expert || n_local > MOE_MAX_EXPERTS ||
        shared_tiles > MOE_MAX_EXPERTS)
        return fail(DFL_ERR_UNSUPPORTED, "moe_route_lists: geometry");
    auto* kernel = n_expert <= ROUTE_NARROW ? moe_route_lists_kernel<ROUTE_NARROW / 32> : moe_route_lists_kernel<MOE_MAX_EXPERTS / 32>;
    const size_t smem = (size_t)MAX_ROWS * (n_expert + 1) * 4;
    if (smem > 40 * 1024) DFL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    launch_k(kernel, dim3(1), dim3(MOE_MAX_EXPERTS), smem, st, x, n_used, n_rows, route_w, shared_gate, route_idx, err,
              moe_list_args(n_expert, e0, n_local, tiles_per_expert, shared_tiles, min_tiles, tile_map, n_tiles, kb_per_expert, min_kb, kb_map, n_kb,
                            kc, down_tiles, max_splits));
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

}  // namespace dfl
