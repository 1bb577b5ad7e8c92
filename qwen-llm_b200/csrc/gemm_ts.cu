// Few-row weight-streaming GEMM on the fifth-generation tensor cores.
//
// Same contract as the mma.sync kernel (gemm_fewrow.cu: y[r, o] = sum_i x[r, i] W[o, i], <= 16
// activation rows, split-K partials, deterministic), different engine.  One CTA per SM, four
// kinds of warps that only meet at mbarriers:
//   * a producer thread streams 128-row x 256-column stages of packed weights with bulk copies
//     into a shared-memory ring; the packed activations of the CTA's column range are copied
//     once and stay resident as the B operand;
//   * eight unpacking warps in two groups turn the integer quants into exact f16 integers q * sc (the
//     6-bit sub-block scale folded in, still exact: q * sc < 2048) and store them with
//     tcgen05.st into tensor memory, thread = weight row = TMEM lane.
//     They do nothing else, so their instruction stream never waits for an accumulator;
//   * four warps, one per scheduler, issue tcgen05.mma (A from tensor memory, B = activations
//     hi / lo planes from shared memory, M = 128, N = 32, K = 16 per instruction), sixteen per
//     256-column block, accumulating it in tensor memory; a seventeenth MMA multiplies the
//     sub-block mins with the per-sub-block activation sums (the K-quant "min" term);
//   * four draining warps (thread = weight row) read the finished block's accumulator back
//     (tcgen05.ld), apply the per-row f16 super-block scales d and dmin in f32 and add to
//     sixteen register accumulators (one per token); at the end of a row tile they write the
//     partial result straight to global memory.  No shared-memory reduction, no atomics.
// The A operand and the accumulators are double-buffered in tensor memory: unpacking pass
// i + 1 overlaps the MMAs of pass i, which overlap the read-back of block i - 1.
#include <mutex>

#include "ops.cuh"
#include "tcgen05_prims.cuh"

namespace dfl {

// Q6_K packing lives in gemm_ts_q6k.cuh (included further down, after the primitives it uses)
__device__ __forceinline__ uint64_t src_block_index(uint64_t row, int kb, int kblocks, uint64_t n_out, int kb_group);
__global__ void retile_ts_q6k_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, uint64_t n_out, int kblocks, int kb_group);
__device__ float decode_ts_q6k_elem(const uint8_t* stage, int r, int k);
__global__ void retile_ts_q80_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, uint64_t n_out, int kblocks, int kb_group);
__device__ float decode_ts_q80_elem(const uint8_t* stage, int r, int k);
__global__ void q80_scale_range_kernel(const uint8_t* __restrict__ src, uint64_t n_blocks, int* flag);
__global__ void retile_tsb_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, uint64_t n_in, uint64_t n_out, int kblocks);
__device__ float decode_tsb_elem(const uint8_t* stage, int r, int k);

// ---------------------------------------------------------------------------------------------
// Re-tiling into row-lane tiles and the inverse decode.
// ---------------------------------------------------------------------------------------------
// Index of the ggml block (row, kb) in the source.  kb_group = 0: plain row-major [n_out][kblocks].  kb_group > 0: the
// source is [kblocks / kb_group] matrices of [n_out][kb_group] blocks one after the other (the experts of
// ffn_down_exps), viewed as one matrix whose columns are the experts' columns side by side.
__device__ __forceinline__ uint64_t src_block_index(uint64_t row, int kb, int kblocks, uint64_t n_out, int kb_group) {
    if (kb_group <= 0) return row * kblocks + kb;
    return ((uint64_t)(kb / kb_group) * n_out + row) * kb_group + kb % kb_group;
}

template <int DT>
__global__ void retile_ts_kernel(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, uint64_t n_out, int kblocks, int kb_group) {
    static_assert(DT == DFL_Q4_K || DT == DFL_Q5_K, "Q6_K and Q8_0 have packers of their own");
    constexpr int SRC_BLK = DT == DFL_Q4_K ? 144 : 176;
    constexpr int STAGE = DT == DFL_Q4_K ? STAGE_Q4_K_TS : STAGE_Q5_K_TS;
    const uint64_t tile_id = blockIdx.x;
    const int kb = (int)(tile_id % kblocks);
    const uint64_t rt = tile_id / kblocks;
    uint8_t* stage = dst + tile_id * STAGE;
    // one item = 16 destination bytes
    for (int idx = threadIdx.x; idx < STAGE / 16; idx += blockDim.x) {
        uint8_t out[16];
#pragma unroll
        for (int b = 0; b < 16; ++b) out[b] = 0;
        const int off = idx * 16;
        const int qs_src = DT == DFL_Q4_K ? 16 : 48;
        auto block_of = [&](int r) -> const uint8_t* {   // null beyond the matrix
            const uint64_t row = rt * TILE_R + r;
            return row < n_out ? src + src_block_index(row, kb, kblocks, n_out, kb_group) * (uint64_t)SRC_BLK : nullptr;
        };
        if (off < TSQ4_OFF_QS) {   // four rows' d, dmin or four rows' scale bytes
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const bool scales = off >= TSQ4_OFF_SC;
                const int w = (off - (scales ? TSQ4_OFF_SC : 0)) / 4 + x, r = w & 127, kp = w >> 7;
                const uint8_t* blk = block_of(r);
                if (!blk) continue;
                if (!scales) {
                    for (int b = 0; b < 4; ++b) out[4 * x + b] = blk[b];
                } else {
                    for (int b = 0; b < 2; ++b) {
                        uint32_t sc, m;
                        k4_scale_min(blk + 4, 2 * kp + b, sc, m);
                        out[4 * x + 2 * b] = (uint8_t)sc;
                        out[4 * x + 2 * b + 1] = (uint8_t)m;
                    }
                }
            }
        } else {
            int r, src_off;
            if (off < TSQ4_OFF_QS + 16384) {                                                  // qs [kp][half][row]
                const int i = idx - TSQ4_OFF_QS / 16;
                r = i & 127;
                src_off = qs_src + 32 * (i >> 8) + 16 * ((i >> 7) & 1);
            } else {                                                                          // Q5_K qh [half][row]
                const int i = idx - TSQ5_OFF_QH / 16;
                r = i & 127;
                src_off = 16 + 16 * (i >> 7);
            }
            if (const uint8_t* blk = block_of(r)) {
#pragma unroll
                for (int b = 0; b < 16; ++b) out[b] = blk[src_off + b];
            }
        }
        *reinterpret_cast<uint4*>(stage + off) = *reinterpret_cast<const uint4*>(out);
    }
}

dfl_status retile_matrix_ts(cudaStream_t st, int dtype, const uint8_t* ggml_dev, uint64_t n_in, uint64_t n_out, uint8_t* dst_tiles,
                            int kb_group) {
    if (n_in % TILE_K) return fail(DFL_ERR_BAD_SHAPE, "retile: n_in must be a multiple of 256");
    const int kblocks = (int)(n_in / TILE_K);
    const uint64_t n_tiles = (uint64_t)kblocks * ((n_out + TILE_R - 1) / TILE_R);
    if (n_tiles == 0 || n_tiles > 0x7fffffffu) return fail(DFL_ERR_BAD_SHAPE, "retile: tile count out of range");
    dim3 grid((unsigned)n_tiles), block(256);
    switch (dtype) {
        case DFL_Q4_K: retile_ts_kernel<DFL_Q4_K><<<grid, block, 0, st>>>(ggml_dev, dst_tiles, n_out, kblocks, kb_group); break;
        case DFL_Q5_K: retile_ts_kernel<DFL_Q5_K><<<grid, block, 0, st>>>(ggml_dev, dst_tiles, n_out, kblocks, kb_group); break;
        case DFL_Q6_K: retile_ts_q6k_kernel<<<grid, block, 0, st>>>(ggml_dev, dst_tiles, n_out, kblocks, kb_group); break;
        case DFL_Q8_0: retile_ts_q80_kernel<<<grid, block, 0, st>>>(ggml_dev, dst_tiles, n_out, kblocks, kb_group); break;
        case DFL_BF16:
            if (kb_group > 0) return fail(DFL_ERR_UNSUPPORTED, "retile: grouped column blocks are not built for bf16");
            retile_tsb_kernel<<<grid, block, 0, st>>>(ggml_dev, dst_tiles, n_in, n_out, kblocks);
            break;
        default: return fail(DFL_ERR_UNSUPPORTED, "retile: dtype has no row-lane tile layout");
    }
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

__global__ void decode_tiles_ts_kernel(const uint8_t* __restrict__ tiles, int dtype, uint64_t n_in, uint64_t n_out, int kblocks,
                                       float* __restrict__ out) {
    const uint64_t idx = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= n_in * n_out) return;
    const uint64_t row = idx / n_in;
    const int kk = (int)(idx % n_in);
    const int kb = kk >> 8, k = kk & 255;
    const uint64_t rt = row / TILE_R;
    const int r = (int)(row % TILE_R);
    const uint8_t* stage = tiles + (rt * kblocks + kb) * (uint64_t)stage_bytes_of(dtype, LAYOUT_TS);
    float v = 0.f;
    if (dtype == DFL_Q4_K || dtype == DFL_Q5_K) {
        const uint8_t* h = stage + r * 4;
        const float d = __half2float(__ushort_as_half((unsigned short)(h[0] | (h[1] << 8))));
        const float dmin = __half2float(__ushort_as_half((unsigned short)(h[2] | (h[3] << 8))));
        const uint8_t* pr = stage + TSQ4_OFF_SC + ((k >> 6) * 128 + r) * 4 + 2 * ((k >> 5) & 1);
        const uint32_t sc = pr[0], m = pr[1];
        const int kp = k >> 6, hi = (k >> 5) & 1, l = k & 31;
        const uint8_t byte = stage[TSQ4_OFF_QS + ((kp * 2 + (l >> 4)) * 128 + r) * 16 + (l & 15)];
        uint32_t q = hi ? (byte >> 4) : (byte & 15);
        if (dtype == DFL_Q5_K) q |= ((stage[TSQ5_OFF_QH + ((l >> 4) * 128 + r) * 16 + (l & 15)] >> (2 * kp + hi)) & 1u) << 4;
        v = __fsub_rn(__fmul_rn(d * (float)sc, (float)q), dmin * (float)m);
    } else if (dtype == DFL_Q6_K) {
        v = decode_ts_q6k_elem(stage, r, k);
    } else if (dtype == DFL_Q8_0) {
        v = decode_ts_q80_elem(stage, r, k);
    } else if (dtype == DFL_BF16) {
        v = decode_tsb_elem(stage, r, k);
    }
    out[idx] = v;
}

// Whether every block scale of a Q8_0 matrix (ggml bytes on the device) leaves q * d inside the f16 range.
dfl_status q80_scales_fit_ts(cudaStream_t st, const uint8_t* ggml_dev, uint64_t n_in, uint64_t n_out, bool* fits) {
    int* flag = nullptr;
    DFL_CUDA(device_malloc(&flag, sizeof(int)));
    cudaMemsetAsync(flag, 0, sizeof(int), st);
    const uint64_t n_blocks = n_in / 32 * n_out;
    q80_scale_range_kernel<<<(unsigned)((n_blocks + 255) / 256), 256, 0, st>>>(ggml_dev, n_blocks, flag);
    count_launch();
    int h = 1;
    cudaError_t e = cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(flag);
    if (e != cudaSuccess) return fail(DFL_ERR_CUDA, std::string("q80 scale range: ") + cudaGetErrorString(e));
    *fits = h == 0;
    return DFL_OK;
}

dfl_status decode_tiles_ts(cudaStream_t st, const QMatrix& m, float* out_dev) {
    const uint64_t n = m.n_in * m.n_out;
    decode_tiles_ts_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(m.tiles, m.dtype, m.n_in, m.n_out, m.kblocks, out_dev);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

// ---------------------------------------------------------------------------------------------
// Standalone activation packing (the model path packs inside its glue kernels).
// One CTA per 256-column block; thread = (token = tid / 16, 16 consecutive columns).
// ---------------------------------------------------------------------------------------------
__global__ void prep_acts_ts_kernel(const float* __restrict__ x, int ld, int n_rows, float pre_scale, uint8_t* __restrict__ acts,
                                    int* err) {
    const int kb = blockIdx.x, tok = threadIdx.x >> 4, seg = threadIdx.x & 15;
    uint8_t* chunk = acts + (uint64_t)kb * ACTTS_CHUNK;
    // the zero half of the small operand (sub-block index 8..15)
    for (int i = threadIdx.x; i < 768 / 4; i += blockDim.x) reinterpret_cast<uint32_t*>(chunk + TS_BMIN_OFF + 768)[i] = 0u;
    float v[16];
    if (tok < n_rows) {
        const float4* src = reinterpret_cast<const float4*>(x + (uint64_t)tok * ld + (uint64_t)kb * TILE_K + seg * 16);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 q = src[j];
            v[4 * j] = q.x * pre_scale; v[4 * j + 1] = q.y * pre_scale; v[4 * j + 2] = q.z * pre_scale; v[4 * j + 3] = q.w * pre_scale;
        }
    } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = 0.f;
    }
    bool over = false;
    float sum = 0.f;
#pragma unroll
    for (int q4 = 0; q4 < 4; ++q4) {
        const float quad[4] = {v[4 * q4], v[4 * q4 + 1], v[4 * q4 + 2], v[4 * q4 + 3]};
        pack_quad_ts(chunk, tok, seg * 16 + 4 * q4, quad, over);
        sum += (quad[0] + quad[1]) + (quad[2] + quad[3]);
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);  // 32-column sub-block = this thread and its neighbour
    if ((seg & 1) == 0) pack_subsum_ts(chunk, tok, seg >> 1, sum, over);
    if (over) atomicCAS(err, 0, DEV_ERR_OVERFLOW);
}

dfl_status launch_prep_acts_ts(cudaStream_t st, const float* x, int ld, int n_rows, uint64_t k, float pre_scale, uint8_t* acts,
                               int* dev_err) {
    if (k % TILE_K || n_rows < 0 || n_rows > MAX_ROWS) return fail(DFL_ERR_BAD_SHAPE, "prep_acts: shape");
    prep_acts_ts_kernel<<<(unsigned)(k / TILE_K), 256, 0, st>>>(x, ld, n_rows, pre_scale, acts, dev_err);
    count_launch();
    DFL_CUDA(cudaGetLastError());
    return DFL_OK;
}

// ---------------------------------------------------------------------------------------------
// tcgen05 / tensor-memory primitives (sm_100a).
// ---------------------------------------------------------------------------------------------
namespace ts {

constexpr int KC_MAX = 6;                               // column blocks whose activations stay resident, at most

// tensor-memory columns (32-bit each, 128 lanes), everything once per group: a 128-column A buffer (256 f16 per row)
// written and consumed in two halves, two 32-column accumulators (even / odd MMA steps), the 8-column A operand of the
// min term and its 48-column accumulator
constexpr uint32_t TM_A = 0, TM_A_STRIDE = 128, TM_D = 256, TM_D_STRIDE = 64, TM_AM = 384, TM_AM_STRIDE = 8, TM_DM = 400, TM_DM_STRIDE = 48,
                   TM_COLS = 512;
static_assert(TM_DM + 2 * TM_DM_STRIDE <= TM_COLS, "tensor memory budget");

__device__ __forceinline__ uint32_t h2sub(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("sub.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t h2mul(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t h2fma(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
// (a & mask) | bits in one instruction: written with operators, half of the unpack's selections came out as two
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t mask, uint32_t bits) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xea;" : "=r"(r) : "r"(a), "r"(mask), "r"(bits));
    return r;
}
constexpr uint32_t MAGIC = 0x64006400u;      // half2(1024, 1024): 1024 + small integer in the mantissa
constexpr uint32_t H2_NEG1024 = 0xe400e400u; // half2(-1024)
constexpr uint32_t H2_16TH = 0x2c002c00u;    // half2(1/16)
constexpr uint32_t H2_NEG64 = 0xd400d400u;   // half2(-64)
struct UnitScales {
    float d, dmin;
};

template <int DT>
struct Fmt;

// Q4_K / Q5_K: two halves per stage.  In half h thread (row, kp2) takes the 64 columns of quarter kp = 2h + kp2:
// sub-blocks 2kp (low nibbles) and 2kp + 1 (high nibbles) of its row into r[0..15] / r[16..31]; r[c] = half2 of
// k-positions 2c, 2c + 1.
template <int DT>
struct FmtK45 {
    static constexpr int STAGE = DT == DFL_Q4_K ? STAGE_Q4_K_TS : STAGE_Q5_K_TS;
    __host__ __device__ static constexpr int stages(int) { return DT == DFL_Q4_K ? 6 : 5; }   // ring slots beside kc resident column blocks
    static constexpr int HALVES = 2;
    static constexpr bool HAS_MIN = true;
    // MMA step jj (0..7) of half h multiplies A-buffer columns a_col .. + 8 with 16-column slice b_slice of the block
    __device__ static __forceinline__ uint32_t a_col(int h, int jj) { return (uint32_t)(64 * h + 8 * jj); }
    __device__ static __forceinline__ uint32_t b_slice(int h, int jj) { return (uint32_t)(8 * h + jj); }
    __device__ static __forceinline__ void store(uint32_t buf, int h, int kp2, const uint32_t (&r)[32]) { tmem_st32(buf + 64 * h + 32 * kp2, r); }
    __device__ static __forceinline__ void unpack(const uint8_t* st, int ps, int row, int kp2, uint32_t (&r)[32], uint32_t& am,
                                                  UnitScales& us) {
        const int kp = 2 * ps + kp2;
        const uint32_t dd = reinterpret_cast<const uint32_t*>(st)[row];
        const uint32_t t = reinterpret_cast<const uint32_t*>(st + TSQ4_OFF_SC)[kp * 128 + row];   // sc0, m0, sc1, m1
        const uint4* qs = reinterpret_cast<const uint4*>(st + TSQ4_OFF_QS);
        const uint4 qa = qs[(kp * 2 + 0) * 128 + row], qb = qs[(kp * 2 + 1) * 128 + row];
        us.d = __half2float(__ushort_as_half((unsigned short)(dd & 0xffffu)));
        us.dmin = __half2float(__ushort_as_half((unsigned short)(dd >> 16)));
        // bytes under the exponent byte of 1024, minus 1024: half2(sc0, sc0), half2(sc1, sc1), half2(m0, m1)
        const uint32_t s0 = h2sub(__byte_perm(t, 0x64646464u, 0x4040), MAGIC), s1 = h2sub(__byte_perm(t, 0x64646464u, 0x4242), MAGIC);
        const uint32_t cml = s0, cal = h2mul(s0, H2_NEG1024);                      // (1024 + q) * sc - 1024 sc
        const uint32_t cmh = h2mul(s1, H2_16TH), cah = h2mul(s1, H2_NEG64);        // (1024 + 16 q) * sc / 16 - 64 sc
        const uint32_t w[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
        if (DT == DFL_Q4_K) {
#pragma unroll
            for (int wi = 0; wi < 8; ++wi) {
                const uint32_t v = w[wi], v8 = v >> 8;
                r[2 * wi] = h2fma(and_or(v, 0x000f000fu, MAGIC), cml, cal);
                r[2 * wi + 1] = h2fma(and_or(v8, 0x000f000fu, MAGIC), cml, cal);
                r[16 + 2 * wi] = h2fma(and_or(v, 0x00f000f0u, MAGIC), cmh, cah);
                r[16 + 2 * wi + 1] = h2fma(and_or(v8, 0x00f000f0u, MAGIC), cmh, cah);
            }
        } else {
            const uint4* qh = reinterpret_cast<const uint4*>(st + TSQ5_OFF_QH);
            const uint4 ha = qh[row], hb = qh[128 + row];
            const uint32_t hw[8] = {ha.x, ha.y, ha.z, ha.w, hb.x, hb.y, hb.z, hb.w};
#pragma unroll
            for (int wi = 0; wi < 8; ++wi) {
                const uint32_t v = w[wi], v8 = v >> 8, t = hw[wi] >> (2 * kp);
                r[2 * wi] = h2fma(and_or(t << 4, 0x00100010u, and_or(v, 0x000f000fu, MAGIC)), cml, cal);
                r[2 * wi + 1] = h2fma(and_or(t >> 4, 0x00100010u, and_or(v8, 0x000f000fu, MAGIC)), cml, cal);
                r[16 + 2 * wi] = h2fma(and_or(t << 7, 0x01000100u, and_or(v, 0x00f000f0u, MAGIC)), cmh, cah);
                r[16 + 2 * wi + 1] = h2fma(and_or(t >> 1, 0x01000100u, and_or(v8, 0x00f000f0u, MAGIC)), cmh, cah);
            }
        }
        // column kp of the min-term A operand: the mins of this thread's two sub-blocks
        am = h2sub(__byte_perm(t, 0x64646464u, 0x4341), MAGIC);
    }
};
template <>
struct Fmt<DFL_Q4_K> : FmtK45<DFL_Q4_K> {};
template <>
struct Fmt<DFL_Q5_K> : FmtK45<DFL_Q5_K> {};

}  // namespace ts

}  // namespace dfl

#include "gemm_ts_q6k.cuh"
#include "gemm_ts_q80.cuh"
#include "gemm_tsb.cuh"
#include "gemm_ts_kernel.cuh"
#include "gemm_tm.cuh"
