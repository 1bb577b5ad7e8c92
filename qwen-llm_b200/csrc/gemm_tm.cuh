// Many-row GEMM over the resident K-quant tiles (prompt passes: 17 rows and more); included by gemm_ts.cu only.
//
// Same weights, same precision as the few-row kernel: weights stay the integers q * sc (exact in f16), activations are f16
// hi + lo, products are summed in f32 and the super-block scale d is applied in f32.
// What changes is the ratio: one unpacked 128 x 256 weight tile is multiplied with up to 128 tokens instead of 16, so that the
// tensor pipe, not the unpack, is what a CTA spends its time on.  Per 256-column block (1 CTA per SM):
//   * MMA: 16 k-steps x {hi, lo} of M 128 N 128 K 16 (64 clocks each) = 2048 clocks, plus two for the K-quant min term;
//     Q6_K: q * sc needs up to 13 bits, A1 = fl16(q * sc) and A2 = q * sc - A1 in {-1, 0, 1}; A1 x {hi, lo} + A2 x hi
//     (A2 x lo is below 2^-24 of the product's range) = 3072 clocks;
//   * unpack: 16 warps, about 1000 - 1300 clocks of issue, hidden under the MMAs;
//   * activations: 1 KiB of hi / lo planes per token, block and CTA from L2.
// An item takes 2500 - 4000 clocks more to end and to start; with few tokens, the latencies of the rings (1600 - 2000 clocks
// a block) are what is left.
// Precision: a step of a tensor-core sum drops what lies below the last place of the running sum, whatever it adds, so the error
// grows with the steps that an accumulator takes at its full size.  A block is summed in two halves of 128 columns that are read back and
// added in f32 one after the other, and in a half the small products (weights times the lo plane, A2 times the hi plane) come first:
// eight steps count, as in the few-row kernel, where one accumulator of 34 left captured rows four layers deep 3.4 times further from the
// float64 result (1.56e-5 against 4.5e-6; now 4.3e-6).  The halves cost 11 % of a prompt's time as long as the running
// sums lay in tensor memory, since every half had to read and write them too; they are registers of the read-back warps now.
// The min term -dmin * m_j * sum(x over sub-block j) rides in the second half: its A operand is -(dmin / s) m_j as
// an f16 hi + lo pair, s = the factor the accumulator is multiplied with afterwards (d, except where dmin / d would leave
// the f16 range), its B operand the sub-block sums as f16 hi + lo.
//
// Warps: 0..15 unpack (two groups of eight; group g owns A buffer g: Q4_K / Q5_K half g of a block, Q6_K quarters g and
// g + 2), 16..23 read the accumulator back (thread = weight row and half of the
// tokens), 24 and 25 issue the MMAs of even and odd blocks, 26 streams weights, 27 activations.  Two issuers, because one
// spends 2400 - 3000 clocks on a block's MMAs, waits and commits whatever the tokens, more than the tensor pipe needs (161 us
// for 4096 -> 24576 Q4_K over 512 rows with one, 41 us over 77).  Barriers that both would wait on exist once for each, so
// that neither ever waits for a barrier phase whose predecessor it has not seen.
// Tensor memory, for a capacity of C tokens: ND accumulators of C columns, taken by the halves in turn (one fills while another is read
// back), and the A buffers of 64 columns.  At 128 tokens that leaves one A buffer a group, whose refill (store,
// wait, two signals: 900 clocks) only the other group's MMAs cover (two, with fewer weight stages, were 1 % slower); tiles of up to 80
// tokens have two, so that what is left of a block is mostly the unpack.
#pragma once

namespace dfl {
namespace ts {

constexpr int TM_WARPS = 28, TM_THREADS = TM_WARPS * 32;
constexpr int TM_GROUP_WARPS = 8, TM_UNPACK_WARPS = 2 * TM_GROUP_WARPS;   // thread = (row = 32 * (warp % 4) + lane, kp2 = (warp / 4) % 2)
constexpr int TM_DRAIN_WARP0 = 16, TM_DRAIN_WARPS = 8, TM_MMA_WARP = 24, TM_W_WARP = 26, TM_B_WARP = 27;   // two MMA warps
constexpr int TM_BAR_BYTES = 512;
// Registers a thread: what the launch gives, and the share of the unpacking and the read-back warps, which hold up to 64 running sums each.
constexpr int TM_REGS = 72, TM_REGS_UNPACK = 56, TM_REGS_DRAIN = 104;
static_assert(TM_THREADS * TM_REGS == 16 * 32 * TM_REGS_UNPACK + TM_DRAIN_WARPS * 32 * TM_REGS_DRAIN + 4 * 32 * TM_REGS, "no more than the launch has");

struct TmParams {
    const uint8_t* w;
    const uint8_t* acts;      // [token tile][column block] chunks of tm_chunk(tokens) bytes
    float* out;               // [splits][rows_pad][ld_out]
    const float* sumsq;       // [n_sumsq][rows_pad]
    int n_sumsq;
    float norm_k, eps, out_scale;
    int kblocks, splits, row_tiles, tok_tiles, tile_tok, n_rows, rows_pad;   // tile_tok: tokens per tile, a multiple of 16 up to 128
    uint32_t n_out, ld_out;
    int* err;
    TmSegments g;             // g.seg != nullptr: segments of gathered rows instead of token tiles
};

constexpr int TM_SMALL = 80;   // the most tokens that leave tensor memory for three accumulators and two A buffers a group: 3 * 80 + 4 * 64 <= 512 columns

template <int DT, int CAP>
struct TmFmt {
    static constexpr int NA = CAP <= TM_SMALL ? 2 : 1;   // A buffers a group
    static constexpr int ND = CAP == TM_TOK ? 2 : CAP == TM_SMALL ? 3 : 4;   // accumulators, a half block each in turn
    static constexpr uint32_t A = ND * CAP;
    static_assert(ND * CAP + NA * 128 <= 512, "tensor memory");
    // Activation stages (64 columns).  A slot is filled again 1400 - 1600 clocks after its MMAs (commit, producer, copy), so a ring of
    // one block bounds a block at some 2000 clocks however few tokens there are: as many as fit.
    static constexpr int NB = CAP == TM_TOK ? 4 : CAP == TM_SMALL ? 6 : 8;
    static constexpr int N_AM = NA == 2 ? 4 : 3;
    static constexpr bool MIN = DT != DFL_Q6_K;
    static constexpr int W_STAGE = Fmt<DT>::STAGE;
    static constexpr int BSTAGE = tm_bstage(CAP), SUMS = tm_sums(CAP);
    // weight stages: what the activation ring leaves room for
    static constexpr int W_STAGES = CAP == TM_TOK ? (DT == DFL_Q6_K ? 2 : 3) : CAP == TM_SMALL ? (DT == DFL_Q4_K ? 4 : 3) : (DT == DFL_Q6_K ? 4 : 6);
    static constexpr int USES = MIN ? 1 : 2;      // how often a block uses each A buffer
    // Activation stages of a ring slot: half a block where tiles are small, so that the issuers wait and commit less often; one where a slot's
    // refill must not have to wait for the other stage of the half.
    static constexpr int SQ = CAP == TM_TOK ? 1 : 2, NS = NB / SQ;
    static constexpr int OFF_W = NB * BSTAGE;
    // [N_AM] min-term A operand, 128 x 16.  The first group writes block e's after the first half of block e - NA has completed,
    // which is behind the issuer's block before it, e - NA - 2, but says nothing of the last MMAs of block e - NA.
    static constexpr int OFF_AM = OFF_W + W_STAGES * W_STAGE;
    static constexpr int OFF_S = OFF_AM + (MIN ? N_AM * 4096 : 0);        // [2] min-term B operand
    static constexpr int OFF_SCL = OFF_S + (MIN ? 2 * SUMS : 0);    // [4][128] block scales
    static constexpr int OFF_BAR = OFF_SCL + 4 * TILE_R * 4;
    static constexpr int SMEM = OFF_BAR + TM_BAR_BYTES;
};

// Scale of a row's accumulator for one block and the factor its min operand is divided by.  Normally s = d; where the
// ratio dmin / d leaves the f16 range of the min operand, s grows by powers of two and the integer operand shrinks with it.
struct TmScale {
    float s, ratio, shrink;   // shrink: factor of the integer operand (1 unless rare)
};
__device__ __forceinline__ TmScale tm_scale(float d, float dmin) {
    TmScale r{d, dmin / d, 1.f};
    if (!(fabsf(r.ratio) <= 512.f)) {   // 512 * 63 < 65504; also d == 0
        if (d == 0.f) { r.s = 1.f; r.shrink = 0.f; }
        for (int i = 0; i < 48 && fabsf(dmin / r.s) > 512.f; ++i) { r.s *= 2.f; r.shrink *= 0.5f; }
        r.ratio = dmin / r.s;
    }
    return r;
}

template <int DT, int CAP>
__global__ void __launch_bounds__(TM_THREADS, 1) gemm_tm_kernel(const TmParams p) {
    using T = TmFmt<DT, CAP>;
    constexpr bool SEG = CAP == TM_SEG;
    static_assert(T::SMEM <= 227 * 1024 && (2 * T::W_STAGES + 3 * T::NS + 16 + 3 * T::ND) * 8 <= TM_BAR_BYTES, "shared memory budget");
    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t* b_ring = smem;
    uint8_t* w_ring = smem + T::OFF_W;
    float* scl = reinterpret_cast<float*>(smem + T::OFF_SCL);
    uint64_t* w_full = reinterpret_cast<uint64_t*>(smem + T::OFF_BAR);
    uint64_t* w_empty = w_full + T::W_STAGES;
    uint64_t* b_full = w_empty + T::W_STAGES;   // [block & 1][slot]
    uint64_t* b_empty = b_full + 2 * T::NS;
    uint64_t* s_full = b_empty + T::NS;   // [2] sub-block sums of a block
    uint64_t* s_empty = s_full + 2;
    uint64_t* a_ready = s_empty + 2;            // [block & 1][use in the block][group] unpacked weights are in tensor memory
    uint64_t* a_free = a_ready + 8;             // [A buffer of the group][group]
    uint64_t* d_ready = a_free + 4;             // [accumulator] every MMA of a half block has completed
    uint64_t* d_free = d_ready + T::ND;         // [issuer that uses it next][accumulator] it has been read back
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(16) float tok_scale[TM_TOK];
    __shared__ int abort_flag;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < T::W_STAGES; ++i) { mbar_init(&w_full[i], 1); mbar_init(&w_empty[i], TM_UNPACK_WARPS); }
        for (int i = 0; i < T::NS; ++i) { mbar_init(&b_full[i], 1); mbar_init(&b_full[T::NS + i], 1); mbar_init(&b_empty[i], 1); }
        for (int i = 0; i < 8; ++i) mbar_init(&a_ready[i], TM_GROUP_WARPS);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&s_full[i], 1);
            mbar_init(&s_empty[i], 1);
            mbar_init(&a_free[i], 1);
            mbar_init(&a_free[2 + i], 1);
        }
        for (int i = 0; i < T::ND; ++i) {
            mbar_init(&d_ready[i], 1);
            mbar_init(&d_free[i], TM_DRAIN_WARPS);
            mbar_init(&d_free[T::ND + i], TM_DRAIN_WARPS);
        }
        abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == TM_MMA_WARP) tmem_alloc(&tmem_slot, 512);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = tmem_slot;
    pdl_launch_dependents();

    // item -> (row tile, split, token tile): the token tiles of one weight tile are neighbours, so that its bytes come from
    // HBM once and from L2 for the others.  Segments: the row tiles of one segment are neighbours, they share its activations.
    int n_items = p.row_tiles * p.splits * p.tok_tiles;
    if (SEG) {   // the list comes from the kernel before
        pdl_wait();
        const int n = p.g.n_seg ? *p.g.n_seg + p.g.n_more : p.g.max_seg;
        n_items = (n < p.g.max_seg ? n : p.g.max_seg) * p.g.n_tiles;
    }
    struct Item { int rt, tt, kb0, n_kb, sp, rows; };   // weight row tile, token tile or segment, column blocks of the matrix, split, live rows
    auto item_of = [&](int idx) {
        Item it;
        if (SEG) {
            it.tt = p.g.first + idx / p.g.n_tiles;
            it.sp = idx % p.g.n_tiles;   // column tile of the output
            const int2 s = p.g.seg[it.tt];
            it.rt = s.x * p.g.tiles_per_block + it.sp + (it.sp >= p.g.half_tiles ? p.g.half_off - p.g.half_tiles : 0);
            it.kb0 = s.x * p.g.kb_per_block;
            it.n_kb = p.g.kblocks;
            it.rows = s.y;
            return it;
        }
        it.tt = idx % p.tok_tiles;
        const int r = idx / p.tok_tiles;
        it.sp = r % p.splits;
        it.rt = r / p.splits;
        it.kb0 = (int)((long long)it.sp * p.kblocks / p.splits);
        it.n_kb = (int)((long long)(it.sp + 1) * p.kblocks / p.splits) - it.kb0;
        it.rows = p.tile_tok;
        return it;
    };
    auto tok_of = [&](const Item& it) { return SEG ? tm_seg_tok(it.rows) : p.tile_tok; };   // tokens its activation chunks hold
    bool ok = true;

    if (warp == TM_W_WARP) {
        // ------------------------------ weights ------------------------------
        if (lane == 0) {
            int s = 0;
            uint32_t round = 0;
            for (int idx = blockIdx.x; idx < n_items && ok; idx += gridDim.x) {
                const Item it = item_of(idx);
                const uint8_t* src = p.w + ((uint64_t)it.rt * p.kblocks + it.kb0) * T::W_STAGE;
                for (int k = 0; k < it.n_kb; ++k, src += T::W_STAGE) {
                    if (round > 0 && !(ok = mbar_wait_one(&w_empty[s], (round - 1) & 1, p.err, DEV_ERR_WAIT_EMPTY))) break;
                    mbar_arrive_expect_tx(&w_full[s], T::W_STAGE);
                    bulk_g2s(w_ring + s * T::W_STAGE, src, T::W_STAGE, &w_full[s]);
                    if (++s == T::W_STAGES) { s = 0; ++round; }
                }
            }
        }
    } else if (warp == TM_B_WARP) {
        // ------------------------------ activations ------------------------------
        if (lane == 0) {
            pdl_wait();
            int s = 0;
            uint32_t round = 0, e = 0;
            for (int idx = blockIdx.x; idx < n_items && ok; idx += gridDim.x) {
                const Item it = item_of(idx);
                const int tok = tok_of(it), spacing = tm_chunk(SEG ? CAP : tok), stage = tm_bstage(tok), sums = tm_sums(tok);
                const uint8_t* src = p.acts + (SEG ? (uint64_t)it.tt * it.n_kb : (uint64_t)it.tt * p.kblocks + it.kb0) * spacing;
                for (int k = 0; k < it.n_kb && ok; ++k, src += spacing, ++e) {
                    if (T::MIN) {
                        if (e >= 2) ok = mbar_wait_one(&s_empty[e & 1], ((e >> 1) - 1) & 1, p.err, DEV_ERR_WAIT_EMPTY);
                        if (!ok) break;
                        mbar_arrive_expect_tx(&s_full[e & 1], sums);
                        bulk_g2s(smem + T::OFF_S + (e & 1) * T::SUMS, src + 4 * stage, sums, &s_full[e & 1]);
                    }
                    for (int q = 0; q < 4; q += T::SQ) {
                        if (round > 0 && !(ok = mbar_wait_one(&b_empty[s], (round - 1) & 1, p.err, DEV_ERR_WAIT_EMPTY))) break;
                        uint64_t* fb = &b_full[(e & 1) * T::NS + s];
                        mbar_arrive_expect_tx(fb, T::SQ * stage);
                        bulk_g2s(b_ring + s * (T::SQ * T::BSTAGE), src + q * stage, T::SQ * stage, fb);
                        if (++s == T::NS) { s = 0; ++round; }
                    }
                }
            }
        }
    } else if (warp >= TM_MMA_WARP) {
        // ------------------------------ MMA issue ------------------------------
        // All tensor-memory addresses are literals (the CTA owns all 512 columns, so the allocation starts at 0), so that the
        // issuing thread spends its slots on MMAs.
        uint32_t IDESC = instr_desc(p.tile_tok), tok = p.tile_tok;
        const uint32_t b_addr = smem_u32(b_ring), am_addr = smem_u32(smem + T::OFF_AM), s_addr = smem_u32(smem + T::OFF_S);
        uint32_t e = 0, am = 0;   // am = e % N_AM
        uint32_t b_phase = 0;             // bit s: parity of this issuer's next use of slot s
        uint32_t d_phase = 0, dn = 0;     // bit i: the same for its accumulators; dn = 2 e % 3, for rings of three
        auto wait = [&](uint64_t* bar, uint32_t parity) {
            ok = mbar_wait_one(bar, parity, p.err, DEV_ERR_WAIT_FULL);
            return ok;
        };
        auto block = [&](auto odd) {   // one 256-column block: a half into one accumulator, a half into the next
            constexpr uint32_t O = decltype(odd)::value;
            constexpr bool HOLD = T::MIN || T::NA == 2;   // both stages' weights stay until the half is complete
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                uint32_t i = T::ND == 4 ? 2 * O + u : u;   // accumulator of half 2 e + u
                if (T::ND == 3) i = dn + u >= 3 ? dn + u - 3 : dn + u;
                const uint32_t D = i * CAP;
                if (2 * e + u >= (uint32_t)T::ND) {
                    if (!wait(&d_free[O * T::ND + i], (d_phase >> i) & 1)) return;
                    d_phase ^= 1u << i;
                }
                uint64_t bd[2];
                uint32_t a_at[2], slot[2];
                auto arrived = [&](int x) {   // the weights and activations of 64 columns
                    const int g = T::MIN ? u : x, ab = T::NA == 1 ? 0 : T::MIN ? (int)O : u;   // use number modulo the group's buffers
                    if ((!T::MIN || x == 0) && !wait(&a_ready[4 * O + (T::MIN ? 0 : 2 * u) + g], (e >> 1) & 1)) return false;
                    a_at[x] = T::A + 128 * ab + 64 * g + (T::MIN ? 32 * x : 0);
                    if (T::SQ == 1 || x == 0) {
                        slot[x] = T::SQ == 1 ? 2 * u + x : T::NS == 4 ? 2 * O + u : (dn + u >= 3 ? dn + u - 3 : dn + u);
                        if (!wait(&b_full[O * T::NS + slot[x]], (b_phase >> slot[x]) & 1)) return false;
                        b_phase ^= 1u << slot[x];
                    } else slot[x] = slot[0];
                    fence_after_sync();
                    bd[x] = smem_desc(b_addr + slot[x] * (T::SQ * T::BSTAGE) + (T::SQ == 2 ? x * tm_bstage((int)tok) : 0), tok * 16, 128);   // address field: 16-byte units
                    return true;
                };
                // What lies below the weights' hi part times the activations' hi plane: beside it some 2^-11, so that what a step drops of
                // the running sum is nothing as long as these come first.
                auto small = [&](int x, bool fresh) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        mma_ts_rt(D, a_at[x] + 8 * j, bd[x] + j * (2 * tok) + 8 * tok, IDESC, !(fresh && j == 0));
                        if (!T::MIN) mma_ts_rt(D, a_at[x] + 8 * j + 32, bd[x] + j * (2 * tok), IDESC, 1u);
                    }
                };
                auto large = [&](int x) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) mma_ts_rt(D, a_at[x] + 8 * j, bd[x] + j * (2 * tok), IDESC, 1u);
                    if (T::SQ == 1 || x == 1) mma_commit(&b_empty[slot[x]]);
                };
                auto weights_free = [&](int x) { mma_commit(&a_free[2 * (T::NA == 1 ? 0 : T::MIN ? (int)O : u) + (T::MIN ? u : x)]); };
                if (!arrived(0)) return;
                small(0, true);
                if (!HOLD) { large(0); weights_free(0); }
                if (!arrived(1)) return;
                small(1, false);
                const bool mins = T::MIN && u == 1;
                const uint64_t ad = smem_desc(am_addr + am * 4096, 2048, 128), sd = smem_desc(s_addr + O * T::SUMS, tok * 16, 128);
                if (mins) {
                    if (!wait(&s_full[O], (e >> 1) & 1)) return;
                    fence_after_sync();
                    mma_ss(D, ad, sd + 2 * tok, IDESC, 1u);
                }
                if (HOLD) large(0);
                large(1);
                if (mins) {
                    mma_ss(D, ad, sd, IDESC, 1u);
                    mma_commit(&s_empty[O]);
                }
                if (HOLD && !T::MIN) weights_free(0);
                weights_free(1);
                mma_commit(&d_ready[i]);
            }
        };
        if (elect_one()) {   // one thread runs the whole loop: nothing to vote on between two MMAs
            if (tmem != 0) {
                atomicCAS(p.err, 0, DEV_ERR_WAIT_FULL);
                ok = false;
            }
            for (int idx = blockIdx.x; idx < n_items && ok; idx += gridDim.x) {
                const Item it = item_of(idx);
                const int n_kb = it.n_kb;
                if (SEG) {
                    tok = tok_of(it);
                    IDESC = instr_desc(tok);
                }
                for (int k = 0; k < n_kb && ok; ++k, ++e, am = am == T::N_AM - 1 ? 0 : am + 1, dn = (dn + 2) % 3) {
                    if ((e & 1) != (uint32_t)(warp - TM_MMA_WARP)) continue;
                    if (e & 1) block(std::integral_constant<uint32_t, 1>{});
                    else block(std::integral_constant<uint32_t, 0>{});
                }
            }
        }
        __syncwarp();
    } else if (warp < TM_UNPACK_WARPS) {
        // ------------------------------ unpack ------------------------------
        if constexpr (CAP != TM_SEG) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(TM_REGS_UNPACK));
        const int g = warp >> 3, q4 = warp & 3, kp2 = (warp >> 2) & 1;
        const int row = 32 * q4 + lane;
        const uint32_t a_buf = tmem + ((uint32_t)(32 * q4) << 16) + T::A + 64 * g;
        uint32_t e = 0, use = 0, am_buf = 0;   // am_buf = e % N_AM
        int s = 0;
        uint32_t round = 0;
        for (int idx = blockIdx.x; idx < n_items && ok; idx += gridDim.x) {
            const int n_kb = item_of(idx).n_kb;
            for (int k = 0; k < n_kb && ok; ++k, ++e, am_buf = am_buf == T::N_AM - 1 ? 0 : am_buf + 1) {
                ok = mbar_wait_warp(&w_full[s], round & 1, p.err, DEV_ERR_WAIT_FULL);
                if (!ok) break;
                const uint8_t* st = w_ring + s * T::W_STAGE;
#pragma unroll
                for (int u = 0; u < T::USES; ++u, ++use) {
                    uint32_t r[32], am = 0u;
                    UnitScales us{0.f, 0.f};
                    TmScale sc{0.f, 0.f, 1.f};
                    if constexpr (T::MIN) {
                        Fmt<DT>::unpack(st, g, row, kp2, r, am, us);
                        sc = tm_scale(us.d, us.dmin);
                        if (sc.shrink != 1.f) {
                            const __half2 f2 = __float2half2_rn(sc.shrink);
                            const uint32_t f = *reinterpret_cast<const uint32_t*>(&f2);
#pragma unroll
                            for (int i = 0; i < 32; ++i) r[i] = h2mul(r[i], f);
                        }
                    } else {
                        tm_unpack_q6k(st, g + 2 * u, row, kp2, r, us);
                        sc.s = us.d;
                    }
                    if (u == T::USES - 1) {
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&w_empty[s]);   // every lane has its bytes in registers
                    }
                    const uint32_t ab = T::NA == 1 ? 0 : use & 1, a_dst = a_buf + 128 * ab;
                    if (use >= T::NA) {
                        ok = mbar_wait_warp(&a_free[2 * ab + g], (T::NA == 1 ? use - 1 : (use >> 1) - 1) & 1, p.err, DEV_ERR_WAIT_FULL);
                        if (!ok) break;
                        fence_after_sync();
                    }
                    if (T::MIN) {
                        tmem_st32(a_dst + 32 * kp2, r);
                        // the min operand of this thread's two sub-blocks, k = 2 kp and 2 kp + 1 (hi) and 8 further (lo)
                        const float2 m = __half22float2(*reinterpret_cast<const __half2*>(&am));
                        const float f0 = -sc.ratio * m.x, f1 = -sc.ratio * m.y;
                        const __half2 hi = __floats2half2_rn(f0, f1);
                        const float2 back = __half22float2(hi);
                        const __half2 lo = __floats2half2_rn(f0 - back.x, f1 - back.y);
                        uint8_t* dst = smem + T::OFF_AM + am_buf * 4096 + (row >> 3) * 128 + (row & 7) * 16 + (2 * g + kp2) * 4;
                        *reinterpret_cast<__half2*>(dst) = hi;
                        *reinterpret_cast<__half2*>(dst + 2048) = lo;
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    } else {
                        uint32_t a1[16], a2[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i) { a1[i] = r[i]; a2[i] = r[16 + i]; }
                        tmem_st16(a_dst + 16 * kp2, a1);
                        tmem_st16(a_dst + 32 + 16 * kp2, a2);
                    }
                    if (g == 0 && u == 0 && kp2 == 0) scl[(e & 3) * TILE_R + row] = sc.s;
                    wait_st();
                    fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&a_ready[4 * (e & 1) + 2 * u + g]);
                }
                if (++s == T::W_STAGES) { s = 0; ++round; }
            }
        }
    } else {
        // ------------------------------ read-back ------------------------------
        if constexpr (CAP != TM_SEG) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(TM_REGS_DRAIN));
        pdl_wait();
        const int row = (threadIdx.x - TM_DRAIN_WARP0 * 32) & 127;   // weight row of the tile = tensor-memory lane
        const int half = (warp - TM_DRAIN_WARP0) >> 2;   // takes the first or the second half of the tile's 16-token columns
        const uint32_t tm_l = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
        constexpr int NC = (CAP / 16 + 1) / 2;        // 16-token pieces that a thread holds at most
        float acc[NC][16];                            // their running sums over the column blocks
        uint32_t e = 0, di = 0, d_par = 0;            // accumulator of the next half, parity of its use
        int scaled_tt = -1;
        // A warp that has given up a wait still walks the items: the named barriers below have no limit, so all eight warps must come.
        for (int idx = blockIdx.x; idx < n_items; idx += gridDim.x) {
            const Item it = item_of(idx);
            const int n_c = (it.rows + 15) / 16, c0 = half ? (n_c + 1) / 2 : 0, n_mine = half ? n_c - c0 : (n_c + 1) / 2;
            const int live = SEG ? it.rows : p.n_rows - it.tt * p.tile_tok;
            if (it.tt != scaled_tt) {   // per-token output scale of the token tile, thread = token
                scaled_tt = it.tt;
                named_sync(1, TM_DRAIN_WARPS * 32);
                if (half == 0 && row < it.rows) {
                    float sc = p.out_scale;
                    if (SEG) {
                        if (p.g.row_scale) sc *= p.g.row_scale[it.tt * CAP + row];
                    } else if (p.sumsq) {
                        float ss = 0.f;
                        for (int q = 0; q < p.n_sumsq; ++q) ss += p.sumsq[(uint64_t)q * p.rows_pad + it.tt * p.tile_tok + row];
                        sc *= 1.0f / sqrtf(ss / p.norm_k + p.eps);
                    }
                    tok_scale[row] = sc;
                }
                named_sync(1, TM_DRAIN_WARPS * 32);
            }
#pragma unroll
            for (int x = 0; x < NC; ++x)
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[x][j] = 0.f;
            for (int k = 0; k < it.n_kb && ok; ++k, ++e) {
                float s = 0.f;
#pragma unroll 1
                for (int u = 0; u < 2; ++u) {
                    ok = CAP == TM_SEG ? mbar_wait_warp(&d_ready[di], d_par, p.err, DEV_ERR_WAIT_FULL) : mbar_wait_warp_inline(&d_ready[di], d_par, p.err, DEV_ERR_WAIT_FULL);
                    if (!ok) break;
                    fence_after_sync();
                    if (u == 0) s = scl[(e & 3) * TILE_R + row];
                    const uint32_t d = tm_l + di * CAP + 16 * c0;
#pragma unroll
                    for (int x = 0; x < NC; ++x) {
                        float v[16];
                        if (x < n_mine) tmem_ld16(d + 16 * x, v);
                        wait_ld();
                        if (x + 1 == NC) {   // read: back to the issuer of the half that uses it next
                            fence_before_sync();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(&d_free[((e + (uint32_t)(u + T::ND) / 2) & 1) * T::ND + di]);
                        }
                        if (x < n_mine) {
#pragma unroll
                            for (int j = 0; j < 16; ++j) acc[x][j] = fmaf(s, v[j], acc[x][j]);
                        }
                    }
                    if (++di == (uint32_t)T::ND) { di = 0; d_par ^= 1; }
                }
                if (!ok) break;
            }
            if (!ok) continue;
            const uint32_t orow = (uint32_t)(SEG ? it.sp : it.rt) * TILE_R + row;
#pragma unroll
            for (int x = 0; x < NC; ++x) {
                if (x >= n_mine) continue;
                const int c = c0 + x;
                // every scale before the first store: a load of shared memory behind a store to global memory waits for its turn in the
                // same queue, 70 - 110 clocks a token
#pragma unroll
                for (int j = 0; j < 16; j += 4) {
                    const float4 t = *reinterpret_cast<const float4*>(tok_scale + 16 * c + j);
                    acc[x][j] *= t.x; acc[x][j + 1] *= t.y; acc[x][j + 2] *= t.z; acc[x][j + 3] *= t.w;
                }
            }
            if (orow < p.n_out) {
#pragma unroll
                for (int x = 0; x < NC; ++x) {
                    if (x >= n_mine) continue;
                    const int c = c0 + x, tok0 = (SEG ? it.tt * CAP : it.sp * p.rows_pad + it.tt * p.tile_tok) + 16 * c;
                    float* dst = p.out + (uint64_t)tok0 * p.ld_out + orow;
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (16 * c + j < live) dst[(uint64_t)j * p.ld_out] = acc[x][j];
                }
            }
            __syncwarp();
        }
    }
    if (!ok) abort_flag = 1;
    fence_before_sync();
    __syncthreads();
    if (abort_flag && threadIdx.x == 0) {
        // error word already set: a bounded chance for copies still in flight before the shared memory is released
        auto settle = [](uint64_t* b) {
            uint32_t spins = 0;
            while (!mbar_try_wait(b, 0) && !mbar_try_wait(b, 1) && ++spins < (1u << 16)) __nanosleep(100);
        };
        for (int i = 0; i < T::W_STAGES; ++i) settle(&w_full[i]);
        for (int i = 0; i < 2 * T::NS; ++i) settle(&b_full[i]);
        for (int i = 0; i < 2; ++i) settle(&s_full[i]);
    }
    __syncthreads();
    if (warp == TM_MMA_WARP) {
        fence_after_sync();
        tmem_free(tmem, 512);
    }
}

template <int DT, int CAP>
static dfl_status launch_tm(cudaStream_t st, const TmParams& p, int n_items) {
    static std::once_flag once[16];
    int dev = 0;
    cudaGetDevice(&dev);
    cudaError_t e = cudaSuccess;
    auto set = [&] { e = cudaFuncSetAttribute(gemm_tm_kernel<DT, CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, TmFmt<DT, CAP>::SMEM); };
    if (dev >= 0 && dev < 16) std::call_once(once[dev], set);
    else set();
    DFL_CUDA(e);
    static std::atomic<bool> regs_seen{false};   // a build with fewer registers at launch would wait for ones that there are not
    if (CAP != TM_SEG && !regs_seen.load(std::memory_order_relaxed)) {
        cudaFuncAttributes a{};
        DFL_CUDA(cudaFuncGetAttributes(&a, gemm_tm_kernel<DT, CAP>));
        if (a.numRegs != TM_REGS) return fail(DFL_ERR_UNSUPPORTED, "many-row gemm: built for " + std::to_string(a.numRegs) + " registers a thread");
        regs_seen.store(true, std::memory_order_relaxed);
    }
    DFL_CUDA(launch_k(gemm_tm_kernel<DT, CAP>, dim3((unsigned)(n_items < sm_count() ? n_items : sm_count())), dim3(TM_THREADS), (size_t)TmFmt<DT, CAP>::SMEM, st, p));
    count_launch();
    return DFL_OK;
}

}  // namespace ts

// Tokens per tile of a pass: as few tiles as possible, of equal size (the time of a block follows the tile's tokens).
int gemm_tm_tile_tok(int n_rows) {
    const int tiles = (n_rows + TM_TOK - 1) / TM_TOK;
    return ((n_rows + tiles - 1) / tiles + 15) / 16 * 16;
}

// Split count of a many-row launch: waves of items times blocks per item (an item pays about a third of a block to start
// and to end), plus the traffic of the partial slices (64 KiB per item written and read again, in units of a block's time).
int gemm_tm_choose_splits(const int* row_tiles, int n_mats, int kblocks, int tok_tiles) {
    int best = 1;
    double best_cost = 1e30;
    for (int s = 1; s <= 8 && s <= kblocks; ++s) {
        double cost = 0.0;
        for (int i = 0; i < n_mats; ++i) {
            const int items = row_tiles[i] * tok_tiles * s;
            const int rounds = (items + sm_count() - 1) / sm_count();
            cost += rounds * ((double)((kblocks + s - 1) / s) + 0.35) + 0.02 * items;
        }
        if (cost < best_cost) { best_cost = cost; best = s; }
    }
    return best;
}

bool gemm_tm_supported(const QMatrix& m) {
    return m.layout == LAYOUT_TS && (m.dtype == DFL_Q4_K || m.dtype == DFL_Q5_K || m.dtype == DFL_Q6_K);
}

dfl_status launch_gemm_tm(cudaStream_t st, const QMatrix& m, const uint8_t* acts, float* out, int splits, int n_rows, int tile_tok,
                          const float* sumsq, int n_sumsq, float norm_k, float eps, float out_scale, uint32_t ld_out, int* dev_err) {
    if (!gemm_tm_supported(m)) return fail(DFL_ERR_UNSUPPORTED, "many-row gemm: weight dtype");
    if (splits < 1 || splits > m.kblocks || n_rows < 1 || tile_tok < 16 || tile_tok > TM_TOK || tile_tok % 16)
        return fail(DFL_ERR_BAD_ARG, "many-row gemm: shape");
    ts::TmParams p;
    p.w = m.tiles; p.acts = acts; p.out = out; p.sumsq = sumsq; p.n_sumsq = n_sumsq; p.norm_k = norm_k; p.eps = eps; p.out_scale = out_scale;
    p.kblocks = m.kblocks; p.splits = splits; p.row_tiles = m.row_tiles; p.tile_tok = tile_tok; p.tok_tiles = (n_rows + tile_tok - 1) / tile_tok;
    p.n_rows = n_rows; p.rows_pad = p.tok_tiles * tile_tok; p.n_out = (uint32_t)m.n_out; p.ld_out = ld_out ? ld_out : (uint32_t)m.n_out; p.err = dev_err;
    const int n_items = p.row_tiles * p.splits * p.tok_tiles;
    // Up to 80 tokens the deeper rings pay for Q4_K and Q5_K (4096 -> 24576 over 77 rows: 41.4 -> 38.7 us, 32 rows 36.4 -> 32.6);
    // Q6_K, whose two passes per block keep the tensor pipe busier, was the same or slower (44.3 -> 45.8).
    if (tile_tok <= ts::TM_SMALL && m.dtype == DFL_Q4_K) return ts::launch_tm<DFL_Q4_K, ts::TM_SMALL>(st, p, n_items);
    if (tile_tok <= ts::TM_SMALL && m.dtype == DFL_Q5_K) return ts::launch_tm<DFL_Q5_K, ts::TM_SMALL>(st, p, n_items);
    switch (m.dtype) {
        case DFL_Q4_K: return ts::launch_tm<DFL_Q4_K, TM_TOK>(st, p, n_items);
        case DFL_Q5_K: return ts::launch_tm<DFL_Q5_K, TM_TOK>(st, p, n_items);
        default: return ts::launch_tm<DFL_Q6_K, TM_TOK>(st, p, n_items);
    }
}

dfl_status launch_gemm_tm_seg(cudaStream_t st, const QMatrix& m, const TmSegments& g, const uint8_t* acts, float* out, float out_scale,
                              uint32_t ld_out, int* dev_err) {
    if (!gemm_tm_supported(m)) return fail(DFL_ERR_UNSUPPORTED, "segment gemm: weight dtype");
    if (!g.seg || g.max_seg < 1 || g.n_tiles < 1 || g.kblocks < 1 || g.kblocks > m.kblocks) return fail(DFL_ERR_BAD_ARG, "segment gemm: shape");
    ts::TmParams p{};
    p.w = m.tiles; p.acts = acts; p.out = out; p.out_scale = out_scale; p.kblocks = m.kblocks;
    p.n_out = (uint32_t)g.n_tiles * TILE_R; p.ld_out = ld_out; p.err = dev_err; p.g = g; p.tile_tok = TM_SEG;
    const int n_items = g.max_seg * g.n_tiles;   // the most there can be
    switch (m.dtype) {
        case DFL_Q4_K: return ts::launch_tm<DFL_Q4_K, TM_SEG>(st, p, n_items);
        case DFL_Q5_K: return ts::launch_tm<DFL_Q5_K, TM_SEG>(st, p, n_items);
        default: return ts::launch_tm<DFL_Q6_K, TM_SEG>(st, p, n_items);
    }
}

}  // namespace dfl
