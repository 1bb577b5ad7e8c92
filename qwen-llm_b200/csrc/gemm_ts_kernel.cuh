// Kernel body and launcher of the tensor-memory few-row GEMM; included by gemm_ts.cu only.
//
// CTA = one split (at most KC column blocks, activations resident) x every ctas_per_split-th
// row tile.  Its work is the sequence of entries e = (tile, column block); the weight stage of
// entry e travels through ring slot e % STAGES.  The eight unpacking warps form two groups of
// four that take the entries alternately (group = e & 1), each with its own A buffer,
// accumulators and barriers, so that one group's arithmetic fills the time the other spends
// storing to tensor memory and waiting.  A group unpacks an entry in HALVES steps of 64 A-buffer
// columns (Q4_K / Q5_K: two halves of 128 weight columns; Q6_K: four of 64, each written as the
// even / odd scale parts); the MMA warp issues eight MMAs per half as soon as it is stored.
//
//   producer thread     ring slot free?   -> bulk copy of the stage          -> full[slot]   (activations: a draining thread)
//   unpacking group g   full[slot]        -> registers -> a_free[g][half]?   -> tcgen05.st -> a_ready[g][half], empty[slot]
//   MMA warp (g, c)     a_ready[g][c], d_free[g]?    -> 8 tcgen05.mma (+ min) -> commit: a_free[g][c], d_ready[g]
//                       (c = half % 2: its MMAs accumulate into accumulator c of the group, so the order in which the
//                       two warps of a group reach the tensor pipe does not change a bit of the result.  Two accumulators are also
//                       what keeps the precision: each step of a tensor-core sum drops what lies below the sum's last place, and
//                       one accumulator of twice the steps was 1.7 times further from the float64 result, for 1.3 % of the time)
//   4 draining warps    d_ready[g]        -> tcgen05.ld -> d_free[g]         -> scale, add; tile end: global store
//
// The super-block scales d / dmin of an entry travel from the unpacking threads to the draining
// thread of the same row through a four-slot shared-memory side buffer (slot = entry & 3).
#pragma once

namespace dfl {
namespace ts {

struct Params {
    const uint8_t* w;
    const uint8_t* acts;
    float* out;
    const float* sumsq;
    int n_sumsq;
    float norm_k, eps, out_scale;
    int kblocks, splits, row_tiles, ctas_per_split;
    uint32_t n_out, ld_out;
    int* err;
    const int32_t* tile_map;   // optional: row tiles to compute, and how many (device memory)
    const int32_t* n_tiles;
    const int32_t* kb_map;     // optional: column blocks to sum over, and how many (device memory)
    const int32_t* n_kb;
    uint32_t* late_word;       // LateMark
    uint32_t late_value;
    int late_mode;             // LATE_FIRST: lets the next kernel start behind the dependency wait instead of at once, and publishes the mark there;
                               // LATE_BEHIND: acquires it before the inputs, the dependency wait is for the kernels behind
};

constexpr int LATE_FIRST = 1, LATE_BEHIND = 2;
// Every launch fetches its parameters cold: with sixteen bytes more a 9B-class verify block of 340 launches took 0.3 - 0.5 % longer.
static_assert(sizeof(Params) <= 128, "parameters of the few-row GEMM");

constexpr int FR_GROUP_WARPS = 4;                           // unpacking warps per group; thread = weight row = 32 * (warp % 4) + lane
constexpr int FR_UNPACK_WARPS = 2 * FR_GROUP_WARPS;         // two groups that take the entries alternately
constexpr int DRAIN_WARP0 = 8, DRAIN_WARPS = 4;             // thread = weight row; warp % 4 = its quarter of the tensor-memory lanes
constexpr int MMA_WARP0 = 12, MMA_WARPS = 4;                // warp 12 + 2 g + c issues the MMAs of group g's halves h with h % 2 == c
constexpr int PRODUCER_WARP = 16;
// 96 registers, the most that five warps on one scheduler leave.  With 88 a small CTA of the next kernel fits beside a GEMM CTA, but the GEMM lost
// more (4096 x 24576 Q4_K 15.9 -> 16.4 us) than the early start gave; fifteen warps, two of which issue the MMAs, were 5 % slower.
constexpr int THREADS = 17 * 32, REGS = 96;
constexpr int SCL_BYTES = 4 * TILE_R * 8;   // four entries' {d, dmin} per row
constexpr int BAR_BYTES = 512;              // up to 64 mbarriers

template <int DT, int KC>
constexpr int smem_bytes() {
    return KC * ACTTS_CHUNK + Fmt<DT>::stages(KC) * Fmt<DT>::STAGE + SCL_BYTES + BAR_BYTES;
}

// named barrier among the draining warps only (every one of them reaches it unconditionally)
__device__ __forceinline__ void named_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }

// Whether the MMA warp of entry e (group e & 1, column block e % n_kb) waits for the block's activations: at its own first use of
// the block.  With an even count a group meets the same blocks in every row tile; with an odd one its second tile brings the blocks that
// only the other group has waited for (one block and two tiles: group 1's first entry).  The barrier has one phase, so a wait
// that is not needed costs a test.
__host__ __device__ constexpr bool waits_for_acts(int e, int n_kb) { return e < ((n_kb & 1) ? 2 * n_kb : n_kb); }
constexpr bool every_first_use_waits() {
    for (int n_kb = 1; n_kb <= KC_MAX; ++n_kb)
        for (int g = 0; g < 2; ++g)
            for (int kb = 0; kb < n_kb; ++kb)
                for (int e = g; e < 4 * n_kb; e += 2)   // the group's entries in order, four row tiles
                    if (e % n_kb == kb) {
                        if (!waits_for_acts(e, n_kb)) return false;
                        break;
                    }
    return true;
}
static_assert(every_first_use_waits(), "an MMA warp would read activations that may not have arrived");

// The eight MMAs of half h = 2 h2 + C of an entry into one accumulator (the first of them overwrites it when the half is
// the accumulator's first of the entry).
template <class F, int C>
__device__ __forceinline__ void issue_half(int h2, uint32_t d, uint32_t a_buf, uint32_t b_lo, uint32_t b_hi, uint32_t idesc) {
#pragma unroll
    for (int hh = 0; hh < F::HALVES / 2; ++hh) {
        if (hh != h2) continue;
        constexpr int dummy = 0;
        (void)dummy;
        const int h = 2 * hh + C;
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
            if (hh == 0 && jj == 0) mma_ts<false>(d, a_buf + F::a_col(h, jj), b_lo + F::b_slice(h, jj) * 64u, b_hi, idesc);
            else mma_ts<true>(d, a_buf + F::a_col(h, jj), b_lo + F::b_slice(h, jj) * 64u, b_hi, idesc);
        }
    }
}

template <int DT, int KC>
__global__ void __maxnreg__(REGS) gemm_ts_kernel(const Params p) {
    using F = Fmt<DT>;
    constexpr int STAGES = F::stages(KC), HALVES = F::HALVES;
    constexpr int OFF_RING = KC * ACTTS_CHUNK;
    constexpr int OFF_SCL = OFF_RING + STAGES * F::STAGE;
    constexpr int OFF_BAR = OFF_SCL + SCL_BYTES;
    // "Stage landed" barriers.  A parity wait is only meaningful to a waiter that knows the phase before is over, i.e. to
    // the one party that waits on that barrier phase after phase.  With an even number of stages a ring slot always
    // serves the same unpacking group; with an odd number its uses alternate between the two groups, and a group that
    // ran ahead could take the other group's still outstanding copy for its own (copies complete out of order).  So with
    // an odd number every slot has one barrier per group, each used by that group's uses of the slot only.
    constexpr int FULL_SETS = (STAGES & 1) ? 2 : 1;
    static_assert(OFF_BAR + BAR_BYTES <= 227 * 1024, "shared memory budget");
    static_assert((FULL_SETS + 1) * STAGES + KC + 12 <= BAR_BYTES / 8, "barrier area");
    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t* acts_res = smem;
    uint8_t* ring = smem + OFF_RING;
    float2* scl = reinterpret_cast<float2*>(smem + OFF_SCL);   // [entry & 3][row] = {d, dmin}
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
    uint64_t* empty = full + FULL_SETS * STAGES;
    auto full_bar = [](uint64_t* f, int e, int s) { return f + ((STAGES & 1) ? (e & 1) * STAGES : 0) + s; };
    // use number of the barrier: every use of the slot (even), or every second one (odd: the group's own)
    auto full_parity = [](int e) { return (uint32_t)((STAGES & 1) ? ((e / STAGES) >> 1) : (e / STAGES)) & 1u; };
    uint64_t* acts_bar = empty + STAGES;  // [column block of the CTA's range] its activations have arrived
    uint64_t* a_ready = acts_bar + KC;    // [group][half buffer] a half of unpacked weights is in tensor memory
    uint64_t* a_free = a_ready + 4;       // [group][half buffer] the MMAs of that half have completed
    uint64_t* d_ready = a_free + 4;       // [group] every MMA of an entry has completed
    uint64_t* d_free = d_ready + 2;       // [group] the draining warps have read the accumulator back
    __shared__ uint32_t tmem_slot;
    __shared__ float tok_scale[MAX_ROWS];
    __shared__ int abort_flag;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;   // warp-uniform by construction
    const uint32_t late_seen = p.late_mode == LATE_BEHIND ? late_peek(p.late_word) : 0u;
    if (threadIdx.x == 0) {
        for (int s = 0; s < FULL_SETS * STAGES; ++s) mbar_init(&full[s], 1);
        for (int s = 0; s < STAGES; ++s) mbar_init(&empty[s], FR_GROUP_WARPS);
        for (int k = 0; k < KC; ++k) mbar_init(&acts_bar[k], 1);
        for (int i = 0; i < 4; ++i) {
            mbar_init(&a_ready[i], FR_GROUP_WARPS);
            mbar_init(&a_free[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&d_ready[i], 2);
            mbar_init(&d_free[i], DRAIN_WARPS);
        }

        abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == MMA_WARP0) tmem_alloc(&tmem_slot, TM_COLS);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = tmem_slot;
    if (p.late_mode != LATE_FIRST) pdl_launch_dependents();
    auto wait_inputs = [&] {
        if (p.late_mode == LATE_BEHIND) late_acquire(p.late_word, p.late_value, late_seen);
        else pdl_wait();
    };
    int row_tiles = p.row_tiles, kblocks = p.kblocks, splits = p.splits, cps = p.ctas_per_split;
    if (p.tile_map || p.kb_map) {   // the lists come from the preceding kernel: nothing may be fetched before it is complete
        wait_inputs();
        if (p.tile_map) row_tiles = *p.n_tiles;
        if (p.kb_map) {
            kblocks = p.n_kb[0];
            if (p.n_kb[1] > 0) {   // the list's author also chose the split geometry for its length (the launch is the worst case)
                splits = p.n_kb[1];
                cps = p.n_kb[2];
            }
        }
    }
    const int sp = blockIdx.x % splits, c = blockIdx.x / splits;
    const int kb0 = (int)((long long)sp * kblocks / splits), kb1 = (int)((long long)(sp + 1) * kblocks / splits);
    const int n_kb = kb1 - kb0;
    const int n_my = (row_tiles - c + cps - 1) / cps;   // row tiles c, c + cps, ... (of the list)
    const int n_it = (int)blockIdx.x < splits * cps ? n_my * n_kb : 0;   // entries; none for a CTA beyond the geometry in use

    // The late form: every thread passes the dependency wait first, each role where it has nothing else to do (it does not matter how many of
    // a CTA's threads the hardware counts, and a second call does nothing).
    auto trigger = [&] {
        if (p.late_mode != LATE_FIRST) return;
        pdl_wait();
        pdl_launch_dependents();
    };

    if (warp == PRODUCER_WARP) {
        // ------------------------------ bulk-copy producer ------------------------------
        // Weights do not depend on the previous kernel: the ring is filled without waiting for it.  (Fetching 3 - 16 stages more into L2 meanwhile
        // made the Q6_K launches 0.7 - 1.2 us shorter and the kernels before, whose loads it delayed, as much longer.)
        // The whole warp walks the loop, one lane issues; slot / round / source are kept by addition.
        const uint64_t tile_stride = (uint64_t)p.kblocks * F::STAGE;
        const bool mapped = p.tile_map != nullptr || p.kb_map != nullptr;
        int pt = 0, pk = 0, s = 0;
        uint32_t round = 0;
        const uint8_t* src = p.w + (uint64_t)c * tile_stride + (uint64_t)kb0 * F::STAGE;   // tile c, first column block of the range
        const uint64_t next_tile = (uint64_t)cps * tile_stride - (uint64_t)n_kb * F::STAGE;   // from the range's end to its start in the CTA's next tile
        bool ok = true;
        for (int e = 0; e < n_it; ++e) {
            if (round > 0) ok = mbar_wait_warp(&empty[s], (round - 1) & 1, p.err, DEV_ERR_WAIT_EMPTY);
            if (!ok) break;
            if (round == 1 && s == 0) trigger();
            if (mapped) {
                const int slot = c + pt * cps;
                src = p.w + (uint64_t)(p.tile_map ? p.tile_map[slot] : slot) * tile_stride +
                      (uint64_t)(p.kb_map ? p.kb_map[kb0 + pk] : kb0 + pk) * F::STAGE;
            }
            if (lane == 0) {
                uint64_t* fb = full_bar(full, e, s);
                mbar_arrive_expect_tx(fb, F::STAGE);
                bulk_g2s(ring + s * F::STAGE, src, F::STAGE, fb);
            }
            src += F::STAGE;
            if (++pk == n_kb) {   // next row tile of this CTA: cps tiles further, back to the first column block
                pk = 0;
                ++pt;
                src += next_tile;
            }
            if (++s == STAGES) { s = 0; ++round; }
        }
        if (!ok) abort_flag = 1;
        trigger();
        // Here the warp has nothing left to do, and the last CTA has the fewest row tiles: the next kernel finds no room before most others have
        // ended.  (From roles of the first CTA that the fence of the release held up, and from its producer, a token took 0.4 - 0.7 % longer.)
        if (p.late_mode == LATE_FIRST && blockIdx.x == gridDim.x - 1 && lane == 0) late_publish(p.late_word, p.late_value);
    } else if (warp >= MMA_WARP0 && warp < MMA_WARP0 + MMA_WARPS) {
        // ------------------------------ MMA issuers ------------------------------
        // Warp (g, c) issues the halves h with h % 2 == c of group g's entries into accumulator c of that group.  The
        // whole warp walks the loop so that addresses and descriptors stay warp-uniform; one elected lane issues.
        trigger();
        constexpr uint32_t IDESC_MAIN = instr_desc(32), IDESC_MIN = instr_desc(48);
        const uint32_t g = (uint32_t)(warp - MMA_WARP0) >> 1, c = (uint32_t)(warp - MMA_WARP0) & 1u;
        bool ok = true;
        const uint32_t acts_addr = smem_u32(acts_res);
        const uint32_t a_buf = tmem + TM_A + g * TM_A_STRIDE, d_buf = tmem + TM_D + g * TM_D_STRIDE + 32 * c;
        uint32_t uses = 0;   // how often this warp's half buffer has been used
        int kb_e = (int)g % n_kb;   // e % n_kb, kept by addition
        const int kb_step = 2 % n_kb;
        for (int e = (int)g; e < n_it && ok; e += 2) {
            const uint32_t chunk = acts_addr + (uint32_t)kb_e * ACTTS_CHUNK;
            if (waits_for_acts(e, n_kb)) ok = mbar_wait_warp(&acts_bar[kb_e], 0, p.err, DEV_ERR_WAIT_FULL);
            kb_e += kb_step;
            if (kb_e >= n_kb) kb_e -= n_kb;
            if (ok && e >= 2) {   // the group's accumulator was last used by entry e - 2
                ok = mbar_wait_warp(&d_free[g], (((uint32_t)e >> 1) - 1) & 1, p.err, DEV_ERR_WAIT_EMPTY);
            }
            // one descriptor per column block; a 16-column slice is 1024 bytes further = 64 in the address field (bits 0-13
            // of the low word, which cannot carry: shared-memory addresses stay below 256 KiB)
            const uint64_t bdesc = smem_desc(chunk, 512, 128), mdesc = smem_desc(chunk + TS_BMIN_OFF, 768, 128);
            const uint32_t b_lo = (uint32_t)bdesc, b_hi = (uint32_t)(bdesc >> 32);
#pragma unroll
            for (int h2 = 0; h2 < HALVES / 2; ++h2, ++uses) {
                const int h = 2 * h2 + (int)c;   // this warp's half; the unrolled code below needs it as a constant: see the switch on c
                if (ok) {
                    ok = mbar_wait_warp(&a_ready[2 * g + c], uses & 1, p.err, DEV_ERR_WAIT_FULL);
                }
                if (ok) {
                    fence_after_sync();
                    if (elect_one()) {
                        if (c == 0) issue_half<F, 0>(h2, d_buf, a_buf, b_lo, b_hi, IDESC_MAIN);
                        else issue_half<F, 1>(h2, d_buf, a_buf, b_lo, b_hi, IDESC_MAIN);
                        if (F::HAS_MIN && h == HALVES - 1)   // every half has stored its column of the min operand by now
                            mma_ts<false>(tmem + TM_DM + g * TM_DM_STRIDE, tmem + TM_AM + g * TM_AM_STRIDE, (uint32_t)mdesc, (uint32_t)(mdesc >> 32),
                                          IDESC_MIN);
                        mma_commit(&a_free[2 * g + c]);
                        if (h2 == HALVES / 2 - 1) mma_commit(&d_ready[g]);   // this warp's share of the entry; the barrier counts both warps
                    }
                    __syncwarp();
                }
            }
        }
        if (!ok) abort_flag = 1;
    } else if (warp < FR_UNPACK_WARPS) {
        // ------------------------------ unpacking warps ------------------------------
        // They read weights only (shared memory filled by the producer), so they never wait for the previous kernel.
        // A half is announced when the first 64 columns of the next one are already unpacked: its stores have long landed by then,
        // so that the wait for them costs nothing.
        const int g = warp >> 2, q4 = warp & 3;
        const int row = 32 * q4 + lane;
        const uint32_t tm_l = tmem + ((uint32_t)(32 * q4) << 16);
        const uint32_t a_buf = tm_l + TM_A + g * TM_A_STRIDE, am_buf = tm_l + TM_AM + g * TM_AM_STRIDE;
        // K padding of the group's min-term operand (sub-block pairs 4..7): written once, never touched again
        if (F::HAS_MIN) tmem_st4(am_buf + 4, 0u, 0u, 0u, 0u);
        bool ok = true;
        int stored = -1;   // half buffer that has been written but not announced
        auto announce = [&] {
            if (stored < 0) return;
            wait_st();
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&a_ready[2 * g + stored]);   // releases this warp's tensor-memory and side-buffer writes
            stored = -1;
        };
        uint32_t uses = 0;   // how often each half buffer of the group has been used
        int s = g;
        for (int e = g; e < n_it; e += 2) {
            uint64_t* fb = full_bar(full, e, s);
            if (!__all_sync(0xffffffffu, mbar_try_wait(fb, full_parity(e)))) {
                announce();
                ok = mbar_wait_warp(fb, full_parity(e), p.err, DEV_ERR_WAIT_FULL);
                if (!ok) break;
            }
            const uint8_t* st = ring + s * F::STAGE;
            uint32_t mins[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int h = 0; h < HALVES; ++h) {
                constexpr int LAST = HALVES - 1;
                const int hb = h & 1;
                uint32_t r[32];
                UnitScales us{0.f, 0.f};
                F::unpack(st, h, row, 0, r, mins[(2 * h) & 3], us);
                announce();
                if (uses == 1) trigger();   // nothing can be stored before an MMA has run, which is behind the dependency wait
                if (uses > 0) {   // the half buffer was last read by the MMAs of the group's half before the last
                    ok = mbar_wait_warp_inline(&a_free[2 * g + hb], (uses - 1) & 1, p.err, DEV_ERR_WAIT_FULL);
                    if (!ok) break;
                    fence_after_sync();
                }
                F::store(a_buf, h, 0, r);
                if (h == 0) scl[(e & 3) * TILE_R + row] = make_float2(us.d, us.dmin);
                F::unpack(st, h, row, 1, r, mins[(2 * h + 1) & 3], us);
                F::store(a_buf, h, 1, r);
                if (h == LAST) {
                    // The min operand is read by the entry's last MMA, so it may only be replaced once the previous
                    // entry's last half has completed - which this half's wait has just established.
                    if (F::HAS_MIN) tmem_st4(am_buf, mins[0], mins[1], mins[2], mins[3]);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&empty[s]);
                }
                stored = hb;
                if (hb == 1) ++uses;
            }
            if (!ok) break;
            s = s + 2 >= STAGES ? s + 2 - STAGES : s + 2;
        }
        if (ok) announce();
        else abort_flag = 1;
        if (uses < 2) trigger();
    } else {
        // ------------------------------ draining warps ------------------------------
        wait_inputs();
        trigger();
        const int dtid = threadIdx.x - DRAIN_WARP0 * 32;   // 0..127 = weight row of the tile = tensor-memory lane
        if (dtid == 0 && n_it > 0) {
            // the activations (the previous kernel's output), in the order of their first use, one barrier each: the
            // first MMA waits for one chunk only.  Issued here rather than by the producer, whose first iterations are
            // busy priming the weight ring.
            if (p.late_mode == LATE_BEHIND) asm volatile("fence.proxy.async.global;" ::: "memory");   // the acquire above counts for bulk copies too
            for (int k = 0; k < n_kb; ++k) {
                mbar_arrive_expect_tx(&acts_bar[k], ACTTS_CHUNK);
                bulk_g2s(acts_res + k * ACTTS_CHUNK, p.acts + (uint64_t)(p.kb_map ? p.kb_map[kb0 + k] : kb0 + k) * ACTTS_CHUNK, ACTTS_CHUNK, &acts_bar[k]);
            }
        }
        {
            // per-token output scale; 8 threads per token add the sum-of-squares partials in a fixed tree
            const int tok = dtid >> 3, part = dtid & 7;
            float ss = 0.f;
            if (p.sumsq)
                for (int q = part; q < p.n_sumsq; q += 8) ss += p.sumsq[q * MAX_ROWS + tok];
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            if (part == 0) tok_scale[tok] = p.sumsq ? p.out_scale * (1.0f / sqrtf(ss / p.norm_k + p.eps)) : p.out_scale;
        }
        named_sync(1, DRAIN_WARPS * 32);
        const int row = dtid;
        const uint32_t tm_l = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
        uint64_t acc[MAX_ROWS / 2];   // pairs of tokens
#pragma unroll
        for (int j = 0; j < MAX_ROWS / 2; ++j) acc[j] = 0ull;
        bool ok = true;
        int kb_e = 0, tile = 0;   // e % n_kb and e / n_kb, kept by addition
        for (int e = 0; e < n_it && ok; ++e) {
            const uint32_t a = (uint32_t)e & 1u;
            ok = mbar_wait_warp(&d_ready[a], ((uint32_t)e >> 1) & 1, p.err, DEV_ERR_WAIT_FULL);
            if (!ok) break;
            fence_after_sync();
            const float2 sc = scl[(e & 3) * TILE_R + row];   // published before the a_ready arrival the MMAs waited for
            // columns 16 plane + token, one load of 32 at a time: two would not fit the registers
            uint64_t t[MAX_ROWS / 2], mn[MAX_ROWS / 2];
            {
                float v[32];
                tmem_ld32(tm_l + TM_D + a * TM_D_STRIDE, v);        // even MMA halves
                wait_ld();
#pragma unroll
                for (int j = 0; j < MAX_ROWS / 2; ++j) t[j] = add2(pack2(v[2 * j], v[2 * j + 1]), pack2(v[16 + 2 * j], v[17 + 2 * j]));
                tmem_ld32(tm_l + TM_D + a * TM_D_STRIDE + 32, v);   // odd MMA halves
                wait_ld();
#pragma unroll
                for (int j = 0; j < MAX_ROWS / 2; ++j) t[j] = add2(t[j], add2(pack2(v[2 * j], v[2 * j + 1]), pack2(v[16 + 2 * j], v[17 + 2 * j])));
                if (F::HAS_MIN) {   // three planes of sixteen tokens
                    tmem_ld32(tm_l + TM_DM + a * TM_DM_STRIDE, v);
                    wait_ld();
#pragma unroll
                    for (int j = 0; j < MAX_ROWS / 2; ++j) mn[j] = add2(pack2(v[2 * j], v[2 * j + 1]), pack2(v[16 + 2 * j], v[17 + 2 * j]));
                    float v2[16];
                    tmem_ld16(tm_l + TM_DM + a * TM_DM_STRIDE + 32, v2);
                    wait_ld();
#pragma unroll
                    for (int j = 0; j < MAX_ROWS / 2; ++j) mn[j] = add2(mn[j], pack2(v2[2 * j], v2[2 * j + 1]));
                }
            }
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&d_free[a]);   // the accumulator may be overwritten
            const uint64_t d2 = pack2(sc.x, sc.x), m2 = pack2(-sc.y, -sc.y);
#pragma unroll
            for (int j = 0; j < MAX_ROWS / 2; ++j) {
                acc[j] = fma2(d2, t[j], acc[j]);
                if (F::HAS_MIN) acc[j] = fma2(m2, mn[j], acc[j]);
            }
            if (++kb_e == n_kb) {   // the tile's last column block: write the partial result
                kb_e = 0;
                const int slot = c + tile * cps;
                ++tile;
                const uint32_t orow = (uint32_t)(p.tile_map ? p.tile_map[slot] : slot) * TILE_R + row;
                if (orow < p.n_out) {
                    float* dst = p.out + (uint64_t)sp * MAX_ROWS * p.ld_out + orow;
#pragma unroll
                    for (int j = 0; j < MAX_ROWS / 2; ++j) {
                        float lo, hi;
                        unpack2(acc[j], lo, hi);
                        dst[(uint64_t)(2 * j) * p.ld_out] = lo * tok_scale[2 * j];
                        dst[(uint64_t)(2 * j + 1) * p.ld_out] = hi * tok_scale[2 * j + 1];
                    }
                }
#pragma unroll
                for (int j = 0; j < MAX_ROWS / 2; ++j) acc[j] = 0ull;
            }
        }
        if (!ok) abort_flag = 1;
    }

    fence_before_sync();
    __syncthreads();
    if (abort_flag && threadIdx.x == 0) {
        // Error word already set.  Give every copy this CTA armed a bounded chance to land before
        // the shared memory is released.
        for (int s = 0; s < FULL_SETS * STAGES; ++s) {
            uint32_t spins = 0;
            while (!mbar_try_wait(&full[s], 0) && !mbar_try_wait(&full[s], 1) && ++spins < (1u << 16)) __nanosleep(100);
        }
        for (int k = 0; k < (n_it > 0 ? (n_kb < KC ? n_kb : KC) : 0); ++k) {
            uint32_t spins = 0;
            while (!mbar_try_wait(&acts_bar[k], 0) && ++spins < (1u << 16)) __nanosleep(100);
        }
    }
    __syncthreads();
    if (warp == MMA_WARP0) {
        fence_after_sync();
        tmem_free(tmem, TM_COLS);
    }
    if (p.late_mode == LATE_BEHIND) pdl_wait();   // this kernel's completion says that those before are complete too
}

template <int DT, int KC>
static dfl_status launch_t(cudaStream_t st, const Params& p, int grid, bool pdl) {
    static std::once_flag attr_once[16];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 16) {
        cudaError_t attr_err = cudaSuccess;
        std::call_once(attr_once[dev], [&] {
            attr_err = cudaFuncSetAttribute(gemm_ts_kernel<DT, KC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes<DT, KC>());
        });
        DFL_CUDA(attr_err);
    } else {
        DFL_CUDA(cudaFuncSetAttribute(gemm_ts_kernel<DT, KC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes<DT, KC>()));
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem_bytes<DT, KC>();
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    DFL_CUDA(cudaLaunchKernelEx(&cfg, gemm_ts_kernel<DT, KC>, p));
    count_launch();
    return DFL_OK;
}

static int ctas_per_split(int row_tiles, int splits) {
    int cps = sm_count() / splits;
    if (cps < 1) cps = 1;
    return cps < row_tiles ? cps : row_tiles;
}

}  // namespace ts

// Split count: every split must fit the resident activation window; beyond that, the count that
// minimises the longest CTA (rounds of row tiles x column blocks per split, plus a per-tile
// and a per-launch overhead measured in stage times).
int gemm_ts_choose_splits(const QMatrix& m) {
    const int tiles = m.row_tiles > 0 ? m.row_tiles : 1;
    return gemm_ts_choose_splits_multi(&tiles, 1, m.kblocks);
}
// CTAs per split of a launch over `row_tiles` row tiles (the least number of tiles a tile list must hold)
int gemm_ts_kc() { return ts::KC_MAX; }   // column blocks a CTA keeps resident
int gemm_ts_ctas_per_split(int row_tiles, int splits) { return ts::ctas_per_split(row_tiles, splits); }
// Several matrices that share their input and their partial buffer are launched one after the other
// with one common split count: minimise the sum of their longest-CTA times.
int gemm_ts_choose_splits_multi(const int* row_tiles, int n_mats, int kblocks) {
    const int s_min = (kblocks + ts::KC_MAX - 1) / ts::KC_MAX;
    int s_max = kblocks < 24 ? kblocks : 24;
    if (s_max < s_min) s_max = s_min;
    int best = s_min;
    double best_cost = 1e30;
    for (int s = s_min; s <= s_max; ++s) {
        double cost = 0.0;
        for (int i = 0; i < n_mats; ++i) {
            const int tiles = row_tiles[i] > 0 ? row_tiles[i] : 1;
            cost += 0.05 * s + 0.0054 * s * tiles;   // partial slices to write and to sum again
            const int cps = ts::ctas_per_split(tiles, s);
            const int rounds = (tiles + cps - 1) / cps;
            cost += rounds * ((double)((kblocks + s - 1) / s) + 0.25);
        }
        if (cost < best_cost) { best_cost = cost; best = s; }
    }
    return best;
}

dfl_status launch_gemm_ts(cudaStream_t st, const QMatrix& m, const uint8_t* acts, float* out, int splits, const GemmEpilogue& ep,
                          int* dev_err, bool pdl, uint32_t ld_out) {
    if (splits < 1 || splits > m.kblocks) return fail(DFL_ERR_BAD_ARG, "gemm: bad split count");
    if ((m.kblocks + splits - 1) / splits > ts::KC_MAX) return fail(DFL_ERR_BAD_ARG, "gemm: too few splits for the resident activation window");
    ts::Params p;
    p.w = m.tiles;
    p.acts = acts;
    p.out = out;
    p.sumsq = ep.sumsq;
    p.n_sumsq = ep.n_sumsq;
    p.norm_k = ep.norm_k;
    p.eps = ep.eps;
    p.out_scale = ep.out_scale;
    p.kblocks = m.kblocks;
    p.splits = splits;
    p.row_tiles = m.row_tiles;
    p.ctas_per_split = ts::ctas_per_split(m.row_tiles, splits);
    p.n_out = (uint32_t)m.n_out;
    p.ld_out = ld_out ? ld_out : (uint32_t)m.n_out;
    p.err = dev_err;
    p.tile_map = ep.tile_map;
    p.n_tiles = ep.n_tiles;
    p.kb_map = ep.kb_map;
    p.n_kb = ep.n_kb;
    p.late_mode = ep.trigger_late ? ts::LATE_FIRST : ep.behind_late ? ts::LATE_BEHIND : 0;
    p.late_word = ep.late.word;
    p.late_value = ep.late.value;
    if ((ep.behind_late && ep.trigger_late) || ((ep.behind_late || ep.trigger_late) && !ep.late.word)) return fail(DFL_ERR_BAD_ARG, "gemm: dependency options");
    int grid = p.ctas_per_split * splits;
    if (ep.kb_map && ep.dynamic_splits && grid < sm_count()) grid = sm_count();   // room for the geometry chosen on the device
    // Four resident column blocks leave room for a fourth ring slot of a 35 KB stage.  It pays where a CTA has more than three stages to fetch
    // (4096 -> 4096 -> 32000 matrix step, its head in Q6_K, 92.3 -> 89.5 us; 9B-class token 2546 -> 2534).  Where it has not, there is nothing to gain, and
    // the other form is the one that the launch behind may use too: the shared expert's down projection, one stage a CTA, ahead of the routed
    // experts' (token of the routed model 2972 us with four slots there, 2849 without; four rows 3647, 3579).
    const int blocks = (m.kblocks + splits - 1) / splits, rounds = (m.row_tiles + p.ctas_per_split - 1) / p.ctas_per_split;
    const bool four = !ep.kb_map && blocks <= 4 && rounds * blocks > 3;
    switch (m.dtype) {
        case DFL_Q4_K: return ts::launch_t<DFL_Q4_K, ts::KC_MAX>(st, p, grid, pdl);
        case DFL_Q5_K: return ts::launch_t<DFL_Q5_K, ts::KC_MAX>(st, p, grid, pdl);
        case DFL_Q6_K: return four ? ts::launch_t<DFL_Q6_K, 4>(st, p, grid, pdl) : ts::launch_t<DFL_Q6_K, ts::KC_MAX>(st, p, grid, pdl);
        case DFL_Q8_0: return four ? ts::launch_t<DFL_Q8_0, 4>(st, p, grid, pdl) : ts::launch_t<DFL_Q8_0, ts::KC_MAX>(st, p, grid, pdl);
        default: return fail(DFL_ERR_UNSUPPORTED, "gemm: weight dtype has no tensor-memory kernel");
    }
}

}  // namespace dfl
