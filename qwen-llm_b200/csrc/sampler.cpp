// Host-side sampler and DFlash accept-prefix decision (f64, version-1 semantics).
// Product implementation of crates/qwen-llm/src/sampling.rs (`Sampler::{new, at_draw, sample,
// diagnose, couple_deterministic_proposal, couple_sparse_proposal}` :340-790, `greedy_token`
// :1159-1181, candidate keys :1206-1235, radix order :1283-1339, weights / top-p / categorical
// :1370-1438, xoshiro256++ / SplitMix64 :1619-1670) and crates/qwen-llm/src/metal_dflash/accept.rs
// (`decide_dflash_accept_prefix` :76-183).  Acceptance runs on the host in the reference too.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstring>
#include <condition_variable>
#include <deque>
#include <pthread.h>
#include <mutex>
#include <system_error>
#include <thread>
#include <limits>
#include <string>
#include <vector>

#if defined(__x86_64__)
#include <immintrin.h>
#endif

#include "../../include/dflash_b200.h"

namespace dfl {
dfl_status fail(dfl_status st, const std::string& msg);
}
using dfl::fail;

namespace {

struct SplitMix64 {
    uint64_t s;
    uint64_t next() {
        s += 0x9e3779b97f4a7c15ull;
        uint64_t v = s;
        v = (v ^ (v >> 30)) * 0xbf58476d1ce4e5b9ull;
        v = (v ^ (v >> 27)) * 0x94d049bb133111ebull;
        return v ^ (v >> 31);
    }
};
inline uint64_t rotl(uint64_t x, int k) { return (x << k) | (x >> (64 - k)); }
struct Xoshiro {
    uint64_t st[4];
    void seed(uint64_t seed) {
        SplitMix64 sm{seed};
        for (auto& v : st) v = sm.next();
    }
    uint64_t next_u64() {
        const uint64_t result = rotl(st[0] + st[3], 23) + st[0];
        const uint64_t t = st[1] << 17;
        st[2] ^= st[0];
        st[3] ^= st[1];
        st[1] ^= st[2];
        st[0] ^= st[3];
        st[2] ^= t;
        st[3] = rotl(st[3], 45);
        return result;
    }
    double next_unit() { return (double)(next_u64() >> 11) / 9007199254740992.0; }
};

enum SErr { S_OK = 0, S_EMPTY, S_NAN, S_TOO_LARGE, S_NO_CANDIDATES, S_MEMORY, S_PROPOSAL_RANGE, S_PROPOSAL_WEIGHT, S_MISSING_PROPOSAL };

// ascending u32 order == descending f32 total order
inline uint32_t descending_bits(float f) {
    uint32_t b;
    std::memcpy(&b, &f, 4);
    return b ^ (~(uint32_t)((int32_t)b >> 31) & 0x7fffffffu);   // no branch on the sign: it is a coin toss
}
inline double key_logit(uint64_t key) {
    const uint32_t d = (uint32_t)(key >> 32), bits = d ^ (~(uint32_t)((int32_t)d >> 31) & 0x7fffffffu);
    float f;
    std::memcpy(&f, &bits, 4);
    return (double)f;
}
inline int32_t key_token(uint64_t key) { return (int32_t)(uint32_t)key; }

struct Buffers {
    std::vector<uint64_t> keys, scratch;
    std::vector<double> cumulative;
};

// Keys of a row from an order made elsewhere (the device): token order[i] is the i-th candidate.  The order is checked
// - every token in range, keys non-decreasing, which for a permutation is exactly "sorted, ties by ascending token"
// when equal keys also ascend in token - and refused (false) when it is not this row's order.
bool keys_from_order(const float* logits, uint64_t n, const uint32_t* order, uint64_t take, std::vector<uint64_t>& keys) {
    keys.resize(take);
    uint64_t prev = 0;
    for (uint64_t i = 0; i < take; ++i) {
        const uint32_t t = order[i];
        if (t >= n) return false;
        const uint64_t k = ((uint64_t)descending_bits(logits[t]) << 32) | t;
        if (i && k <= prev) return false;   // strictly increasing 64-bit keys: sorted by logit, then by token, no repeats
        keys[i] = k;
        prev = k;
    }
    return true;
}

// Orders candidate keys: whole row when top-k is off, else the top_k best.  Returns count or error.
SErr order_keys(const float* logits, uint64_t n, uint64_t top_k, Buffers& b, uint64_t* count, uint64_t* nan_token,
                const uint32_t* order = nullptr, bool* order_used = nullptr, const std::atomic<bool>* stop = nullptr) {
    auto stopped = [&] { return stop && stop->load(std::memory_order_relaxed); };   // nobody wants the result any more: any will do
    if (n == 0) return S_EMPTY;
    if (n > 0x7fffffffull) return S_TOO_LARGE;
    const bool full = top_k == 0 || top_k >= n;
    if (order) {
        for (uint64_t t = 0; t < n; ++t)
            if (std::isnan(logits[t])) { *nan_token = t; return S_NAN; }
        const uint64_t take = full ? n : top_k;
        // a prefix of a sorted permutation is the sorted top-k; for the whole row the strict increase over n keys in
        // [0, n) token range makes it a permutation
        if (keys_from_order(logits, n, order, take, b.keys)) {
            *count = take;
            if (order_used) *order_used = true;
            return S_OK;
        }
    }
    b.keys.resize(n);
    // keys in token order; the four byte histograms of the logit half are taken in the same pass
    uint32_t hist[4][256];
    if (full) std::memset(hist, 0, sizeof(hist));
    for (uint64_t t = 0; t < n; ++t) {
        if (std::isnan(logits[t])) { *nan_token = t; return S_NAN; }
        const uint32_t d = descending_bits(logits[t]);
        b.keys[t] = ((uint64_t)d << 32) | t;
        if (full) { ++hist[0][d & 255]; ++hist[1][(d >> 8) & 255]; ++hist[2][(d >> 16) & 255]; ++hist[3][d >> 24]; }
    }
    if (full) {
        // stable LSD radix over the logit half, one byte per pass (256 write streams stay in the first-level cache);
        // keys were built in token order, so equal logits keep ascending token order
        if (n >= 2) {
            b.scratch.resize(n);
            for (int digit = 0; digit < 4; ++digit) {
                const int shift = 32 + 8 * digit;
                uint32_t* h = hist[digit];
                if (h[(b.keys[0] >> shift) & 255] == n) continue;   // every key has the same byte here
                if (stopped()) break;
                uint32_t off = 0;
                for (int i = 0; i < 256; ++i) { const uint32_t c = h[i]; h[i] = off; off += c; }
                const uint64_t* src = b.keys.data();
                uint64_t* dst = b.scratch.data();
                for (uint64_t i = 0; i < n; ++i) dst[h[(src[i] >> shift) & 255]++] = src[i];
                b.keys.swap(b.scratch);
            }
        }
        *count = n;
    } else {
        std::nth_element(b.keys.begin(), b.keys.begin() + top_k, b.keys.end());
        std::sort(b.keys.begin(), b.keys.begin() + top_k);
        *count = top_k;
    }
    return S_OK;
}

// ---- bounds for the nucleus ------------------------------------------------------------------------------------
// exp(x) for x <= 0 to about 1e-12: x = n ln 2 + r, Taylor polynomial of degree 10 in |r| <= ln 2 / 2.  It only ever decides which
// tokens the exact computation has to look at, never a value that is returned.
constexpr double kLn2 = 0.6931471805599453, kLog2e = 1.4426950408889634;
constexpr int kDegree = 10;
constexpr double kInvFact[kDegree + 1] = {1.0, 1.0, 1.0 / 2, 1.0 / 6, 1.0 / 24, 1.0 / 120, 1.0 / 720, 1.0 / 5040, 1.0 / 40320, 1.0 / 362880, 1.0 / 3628800};
inline double exp_bound(double x) {
    if (!(x > -700.0)) return 0.0;
    const double n = std::nearbyint(x * kLog2e), r = x - n * kLn2;
    double p = kInvFact[kDegree];
    for (int i = kDegree - 1; i >= 0; --i) p = p * r + kInvFact[i];
    uint64_t b = (uint64_t)(int64_t)(n + 1023.0) << 52;
    double scale;
    std::memcpy(&scale, &b, 8);
    return p * scale;
}
// weights exp(l inv_t - shift) of a row summed by steps of 1/16 below the maximum in log weight (the last step takes the rest);
// two tables, so that neighbours of one step do not wait for each other
constexpr int kSteps = 1024;
constexpr double kPerUnit = 16.0;
constexpr double kNothing = -48.0;   // weights below e^-48 = 1.4e-21: 2^31 of them weigh 3e-12 of the largest, less than the bound on the sum
struct StepMass { double m[2][kSteps]; };
inline void add_mass(StepMass& sm, int table, double x) {
    const double below = -x * kPerUnit;
    sm.m[table][below < (double)(kSteps - 1) ? (below > 0.0 ? (int)below : 0) : kSteps - 1] += exp_bound(x);
}
void step_mass_plain(const float* l, uint64_t n, double inv_t, double shift, StepMass& sm) {
    for (uint64_t i = 0; i < n; ++i) add_mass(sm, (int)(i & 1), (double)l[i] * inv_t - shift);
}
// a row's largest logit; false if it holds a NaN
bool max_of_plain(const float* l, uint64_t n, float* mx) {
    float m = l[0];
    bool nan = false;
    for (uint64_t i = 0; i < n; ++i) { nan |= std::isnan(l[i]); m = l[i] > m ? l[i] : m; }
    *mx = m;
    return !nan;
}
// keys of the tokens with logits of at least thr, in token order (keys: n + 1 entries)
uint64_t collect_plain(const float* l, uint64_t n, float thr, uint64_t* keys) {
    uint64_t c = 0;
    for (uint64_t i = 0; i < n; ++i) {
        keys[c] = ((uint64_t)descending_bits(l[i]) << 32) | i;
        c += l[i] >= thr;
    }
    return c;
}
#if defined(__x86_64__)
#define DFL_AVX2 __attribute__((target("avx2,fma")))
DFL_AVX2 void step_mass_avx2(const float* l, uint64_t n, double inv_t, double shift, StepMass& sm) {
    const __m256d it = _mm256_set1_pd(inv_t), sh = _mm256_set1_pd(shift), l2e = _mm256_set1_pd(kLog2e), ln2 = _mm256_set1_pd(kLn2),
                  floor_x = _mm256_set1_pd(-700.0), per_unit = _mm256_set1_pd(-kPerUnit);
    const __m256d last_step = _mm256_set1_pd((double)(kSteps - 1)), zero = _mm256_setzero_pd(), nothing = _mm256_set1_pd(kNothing);
    alignas(32) double w[16];
    alignas(16) int32_t step[16];
    uint64_t i = 0;
    for (; i + 16 <= n; i += 16) {
        __m256d x[4], k[4], r[4], p[4];
        for (int j = 0; j < 4; ++j) x[j] = _mm256_fmsub_pd(_mm256_cvtps_pd(_mm_loadu_ps(l + i + 4 * j)), it, sh);
        const __m256d top = _mm256_max_pd(_mm256_max_pd(x[0], x[1]), _mm256_max_pd(x[2], x[3]));
        if (_mm256_movemask_pd(_mm256_cmp_pd(top, nothing, _CMP_GT_OQ)) == 0) continue;
        for (int j = 0; j < 4; ++j) k[j] = _mm256_round_pd(_mm256_mul_pd(x[j], l2e), _MM_FROUND_TO_NEAREST_INT | _MM_FROUND_NO_EXC);
        for (int j = 0; j < 4; ++j) r[j] = _mm256_fnmadd_pd(k[j], ln2, x[j]);
        for (int j = 0; j < 4; ++j) p[j] = _mm256_set1_pd(kInvFact[kDegree]);
        for (int d = kDegree - 1; d >= 0; --d)
            for (int j = 0; j < 4; ++j) p[j] = _mm256_fmadd_pd(p[j], r[j], _mm256_set1_pd(kInvFact[d]));
        for (int j = 0; j < 4; ++j) {
            const __m256i e = _mm256_slli_epi64(_mm256_cvtepi32_epi64(_mm_add_epi32(_mm256_cvtpd_epi32(k[j]), _mm_set1_epi32(1023))), 52);
            const __m256d v = _mm256_mul_pd(p[j], _mm256_castsi256_pd(e));
            _mm256_store_pd(w + 4 * j, _mm256_and_pd(v, _mm256_cmp_pd(x[j], floor_x, _CMP_GT_OQ)));
            _mm_store_si128((__m128i*)(step + 4 * j), _mm256_cvttpd_epi32(_mm256_max_pd(_mm256_min_pd(_mm256_mul_pd(x[j], per_unit), last_step), zero)));
        }
        for (int j = 0; j < 16; ++j) sm.m[j & 1][step[j]] += w[j];
    }
    for (; i < n; ++i) add_mass(sm, (int)(i & 1), (double)l[i] * inv_t - shift);
}
#define DFL_AVX512 __attribute__((target("avx512f,avx512dq,avx2,fma")))
DFL_AVX512 void step_mass_avx512(const float* l, uint64_t n, double inv_t, double shift, StepMass& sm) {
    const __m512d it = _mm512_set1_pd(inv_t), sh = _mm512_set1_pd(shift), l2e = _mm512_set1_pd(kLog2e), ln2 = _mm512_set1_pd(kLn2),
                  floor_x = _mm512_set1_pd(-700.0), per_unit = _mm512_set1_pd(-kPerUnit), nothing = _mm512_set1_pd(kNothing);
    const __m512d last_step = _mm512_set1_pd((double)(kSteps - 1)), zero = _mm512_setzero_pd();
    alignas(64) double w[32];
    alignas(32) int32_t step[32];
    uint64_t i = 0;
    for (; i + 32 <= n; i += 32) {
        __m512d x[4], k[4], r[4], p[4];
        for (int j = 0; j < 4; ++j) x[j] = _mm512_fmsub_pd(_mm512_cvtps_pd(_mm256_loadu_ps(l + i + 8 * j)), it, sh);
        const __m512d top = _mm512_max_pd(_mm512_max_pd(x[0], x[1]), _mm512_max_pd(x[2], x[3]));
        if (_mm512_cmp_pd_mask(top, nothing, _CMP_GT_OQ) == 0) continue;
        for (int j = 0; j < 4; ++j) k[j] = _mm512_roundscale_pd(_mm512_mul_pd(x[j], l2e), _MM_FROUND_TO_NEAREST_INT | _MM_FROUND_NO_EXC);
        for (int j = 0; j < 4; ++j) r[j] = _mm512_fnmadd_pd(k[j], ln2, x[j]);
        for (int j = 0; j < 4; ++j) p[j] = _mm512_set1_pd(kInvFact[kDegree]);
        for (int d = kDegree - 1; d >= 0; --d)
            for (int j = 0; j < 4; ++j) p[j] = _mm512_fmadd_pd(p[j], r[j], _mm512_set1_pd(kInvFact[d]));
        for (int j = 0; j < 4; ++j) {
            _mm512_store_pd(w + 8 * j, _mm512_maskz_scalef_pd(_mm512_cmp_pd_mask(x[j], floor_x, _CMP_GT_OQ), p[j], k[j]));
            _mm256_store_si256((__m256i*)(step + 8 * j),
                               _mm512_cvttpd_epi32(_mm512_max_pd(_mm512_min_pd(_mm512_mul_pd(x[j], per_unit), last_step), zero)));
        }
        for (int j = 0; j < 32; ++j) sm.m[j & 1][step[j]] += w[j];
    }
    for (; i < n; ++i) add_mass(sm, (int)(i & 1), (double)l[i] * inv_t - shift);
}
DFL_AVX512 uint64_t collect_avx512(const float* l, uint64_t n, float thr, uint64_t* keys) {
    const __m512 t = _mm512_set1_ps(thr);
    const __m512i magnitude = _mm512_set1_epi32(0x7fffffff), lanes = _mm512_set_epi64(7, 6, 5, 4, 3, 2, 1, 0);
    uint64_t c = 0, i = 0;
    for (; i + 16 <= n; i += 16) {
        const __m512 v = _mm512_loadu_ps(l + i);
        const unsigned m = _mm512_cmp_ps_mask(v, t, _CMP_GE_OQ);
        if (!m) continue;
        const __m512i b = _mm512_castps_si512(v), d = _mm512_xor_si512(b, _mm512_andnot_si512(_mm512_srai_epi32(b, 31), magnitude));
        const __m512i at = _mm512_add_epi64(_mm512_set1_epi64((long long)i), lanes);
        const __m512i k0 = _mm512_or_si512(_mm512_slli_epi64(_mm512_cvtepu32_epi64(_mm512_castsi512_si256(d)), 32), at);
        const __m512i k1 = _mm512_or_si512(_mm512_slli_epi64(_mm512_cvtepu32_epi64(_mm512_extracti64x4_epi64(d, 1)), 32),
                                           _mm512_add_epi64(at, _mm512_set1_epi64(8)));
        _mm512_mask_compressstoreu_epi64(keys + c, (__mmask8)(m & 255u), k0);
        c += (uint64_t)__builtin_popcount(m & 255u);
        _mm512_mask_compressstoreu_epi64(keys + c, (__mmask8)(m >> 8), k1);
        c += (uint64_t)__builtin_popcount(m >> 8);
    }
    for (; i < n; ++i)
        if (l[i] >= thr) keys[c++] = ((uint64_t)descending_bits(l[i]) << 32) | i;
    return c;
}
DFL_AVX2 bool max_of_avx2(const float* l, uint64_t n, float* mx) {
    if (n < 16) return max_of_plain(l, n, mx);
    __m256 m0 = _mm256_loadu_ps(l), m1 = _mm256_loadu_ps(l + 8), bad = _mm256_setzero_ps();
    uint64_t i = 0;
    for (; i + 16 <= n; i += 16) {
        const __m256 a = _mm256_loadu_ps(l + i), b = _mm256_loadu_ps(l + i + 8);
        bad = _mm256_or_ps(bad, _mm256_or_ps(_mm256_cmp_ps(a, a, _CMP_UNORD_Q), _mm256_cmp_ps(b, b, _CMP_UNORD_Q)));
        m0 = _mm256_max_ps(m0, a);
        m1 = _mm256_max_ps(m1, b);
    }
    float t[8];
    _mm256_storeu_ps(t, _mm256_max_ps(m0, m1));
    float m = t[0];
    bool nan = _mm256_movemask_ps(bad) != 0;
    for (int j = 1; j < 8; ++j) m = t[j] > m ? t[j] : m;
    for (; i < n; ++i) { nan |= std::isnan(l[i]); m = l[i] > m ? l[i] : m; }
    *mx = m;
    return !nan;
}
DFL_AVX2 uint64_t collect_avx2(const float* l, uint64_t n, float thr, uint64_t* keys) {
    const __m256 t = _mm256_set1_ps(thr);
    uint64_t c = 0, i = 0;
    for (; i + 8 <= n; i += 8) {
        unsigned m = (unsigned)_mm256_movemask_ps(_mm256_cmp_ps(_mm256_loadu_ps(l + i), t, _CMP_GE_OQ));
        if (!m) continue;
        for (uint64_t j = i; j < i + 8; ++j, m >>= 1) {   // all eight written, the count moves past those that belong
            keys[c] = ((uint64_t)descending_bits(l[j]) << 32) | j;
            c += m & 1u;
        }
    }
    for (; i < n; ++i)
        if (l[i] >= thr) keys[c++] = ((uint64_t)descending_bits(l[i]) << 32) | i;
    return c;
}
inline bool have_avx2() {
    static const bool yes = __builtin_cpu_supports("avx2") && __builtin_cpu_supports("fma");
    return yes;
}
inline bool have_avx512() {
    static const bool yes = __builtin_cpu_supports("avx512f") && __builtin_cpu_supports("avx512dq");
    return yes;
}
inline void step_mass(const float* l, uint64_t n, double inv_t, double shift, StepMass& sm) {
    have_avx512() ? step_mass_avx512(l, n, inv_t, shift, sm) : have_avx2() ? step_mass_avx2(l, n, inv_t, shift, sm) : step_mass_plain(l, n, inv_t, shift, sm);
}
inline bool max_of(const float* l, uint64_t n, float* mx) { return have_avx2() ? max_of_avx2(l, n, mx) : max_of_plain(l, n, mx); }
inline uint64_t collect(const float* l, uint64_t n, float thr, uint64_t* keys) {
    return have_avx512() ? collect_avx512(l, n, thr, keys) : have_avx2() ? collect_avx2(l, n, thr, keys) : collect_plain(l, n, thr, keys);
}
#else
inline void step_mass(const float* l, uint64_t n, double inv_t, double shift, StepMass& sm) { step_mass_plain(l, n, inv_t, shift, sm); }
inline bool max_of(const float* l, uint64_t n, float* mx) { return max_of_plain(l, n, mx); }
inline uint64_t collect(const float* l, uint64_t n, float thr, uint64_t* keys) { return collect_plain(l, n, thr, keys); }
#endif
// keys in ascending order; they arrive in token order, so long lists take a stable radix over the logit half, 11 bits a pass, as
// many passes as the spread of the logits has bits
void sort_keys(std::vector<uint64_t>& keys, std::vector<uint64_t>& scratch, uint64_t n) {
    if (n < 2048) { std::sort(keys.begin(), keys.begin() + (ptrdiff_t)n); return; }
    uint32_t lo = 0xffffffffu, hi = 0;
    for (uint64_t i = 0; i < n; ++i) { const uint32_t d = (uint32_t)(keys[i] >> 32); lo = std::min(lo, d); hi = std::max(hi, d); }
    int bits = 0;
    while (bits < 32 && ((hi - lo) >> bits) != 0) ++bits;
    const int passes = (bits + 10) / 11;
    const uint64_t base = (uint64_t)lo << 32;
    uint32_t hist[3][2048];
    std::memset(hist, 0, sizeof(uint32_t) * 2048 * passes);
    for (uint64_t i = 0; i < n; ++i)
        for (int p = 0; p < passes; ++p) ++hist[p][((keys[i] - base) >> (32 + 11 * p)) & 2047];
    if (scratch.size() < keys.size()) scratch.resize(keys.size());   // the two change places: a short one would have to grow again
    for (int p = 0; p < passes; ++p) {
        uint32_t off = 0, *h = hist[p];
        for (int i = 0; i < 2048; ++i) { const uint32_t c = h[i]; h[i] = off; off += c; }
        const int shift = 32 + 11 * p;
        for (uint64_t i = 0; i < n; ++i) scratch[h[((keys[i] - base) >> shift) & 2047]++] = keys[i];
        keys.swap(scratch);
    }
}

// ---- threads that build rows ahead ------------------------------------------------------------------------------
// One crew for all samplers of the process.  A sampler offers the rows of the block it is deciding; a free thread takes the next row of a
// block that may have one more helper.  At most as many threads as the host runs at once, started when a block
// finds none idle; one that has had nothing to do for two seconds ends.  (Threads of each sampler's own: 32 samplers held 224
// idle threads on eight cores, and a limit set after the first block came too late.)
class Crew {
public:
    struct Block {   // guarded by the crew's mutex, except `stop`
        uint32_t next = 0, limit = 0;        // rows [next, limit) may be taken
        uint32_t running = 0, helpers = 0;   // threads at work on it, and the most there may be
        std::condition_variable idle;
        std::atomic<bool> stop{false};       // the block has been decided: rows still being built are not wanted any more
        void* owner = nullptr;
        void (*build)(void* owner, uint32_t row) = nullptr;   // must not throw
    };
    static Crew& get() {
        static std::once_flag once;
        std::call_once(once, [] {
            instance() = new Crew();
            pthread_atfork(nullptr, nullptr, [] { instance() = new Crew(); });   // a child has none of its parent's threads
        });
        return *instance();
    }
    void begin(Block& b) {
        std::lock_guard<std::mutex> lock(mu);
        b.next = b.limit = b.running = 0;
        b.stop.store(false, std::memory_order_relaxed);
        blocks.push_back(&b);
    }
    // rows before `limit` may be built ahead
    void allow(Block& b, uint32_t limit) {
        std::lock_guard<std::mutex> lock(mu);
        if (limit <= b.limit) return;
        b.limit = limit;
        const uint32_t wanted = std::min(b.helpers > b.running ? b.helpers - b.running : 0, b.limit > b.next ? b.limit - b.next : 0);
        const uint32_t most = std::max(2u, std::thread::hardware_concurrency());
        try {
            for (; n_idle < wanted && threads.size() - ended.size() < most; ++n_idle) {
                ended.reserve(threads.size() + 1);
                threads.emplace_back([this] { main(); });
            }
        } catch (...) {   // no more threads to be had: the caller builds what they do not
        }
        for (const std::thread::id id : ended) {
            auto it = std::find_if(threads.begin(), threads.end(), [&](const std::thread& t) { return t.get_id() == id; });
            it->join();
            threads.erase(it);
        }
        ended.clear();
        for (uint32_t i = 0; i < wanted; ++i) work.notify_one();
    }
    // whether nobody has taken the row; it is the caller's then
    bool claim(Block& b, uint32_t row) {
        std::lock_guard<std::mutex> lock(mu);
        if (row < b.next) return false;
        b.next = row + 1;
        return true;
    }
    // when it returns no thread works on the block, and none will
    void end(Block& b) {
        b.stop.store(true, std::memory_order_relaxed);
        std::unique_lock<std::mutex> lock(mu);
        b.limit = 0;
        blocks.erase(std::remove(blocks.begin(), blocks.end(), &b), blocks.end());
        b.idle.wait(lock, [&] { return b.running == 0; });
    }
    // before the code of the threads goes away (process exit, library unloaded)
    static void shut_down() {
        Crew* c = instance();
        if (!c) return;
        std::vector<std::thread> all;
        {
            std::lock_guard<std::mutex> lock(c->mu);
            c->quit = true;
            all.swap(c->threads);
            c->ended.clear();
        }
        c->work.notify_all();
        for (std::thread& t : all) t.join();
    }

private:
    static Crew*& instance() { static Crew* c = nullptr; return c; }   // never destroyed
    Block* pick() {
        for (size_t i = 0; i < blocks.size(); ++i) {
            Block* b = blocks[i];
            if (b->next >= b->limit || b->running >= b->helpers) continue;
            std::rotate(blocks.begin(), blocks.begin() + (ptrdiff_t)i + 1, blocks.end());   // blocks take turns
            return b;
        }
        return nullptr;
    }
    void main() {   // counted as idle by whoever started it
        std::unique_lock<std::mutex> lock(mu);
        for (bool rested = false;;) {
            Block* b = quit ? nullptr : pick();
            if (!b) {
                if (quit || rested) break;
                rested = work.wait_for(lock, std::chrono::seconds(2)) == std::cv_status::timeout;
                continue;
            }
            rested = false;
            const uint32_t row = b->next++;
            ++b->running;
            --n_idle;
            lock.unlock();
            b->build(b->owner, row);
            lock.lock();
            ++n_idle;
            if (--b->running == 0) b->idle.notify_all();
        }
        --n_idle;
        if (!quit) ended.push_back(std::this_thread::get_id());   // joined by the next block that asks for threads; the space is reserved
    }
    std::mutex mu;
    std::condition_variable work;
    std::vector<Block*> blocks;
    std::vector<std::thread> threads;
    std::vector<std::thread::id> ended;
    uint32_t n_idle = 0;
    bool quit = false;
};
__attribute__((destructor)) void crew_shut_down() { Crew::shut_down(); }

struct Dist {
    std::vector<int32_t> tokens;
    std::vector<double> weights;
    double total = 0;
    int32_t sampled = 0;
    uint64_t index = 0;
};

}  // namespace

struct dfl_sampler {
    dfl_sampling_config cfg;
    Xoshiro rng;
    uint64_t draws = 0;
    Buffers buf;
    // Distributions of a block's rows built ahead of the sequential accept loop: building a row's distribution draws nothing from
    // the generator, so only the picks have to stay in row order.  The crew takes rows in order up to a
    // limit that moves with the loop (the first six cover a typical accepted prefix), so a block rejected early does
    // not pay for all of its rows; a row that no thread has taken yet when the loop reaches it is built by the loop's own
    // thread, so nothing waits for a thread to wake.  The threads outlive the block: starting five of them a
    // block cost 0.2 - 0.3 ms, as much as the rows themselves when each has a clear favourite.
    struct Prepared {
        const float* logits = nullptr;
        Dist dist;
        SErr err = S_OK;
        uint64_t nan_token = 0;
        std::atomic<bool> done{false};
        Buffers buf;
    };
    // rows whose order was made elsewhere (dfl_sampler_set_row_order)
    const float* ord_logits = nullptr;
    const uint32_t* ord_base = nullptr;
    uint32_t ord_rows = 0;
    uint64_t ord_vocab = 0;
    mutable std::atomic<uint64_t> ord_used{0};   // rows that took a registered order (rows are built on several threads)
    uint32_t workers = 0;   // threads that build a block's rows ahead of the accept loop: 0 = the host's concurrency, 1 = none
    const uint32_t* order_for(const float* logits, uint64_t n) const {
        if (!ord_logits || n != ord_vocab || logits < ord_logits) return nullptr;
        const uint64_t off = (uint64_t)(logits - ord_logits);
        if (off % ord_vocab || off / ord_vocab >= ord_rows) return nullptr;
        return ord_base + off;
    }
    std::deque<Prepared> prepared;   // rows stay where they are when it grows
    const float* block_logits = nullptr;
    uint64_t block_vocab = 0;
    uint32_t block_rows = 0;
    Crew::Block ahead;

    bool nucleus_path() const { return cfg.top_k == 0 && !(cfg.min_p > 0.0f) && cfg.top_p < 1.0f; }
    void build_row(uint32_t r) {
        Prepared& p = prepared[r];
        try {
            p.err = distribution(p.logits, block_vocab, p.dist, &p.nan_token, p.buf, &ahead.stop);
        } catch (...) {   // on a thread of the crew nobody could catch it
            p.err = S_MEMORY;
        }
        p.done.store(true, std::memory_order_release);
    }
    void prepare_rows(const float* logits, uint32_t n_rows, uint64_t vocab) {
        block_logits = nullptr;
        block_rows = 0;
        if (cfg.temperature == 0.0f || n_rows < 2 || vocab < 4096 || worker_limit() < 2) return;
        while (prepared.size() < n_rows) prepared.emplace_back();
        for (uint32_t r = 0; r < n_rows; ++r) {
            prepared[r].logits = logits + (uint64_t)r * vocab;
            prepared[r].done.store(false, std::memory_order_relaxed);
        }
        ahead.owner = this;
        ahead.build = [](void* self, uint32_t r) { static_cast<dfl_sampler*>(self)->build_row(r); };
        ahead.helpers = std::min(worker_limit() - 1, 10u);   // the loop's own thread is one of the workers
        Crew::get().begin(ahead);
        block_vocab = vocab;
        block_rows = n_rows;
        block_logits = logits;
        Crew::get().allow(ahead, std::min(6u, n_rows));
    }
    // no thread reads the block's logits any more
    void end_block() {
        if (block_logits) Crew::get().end(ahead);
        block_logits = nullptr;
        block_rows = 0;
    }
    unsigned worker_limit() const { return workers ? workers : std::thread::hardware_concurrency(); }
    // the prepared distribution of this row, if it belongs to the current block (moved out: a row is consumed once)
    bool take_prepared(const float* logits, Dist& d, SErr* e, uint64_t* nan_token) {
        if (!block_logits || logits < block_logits) return false;
        const uint64_t off = (uint64_t)(logits - block_logits);
        if (off % block_vocab || off / block_vocab >= block_rows) return false;
        const uint32_t r = (uint32_t)(off / block_vocab);
        Prepared& p = prepared[r];
        if (p.logits != logits) return false;
        const bool mine = Crew::get().claim(ahead, r);
        // Where rows take the nucleus path they are cheap and stop quickly, so the limit keeps ahead of the loop; the ordered path's rows,
        // milliseconds each, are only added when the loop has used up those it has.
        if (nucleus_path() ? r >= 4 : r >= 6) Crew::get().allow(ahead, std::min(nucleus_path() ? r + 8 : (r + 4) / 10 * 10 + 6, block_rows));
        if (mine) build_row(r);
        while (!p.done.load(std::memory_order_acquire)) std::this_thread::yield();
        *e = p.err;
        *nan_token = p.nan_token;
        std::swap(d, p.dist);
        p.logits = nullptr;
        return true;
    }

    // The filtered categorical distribution of sampler-v1 (diagnose_candidates, sampling.rs:1541-1614).
    SErr distribution(const float* logits, uint64_t n, Dist& d, uint64_t* nan_token) {
        SErr e;
        if (take_prepared(logits, d, &e, nan_token)) return e;
        return distribution(logits, n, d, nan_token, buf);
    }
    // The nucleus without ordering the row.  The general path orders all n tokens and takes exp of each, although what leaves it
    // is the short sorted prefix whose weights reach top_p of the total; the total itself only enters one comparison.  So: the
    // total to EPS and its split by steps of log weight in one vectorised pass, the tokens of the steps that hold the share, then
    // ordering, exact weights and exact running sum over those alone.  Where the running sum comes within EPS of the target
    // the general path decides: tokens, weights, total and draws are its own, bit for bit.  Below 1024 tokens the step tables
    // cost more than ordering.  16 rows of 151 936, four accepted: 4.4 -> 1.2 ms; one row with 44 600 in its nucleus 4.3 -> 2.6 ms.
    // `stop` (optional): return at the next step with nothing of use.
    bool nucleus(const float* logits, uint64_t n, Dist& d, Buffers& buf, const std::atomic<bool>* stop) const {
        auto stopped = [&] { return stop && stop->load(std::memory_order_relaxed); };
        if (!nucleus_path() || n < 1024 || n > 0x7fffffffull) return false;
        float mx;
        if (!max_of(logits, n, &mx) || !std::isfinite(mx)) return false;
        const double t = (double)cfg.temperature, inv_t = 1.0 / t, max_logit = (double)mx / t;
        StepMass sm{};
        for (uint64_t off = 0; off < n; off += 16384) {
            if (stopped()) return true;
            step_mass(logits + off, std::min<uint64_t>(16384, n - off), inv_t, (double)mx * inv_t, sm);
        }
        double total = 0.0;
        for (int b = 0; b < kSteps; ++b) total += sm.m[0][b] + sm.m[1][b];
        if (!std::isfinite(max_logit) || !std::isfinite(total) || total < 0.5) return false;
        // what separates this sum from one taken in sorted order: the polynomial, n roundings, and those of l / t
        const double EPS = 1e-11 + 4e-16 * (double)n + 1e-15 * (std::fabs(max_logit) + 700.0);
        const double share = (double)cfg.top_p;
        const double lo = total * (1.0 - EPS) * share, hi = total * (1.0 + EPS) * share;
        double mass = 0.0;
        int b = 0;
        for (; b < kSteps - 1; ++b) {
            mass += sm.m[0][b] + sm.m[1][b];
            if (mass > hi) break;
        }
        if (b == kSteps - 1) return false;
        // the smallest logit of steps 0..b, less what rounding can move it
        const double l_low = t * (max_logit - (double)(b + 1) / kPerUnit);
        const float thr = std::nextafterf((float)(l_low - 1e-6 * (std::fabs(l_low) + std::fabs((double)mx))), -std::numeric_limits<float>::infinity());
        if (!std::isfinite(thr)) return false;
        if (buf.keys.size() < n + 1) buf.keys.resize(n + 1);
        const uint64_t len = collect(logits, n, thr, buf.keys.data());
        if (len == 0) return false;
        if (stopped()) return true;
        sort_keys(buf.keys, buf.scratch, len);
        const uint64_t* keys = buf.keys.data();
        d.weights.resize(len);
        double cum = 0.0, *w = d.weights.data();
        for (uint64_t first = 0; first < len; first += 1024) {
            if (stopped()) return true;
            const uint64_t last = std::min<uint64_t>(len, first + 1024);
            for (uint64_t i = first; i < last; ++i) w[i] = key_logit(keys[i]) / t - max_logit;
            for (uint64_t i = first; i < last; ++i) w[i] = std::exp(w[i]);
            for (uint64_t i = first; i < last; ++i) {
                cum += w[i];
                if (cum < lo) continue;
                if (cum < hi) return false;   // too close to call with a bound on the total
                d.weights.resize(i + 1);
                d.tokens.resize(i + 1);
                for (uint64_t j = 0; j <= i; ++j) d.tokens[j] = key_token(keys[j]);
                d.total = cum;
                return true;
            }
        }
        return false;
    }
    SErr distribution(const float* logits, uint64_t n, Dist& d, uint64_t* nan_token, Buffers& buf, const std::atomic<bool>* stop = nullptr) const {
        if (!order_for(logits, n) && nucleus(logits, n, d, buf, stop)) return S_OK;
        uint64_t len = 0;
        bool order_used = false;
        SErr e = order_keys(logits, n, cfg.top_k, buf, &len, nan_token, order_for(logits, n), &order_used, stop);
        if (order_used) ord_used.fetch_add(1, std::memory_order_relaxed);
        if (e != S_OK) return e;
        const uint64_t* keys = buf.keys.data();
        if (cfg.min_p > 0.0f) {
            const double max_logit = key_logit(keys[0]);
            if (std::isfinite(max_logit)) {
                const double threshold = max_logit + std::log((double)cfg.min_p);
                uint64_t keep = 0;
                while (keep < len && key_logit(keys[keep]) >= threshold) ++keep;  // monotone along the order
                len = keep;
            }
        }
        if (len == 0) return S_NO_CANDIDATES;
        const double inf = std::numeric_limits<double>::infinity();
        if (key_logit(keys[0]) == inf) {
            uint64_t keep = 0;
            while (keep < len && key_logit(keys[keep]) == inf) ++keep;
            len = keep;
        }
        d.tokens.resize(len);
        d.weights.resize(len);
        const double t = (double)cfg.temperature;
        if (key_logit(keys[0]) == inf) {
            for (uint64_t i = 0; i < len; ++i) d.weights[i] = 1.0;
        } else {
            const double max_logit = key_logit(keys[0]) / t;
            if (max_logit == -inf) return S_NO_CANDIDATES;
            bool finite = true;
            double* w = d.weights.data();
            for (uint64_t i = 0; i < len; ++i) w[i] = key_logit(keys[i]) / t - max_logit;   // vectorisable part first
            for (uint64_t first = 0; first < len; first += 8192) {
                if (stop && stop->load(std::memory_order_relaxed)) return S_OK;
                const uint64_t last = std::min<uint64_t>(len, first + 8192);
                for (uint64_t i = first; i < last; ++i) {
                    w[i] = std::exp(w[i]);
                    finite &= std::isfinite(w[i]);
                }
            }
            if (!finite) return S_NO_CANDIDATES;
        }
        for (uint64_t i = 0; i < len; ++i) d.tokens[i] = key_token(keys[i]);
        if (cfg.top_p < 1.0f) {
            double total = 0.0;
            for (uint64_t i = 0; i < len; ++i) total += d.weights[i];
            const double target = total * (double)cfg.top_p;
            double cum = 0.0;
            uint64_t keep = 0;
            for (uint64_t i = 0; i < len; ++i) {
                cum += d.weights[i];
                ++keep;
                if (cum >= target) break;
            }
            keep = std::max<uint64_t>(keep, 1);
            d.tokens.resize(keep);
            d.weights.resize(keep);
        }
        double total = 0.0;
        for (double w : d.weights) total += w;
        if (!(std::isfinite(total) && total > 0.0)) return S_NO_CANDIDATES;
        d.total = total;
        return S_OK;
    }

    static void pick(Dist& d, double uniform) {
        const double target = uniform * d.total;
        double cum = 0.0;
        uint64_t idx = d.weights.size() - 1;
        for (uint64_t i = 0; i < d.weights.size(); ++i) {
            cum += d.weights[i];
            if (target < cum) { idx = i; break; }
        }
        d.index = idx;
        d.sampled = d.tokens[idx];
    }

    static SErr greedy(const float* logits, uint64_t n, int32_t* tok, uint64_t* nan_token) {
        if (n == 0) return S_EMPTY;
        if (n > 0x7fffffffull) return S_TOO_LARGE;
        if (std::isnan(logits[0])) { *nan_token = 0; return S_NAN; }
        uint64_t best = 0;
        uint32_t best_key = descending_bits(logits[0]);
        for (uint64_t t = 1; t < n; ++t) {
            if (std::isnan(logits[t])) { *nan_token = t; return S_NAN; }
            const uint32_t k = descending_bits(logits[t]);
            if (k < best_key) { best = t; best_key = k; }  // strictly greater in total order: lowest index wins ties
        }
        *tok = (int32_t)best;
        return S_OK;
    }

    // Sampler::diagnose with uniform 0 (used by the sparse coupling)
    SErr diagnose0(const float* logits, uint64_t n, Dist& d, uint64_t* nan_token) {
        if (cfg.temperature == 0.0f) {
            int32_t tok;
            SErr e = greedy(logits, n, &tok, nan_token);
            if (e != S_OK) return e;
            d.tokens.assign(1, tok);
            d.weights.assign(1, 1.0);
            d.total = 1.0;
            d.sampled = tok;
            d.index = 0;
            return S_OK;
        }
        SErr e = distribution(logits, n, d, nan_token);
        if (e != S_OK) return e;
        pick(d, 0.0);
        return S_OK;
    }

    SErr sample(const float* logits, uint64_t n, int32_t* tok, uint64_t* idx, uint64_t* nan_token) {
        if (cfg.temperature == 0.0f) {
            *idx = 0;
            return greedy(logits, n, tok, nan_token);
        }
        Dist d;
        SErr e = distribution(logits, n, d, nan_token);
        if (e != S_OK) return e;
        ++draws;
        pick(d, rng.next_unit());
        *tok = d.sampled;
        *idx = d.index;
        return S_OK;
    }

    // returns accepted flag; on rejection *correction is the residual draw (sampling.rs:708-790)
    SErr couple_sparse(const float* logits, uint64_t n, int32_t ptoken, const int32_t* ctok, const double* cw, uint32_t nc, bool* accepted,
                       int32_t* correction, uint64_t* nan_token) {
        if (ptoken < 0 || (uint64_t)ptoken >= n) return S_PROPOSAL_RANGE;
        if (nc == 0) return S_NO_CANDIDATES;
        double ptotal = 0.0, pw = 0.0;
        for (uint32_t i = 0; i < nc; ++i) {
            if (ctok[i] < 0 || (uint64_t)ctok[i] >= n) return S_PROPOSAL_RANGE;
            if (!std::isfinite(cw[i]) || cw[i] < 0.0) return S_PROPOSAL_WEIGHT;
            ptotal += cw[i];
            if (ctok[i] == ptoken) pw += cw[i];
        }
        if (!(std::isfinite(ptotal) && ptotal > 0.0)) return S_NO_CANDIDATES;
        if (!(std::isfinite(pw) && pw > 0.0)) return S_MISSING_PROPOSAL;
        Dist d;
        SErr e = diagnose0(logits, n, d, nan_token);
        if (e != S_OK) return e;
        double tsum = 0.0;
        for (size_t i = 0; i < d.tokens.size(); ++i)
            if (d.tokens[i] == ptoken) tsum += d.weights[i];
        const double tp = tsum / d.total;
        const double pp = pw / ptotal;
        const double acc = std::min(tp / pp, 1.0);
        ++draws;
        if (rng.next_unit() < acc) { *accepted = true; return S_OK; }
        std::vector<double> residual(d.tokens.size());
        double rtotal = 0.0;
        for (size_t i = 0; i < d.tokens.size(); ++i) {
            const double tpi = d.weights[i] / d.total;
            double ps = 0.0;
            for (uint32_t j = 0; j < nc; ++j)
                if (ctok[j] == d.tokens[i]) ps += cw[j];
            const double w = std::max(tpi - ps / ptotal, 0.0);
            rtotal += w;
            residual[i] = w;
        }
        if (!(std::isfinite(rtotal) && rtotal > 0.0)) return S_NO_CANDIDATES;
        ++draws;
        const double threshold = rng.next_unit() * rtotal;
        double cum = 0.0;
        *accepted = false;
        for (size_t i = 0; i < residual.size(); ++i) {
            cum += residual[i];
            if (threshold < cum) { *correction = d.tokens[i]; return S_OK; }
        }
        *correction = d.tokens.back();
        return S_OK;
    }
};

namespace {
dfl_status sampling_fail(SErr e, uint64_t nan_token, int row) {
    const std::string where = row >= 0 ? "DFlash target row " + std::to_string(row) + ": " : "";
    switch (e) {
        case S_EMPTY: return fail(DFL_ERR_SAMPLING, where + "sampling requires a non-empty logits row");
        case S_NAN: return fail(DFL_ERR_SAMPLING, where + "logit at token " + std::to_string(nan_token) + " is NaN");
        case S_TOO_LARGE: return fail(DFL_ERR_SAMPLING, where + "vocabulary size exceeds i32 token ids");
        case S_NO_CANDIDATES: return fail(DFL_ERR_SAMPLING, where + "sampling retained no finite-probability candidates");
        case S_MEMORY: return fail(DFL_ERR_OOM, where + "no memory for the filtered distribution");
        case S_PROPOSAL_RANGE: return fail(DFL_ERR_SAMPLING, where + "proposal token is outside the target vocabulary");
        case S_PROPOSAL_WEIGHT: return fail(DFL_ERR_SAMPLING, where + "proposal weight must be finite and non-negative");
        case S_MISSING_PROPOSAL: return fail(DFL_ERR_SAMPLING, where + "sampled proposal token has no positive proposal weight");
        default: return DFL_OK;
    }
}
bool valid_config(const dfl_sampling_config& c, std::string* why) {
    if (!std::isfinite(c.temperature) || c.temperature < 0.0f) { *why = "sampling temperature must be finite and >= 0"; return false; }
    if (!std::isfinite(c.top_p) || !(0.0f < c.top_p && c.top_p <= 1.0f)) { *why = "top_p must be finite and in (0, 1]"; return false; }
    if (!std::isfinite(c.min_p) || !(0.0f <= c.min_p && c.min_p <= 1.0f)) { *why = "min_p must be finite and in [0, 1]"; return false; }
    return true;
}
}  // namespace

extern "C" {

dfl_status dfl_sampler_create(const dfl_sampling_config* cfg, dfl_sampler** out) {
    if (!cfg || !out) return fail(DFL_ERR_BAD_ARG, "sampler_create: null argument");
    *out = nullptr;
    std::string why;
    if (!valid_config(*cfg, &why)) return fail(DFL_ERR_SAMPLING, why);
    auto* s = new dfl_sampler();
    s->cfg = *cfg;
    s->rng.seed(cfg->seed);
    *out = s;
    return DFL_OK;
}
dfl_status dfl_sampler_create_at_draw(const dfl_sampling_config* cfg, uint64_t draws, dfl_sampler** out) {
    dfl_status st = dfl_sampler_create(cfg, out);
    if (st != DFL_OK) return st;
    for (uint64_t i = 0; i < draws; ++i) (*out)->rng.next_u64();
    (*out)->draws = draws;
    return DFL_OK;
}
void dfl_sampler_destroy(dfl_sampler* s) { delete s; }

dfl_status dfl_sampler_set_worker_threads(dfl_sampler* s, uint32_t n) {
    if (!s) return DFL_ERR_BAD_ARG;
    s->workers = n;
    return DFL_OK;
}

uint64_t dfl_sampler_preordered_rows(const dfl_sampler* s) { return s ? s->ord_used.load(std::memory_order_relaxed) : 0; }

dfl_status dfl_sampler_set_row_order(dfl_sampler* s, const float* logits_base, const uint32_t* order_base, uint32_t n_rows,
                                     uint64_t vocab) {
    if (!s) return DFL_ERR_BAD_ARG;
    if (!logits_base || !order_base || n_rows == 0 || vocab == 0) {
        s->ord_logits = nullptr;
        s->ord_base = nullptr;
        s->ord_rows = 0;
        s->ord_vocab = 0;
        return DFL_OK;
    }
    s->ord_logits = logits_base;
    s->ord_base = order_base;
    s->ord_rows = n_rows;
    s->ord_vocab = vocab;
    return DFL_OK;
}
void dfl_sampler_get_config(const dfl_sampler* s, dfl_sampling_config* out) { if (s && out) *out = s->cfg; }
uint64_t dfl_sampler_draws(const dfl_sampler* s) { return s ? s->draws : 0; }
void dfl_sampler_rng_state(const dfl_sampler* s, uint64_t out_state[4]) {
    if (s) std::memcpy(out_state, s->rng.st, 32);
}
uint64_t dfl_splitmix64_next(uint64_t* state) {
    SplitMix64 sm{*state};
    const uint64_t v = sm.next();
    *state = sm.s;
    return v;
}
uint64_t dfl_sampler_next_u64(dfl_sampler* s) { return s->rng.next_u64(); }
double dfl_sampler_next_unit_f64(dfl_sampler* s) { return s->rng.next_unit(); }

dfl_status dfl_sampler_sample(dfl_sampler* s, const float* logits, uint64_t vocab, int32_t* token_out, uint64_t* candidate_index_out) {
    if (!s || !token_out) return fail(DFL_ERR_BAD_ARG, "sampler_sample: null argument");
    if (vocab && !logits) return fail(DFL_ERR_BAD_ARG, "sampler_sample: logits is null");
    uint64_t nan_token = 0, idx = 0;
    SErr e = s->sample(logits, vocab, token_out, &idx, &nan_token);
    if (candidate_index_out) *candidate_index_out = idx;
    return e == S_OK ? DFL_OK : sampling_fail(e, nan_token, -1);
}

dfl_status dfl_sampler_sample_with_distribution(dfl_sampler* s, const float* logits, uint64_t vocab, int32_t* token_out,
                                                uint64_t* candidate_index_out, int32_t* dist_tokens, double* dist_weights, uint64_t cap,
                                                uint64_t* count, double* total_weight) {
    if (!s || !token_out || (vocab && !logits)) return fail(DFL_ERR_BAD_ARG, "sample_with_distribution: null argument");
    uint64_t nan_token = 0;
    Dist d;
    SErr e;
    if (s->cfg.temperature == 0.0f) {
        e = s->diagnose0(logits, vocab, d, &nan_token);
    } else {
        e = s->distribution(logits, vocab, d, &nan_token);
        if (e == S_OK) {
            ++s->draws;
            dfl_sampler::pick(d, s->rng.next_unit());
        }
    }
    if (e != S_OK) return sampling_fail(e, nan_token, -1);
    *token_out = d.sampled;
    if (candidate_index_out) *candidate_index_out = d.index;
    if (count) *count = d.tokens.size();
    if (total_weight) *total_weight = d.total;
    for (uint64_t i = 0; i < d.tokens.size() && i < cap; ++i) {
        if (dist_tokens) dist_tokens[i] = d.tokens[i];
        if (dist_weights) dist_weights[i] = d.weights[i];
    }
    return DFL_OK;
}

dfl_status dfl_greedy_token(const float* logits, uint64_t vocab, int32_t* token_out) {
    if (!token_out || (vocab && !logits)) return fail(DFL_ERR_BAD_ARG, "greedy_token: null argument");
    uint64_t nan_token = 0;
    SErr e = dfl_sampler::greedy(logits, vocab, token_out, &nan_token);
    return e == S_OK ? DFL_OK : sampling_fail(e, nan_token, -1);
}

dfl_status dfl_sampler_couple_sparse(dfl_sampler* s, const float* logits, uint64_t vocab, int32_t proposal_token, const int32_t* cand_tokens,
                                     const double* cand_weights, uint32_t n_cand, int32_t* accepted, int32_t* correction) {
    if (!s || !logits || !accepted || !correction || (n_cand && (!cand_tokens || !cand_weights)))
        return fail(DFL_ERR_BAD_ARG, "couple_sparse: null argument");
    bool acc = false;
    uint64_t nan_token = 0;
    const Xoshiro saved_rng = s->rng;  // an error consumes no RNG state
    const uint64_t saved_draws = s->draws;
    SErr e = s->couple_sparse(logits, vocab, proposal_token, cand_tokens, cand_weights, n_cand, &acc, correction, &nan_token);
    if (e != S_OK) {
        s->rng = saved_rng;
        s->draws = saved_draws;
        return sampling_fail(e, nan_token, -1);
    }
    *accepted = acc ? 1 : 0;
    return DFL_OK;
}

dfl_status dfl_accept_prefix(const int32_t* verified_tokens, uint32_t n_tokens, const float* target_logits, uint64_t n_logits, uint64_t vocab,
                             const dfl_sparse_proposals* proposals, dfl_sampler* sampler, uint64_t remaining_output_budget,
                             const int32_t* stop_ids, uint32_t n_stop_ids, dfl_accept_decision* out) {
    if (!out || !sampler) return fail(DFL_ERR_BAD_ARG, "accept_prefix: null argument");
    std::memset(out, 0, sizeof(*out));
    out->error_row = -1;
    if (n_tokens == 0 || !verified_tokens) return fail(DFL_ERR_BAD_ARG, "invalid DFlash accept-prefix input: missing carry token");
    if (n_tokens > DFL_MAX_BLOCK) return fail(DFL_ERR_BAD_SHAPE, "invalid DFlash accept-prefix input: more than 16 verified tokens");
    if (vocab == 0 || vocab > 0x7fffffffull) return fail(DFL_ERR_BAD_ARG, "invalid DFlash accept-prefix input: invalid vocabulary size");
    if ((uint64_t)n_tokens * vocab != n_logits || !target_logits)
        return fail(DFL_ERR_BAD_SHAPE, "invalid DFlash accept-prefix input: target logits extent mismatch");
    for (uint32_t i = 0; i < n_tokens; ++i)
        if (verified_tokens[i] < 0 || (uint64_t)verified_tokens[i] >= vocab)
            return fail(DFL_ERR_BAD_TOKEN, "verified input token at index " + std::to_string(i) + " is outside the vocabulary");
    const uint32_t n_drafts = n_tokens - 1;
    if (proposals) {
        if (proposals->n_rows != n_drafts) return fail(DFL_ERR_BAD_SHAPE, "invalid DFlash accept-prefix input: proposal row count mismatch");
        for (uint32_t row = 0; row < n_drafts; ++row) {
            if (proposals->tokens[row] != verified_tokens[row + 1])
                return fail(DFL_ERR_BAD_ARG, "proposal row " + std::to_string(row) + " sampled a token that is not the verified draft");
            for (uint32_t c = proposals->cand_offsets[row]; c < proposals->cand_offsets[row + 1]; ++c)
                if (proposals->cand_tokens[c] < 0 || (uint64_t)proposals->cand_tokens[c] >= vocab) {
                    out->error_row = (int32_t)row;
                    return sampling_fail(S_PROPOSAL_RANGE, 0, (int)row);
                }
        }
    }
    auto is_stop = [&](int32_t t) {
        for (uint32_t i = 0; i < n_stop_ids; ++i)
            if (stop_ids[i] == t) return true;
        return false;
    };
    if (is_stop(verified_tokens[0])) { out->stop_reason = DFL_STOP_EOS; return DFL_OK; }
    if (remaining_output_budget == 0) { out->stop_reason = DFL_STOP_TOKEN_LIMIT; return DFL_OK; }

    // The request sampler advances in place and is rolled back on any error (accept.rs:147,176).
    dfl_sampler& next = *sampler;
    next.prepare_rows(target_logits, n_tokens, vocab);
    struct Unprepare {
        dfl_sampler& s;
        ~Unprepare() { s.end_block(); }
    } unprepare{next};
    const Xoshiro saved_rng = sampler->rng;
    const uint64_t saved_draws = sampler->draws;
    auto rollback = [&]() { sampler->rng = saved_rng; sampler->draws = saved_draws; };
    uint32_t n_acc = 0;
    int32_t carry_kind = DFL_CARRY_NONE, carry = 0, stop = DFL_STOP_NONE;
    for (;;) {
        const uint32_t row = n_acc;
        const float* logits = target_logits + (uint64_t)row * vocab;
        uint64_t nan_token = 0, idx = 0;
        if (row == n_drafts) {
            int32_t bonus = 0;
            SErr e = next.sample(logits, vocab, &bonus, &idx, &nan_token);
            if (e != S_OK) { rollback(); out->error_row = (int32_t)row; return sampling_fail(e, nan_token, (int)row); }
            carry_kind = DFL_CARRY_BONUS;
            carry = bonus;
            break;
        }
        const int32_t draft = verified_tokens[row + 1];
        bool accepted = false;
        int32_t correction = 0;
        SErr e;
        if (proposals) {
            const uint32_t c0 = proposals->cand_offsets[row], c1 = proposals->cand_offsets[row + 1];
            e = next.couple_sparse(logits, vocab, proposals->tokens[row], proposals->cand_tokens + c0, proposals->cand_weights + c0, c1 - c0,
                                   &accepted, &correction, &nan_token);
        } else {
            int32_t target = 0;
            e = next.sample(logits, vocab, &target, &idx, &nan_token);
            accepted = target == draft;
            correction = target;
        }
        if (e != S_OK) { rollback(); out->error_row = (int32_t)row; return sampling_fail(e, nan_token, (int)row); }
        if (!accepted) { carry_kind = DFL_CARRY_CORRECTION; carry = correction; break; }
        out->accepted_drafts[n_acc++] = draft;
        if (is_stop(draft)) { stop = DFL_STOP_EOS; break; }
        if (n_acc == remaining_output_budget) { stop = DFL_STOP_TOKEN_LIMIT; break; }
    }
    out->n_accepted = n_acc;
    out->next_carry_kind = carry_kind;
    out->next_carry = carry;
    out->stop_reason = stop;
    out->retain_input_count = 1 + n_acc - (stop != DFL_STOP_NONE ? 1 : 0);
    return DFL_OK;
}

}  // extern "C"
