// scan.cu -- word finder, two-hit seeding and ungapped X-drop extension of
// the BLASTP preliminary search on GB300 (sm_103a). Integer work only.
//
// One warp per group of subjects (or band of its diagonals); persistent warps
// pull groups, longest subjects first, from a device cursor (batched: one per
// query, and blocks go from query to query). Per block in shared memory: the
// BLOSUM62 matrix, the query's word table or word-presence bitset (neither next
// to the very longest diagonal tables) and, for queries up to kQuerySmemMax, the
// query residues. Per warp: the diagonal table, the deferred-hit and seed queues,
// the list of a chunk's words with hits and a staging buffer for the group, so
// the word scan and the extensions read shared memory instead of making
// dependent global loads.
//
// Reference counterpart: gpuBLAZE_full (BLAZE_gpu/gpuBLAZE.cu:885-1252), which
// is a filter; this kernel produces the exact ungapped HSPs of the
// sequential algorithm.
#include <algorithm>
#include <cstdint>
#include <mutex>
#include <set>
#include <utility>

#include "common.cuh"

namespace blaze {
namespace {

__device__ const int8_t g_blosum8[kAlphabet * kAlphabet] = {
#include "blosum62_i8.inc"
};

constexpr unsigned kFull = 0xffffffffu;
__device__ __forceinline__ unsigned lanemask_lt() { return (1u << (threadIdx.x & 31u)) - 1u; }
__device__ __forceinline__ unsigned lanemask_le() { return 0xffffffffu >> (31u - (threadIdx.x & 31u)); }

// idx mod L for idx < 2^32, with magic = floor(2^32 / L) + 1: the estimated
// quotient is the true one or one more.
__device__ __forceinline__ uint32_t fast_mod(uint32_t idx, uint32_t L, uint32_t magic) {
    const uint32_t qt = __umulhi(idx, magic);
    const int32_t r = static_cast<int32_t>(idx - qt * L);
    return static_cast<uint32_t>(r < 0 ? r + static_cast<int32_t>(L) : r);
}

// ------------------------------------------------------------------------
// Shared-memory layout (byte offsets into the dynamic array). Every table is
// reached through a 32-bit offset into `smem` itself, so all of them compile
// to shared-space accesses.

constexpr uint32_t kMatOff = 0;
constexpr uint32_t kTabOff = kScanMatBytes;  // the word table, or the word-presence bitset
template <Words W>
constexpr uint32_t kQueryOff = kTabOff + words_bytes(W);
// a warp's region, from Finder::w
constexpr uint32_t kBarAt = 0;                                // the stage buffer's mbarrier
constexpr uint32_t kDeferAt = 16;                             // two buffers of deferred hits
constexpr uint32_t kSeedAt = kDeferAt + 2 * kDeferCap * 4;    // queued seeds
constexpr uint32_t kListAt = kSeedAt + kSeedCap * 8;          // words with hits: the chunk's, and those waiting
constexpr uint32_t kDiagAt = kListAt + (kChunk + 32) * 8;     // diagonal table, then the stage buffer
static_assert(kDiagAt == kScanWarpFixedBytes, "a warp's region");

extern __shared__ __align__(16) unsigned char smem[];

__device__ __forceinline__ uint32_t lds16(uint32_t off) { return *reinterpret_cast<const uint16_t *>(smem + off); }
__device__ __forceinline__ uint32_t lds32(uint32_t off) { return reinterpret_cast<const uint32_t *>(smem)[off >> 2]; }
__device__ __forceinline__ void sts32(uint32_t off, uint32_t v) { reinterpret_cast<uint32_t *>(smem)[off >> 2] = v; }
__device__ __forceinline__ uint2 lds64(uint32_t off) { return reinterpret_cast<const uint2 *>(smem)[off >> 3]; }
__device__ __forceinline__ void sts64(uint32_t off, uint2 v) { reinterpret_cast<uint2 *>(smem)[off >> 3] = v; }
// The matrix holds keys: the score times 2^14, less one. A walk that sums them
// has 2^14 x (its score) - (its length), so the largest sum it passes gives the
// best score and, among equals, the first position that reached it.
constexpr int kKeyBits = 14;
constexpr int32_t kKeyMask = (1 << kKeyBits) - 1;
constexpr int32_t kKeyedLength = 11900;  // of a walk: 11 x its length times 2^14 stays below 2^31
__device__ __forceinline__ int32_t key_of(uint32_t qa, uint32_t sb) {
    return reinterpret_cast<const int32_t *>(smem + kMatOff)[qa * kAlphabet + sb];
}
__device__ __forceinline__ int32_t score_of(uint32_t qa, uint32_t sb) { return (key_of(qa, sb) + 1) >> kKeyBits; }
__device__ __forceinline__ int32_t key_score(int32_t k) { return (k + kKeyMask) >> kKeyBits; }
__device__ __forceinline__ int32_t key_length(int32_t k) { return (0 - k) & kKeyMask; }

// ------------------------------------------------------------------------
// Staging by the bulk-copy (TMA) engine: one lane arms the warp's mbarrier
// with the group's bytes, and each lane issues its subject's cp.async.bulk
// global -> shared; the warp waits on the barrier's phase. A warp stages one
// group at a time, just before scanning it, in one stage buffer. Waits are
// bounded: a copy that never lands sets kFlagBadState.

constexpr uint32_t kBulkSpinLimit = 1u << 22;

__device__ __forceinline__ uint32_t smem_base() { return static_cast<uint32_t>(__cvta_generic_to_shared(smem)); }

__device__ __forceinline__ void mbar_init(uint32_t bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void mbar_inval(uint32_t bar) {
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0u;
}

// Lane 0 of the calling warp: arms the barrier with the bytes to come.
__device__ __forceinline__ void stage_expect(uint32_t bytes, uint32_t bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_base() + bar), "r"(bytes)
                 : "memory");
}

// A lane copies `bytes` (a multiple of 16) from 16-byte aligned global `src`
// to shared offset `dst`, reported to the barrier.
__device__ __forceinline__ void bulk_stage(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    const uint32_t d = smem_base() + dst, b = smem_base() + bar;
    // earlier generic accesses of this buffer come before the async overwrite
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(d), "l"(src), "r"(bytes), "r"(b)
                 : "memory");
}

// A group's residues by position x: in the stage buffer, or, for a subject too
// long for it, in global memory. In the stage buffer each subject begins in a
// 16-byte block of its own, with zeros around it: no word with a zero letter
// has a hit.
template <bool STAGED>
struct Span {
    uint32_t off;        // shared offset of x = 0 (staged)
    const uint8_t *ptr;  // global address of x = 0 (not staged)
    __device__ __forceinline__ uint32_t at(int32_t x) const {
        if (STAGED) return smem[off + x];
        return __ldg(ptr + x);
    }
};

// One subject of the span.
template <bool STAGED>
struct Subject {
    Span<STAGED> span;
    int32_t first, len;  // position of its residue 0, its length
    __device__ __forceinline__ uint32_t at(int32_t i) const { return span.at(first + i); }
};

// The query: in shared memory for queries up to kQuerySmemMax, else global.
template <bool QSMEM, Words W>
struct Query {
    const uint8_t *ptr;
    int32_t len;
    __device__ __forceinline__ uint32_t at(int32_t i) const {
        if (QSMEM) return smem[kQueryOff<W> + i];
        return __ldg(ptr + i);
    }
};

// ------------------------------------------------------------------------
// Ungapped extension (scalar, one lane per seed), same walks as the oracle:
// left from the end of the best word prefix, right only when the left walk
// reached the first hit (BLAZE_gpu/gpuBLAZE.cu:1096-1152 is the warp form).

template <typename Q, typename S>
__device__ __forceinline__ int32_t extend_left(const Q &q, const S &s, int32_t q_off,
                                               int32_t s_off, int32_t xdrop, int32_t *length) {
    const int32_t n = min(s_off, q_off);
    int32_t best_k = -1, score = 0, maxscore = 0;
    for (int32_t k = 0; k <= n; ++k) {
        score += score_of(q.at(q_off - k), s.at(s_off - k));
        if (score > maxscore) {
            maxscore = score;
            best_k = k;
        }
        if (maxscore - score >= xdrop) break;
    }
    *length = best_k + 1;
    return maxscore;
}

template <typename Q, typename S>
__device__ __forceinline__ int32_t extend_right(const Q &q, const S &s, int32_t q_off,
                                                int32_t s_off, int32_t xdrop, int32_t maxscore,
                                                int32_t *length, int32_t *s_last_off) {
    const int32_t n = min(s.len - s_off, q.len - q_off);
    int32_t best_i = -1, score = maxscore, i;
    for (i = 0; i < n; ++i) {
        score += score_of(q.at(q_off + i), s.at(s_off + i));
        if (score > maxscore) {
            maxscore = score;
            best_i = i;
        }
        if (score <= 0 || maxscore - score >= xdrop) break;
    }
    *length = best_i + 1;
    *s_last_off = s_off + i;
    return maxscore;
}

// The same walks on keys, for sequences of which one is at most kKeyedLength
// long: one sum, one maximum and one comparison a position, kWalkStep positions
// a step: their loads do not wait for the comparisons before them. A walk that
// ends inside a step takes nothing from the step's rest. 139 M residues at 300 /
// 1,000 / 3,000 query residues, by positions a step: 1 1.09 / 2.78 / 9.11 ms, 2
// 1.01 / 2.58 / 8.27, 4 1.02 / 2.58 / 8.30, 8 1.08 / 2.71 / 8.55.
constexpr int32_t kWalkStep = 2;
template <typename Q, typename S>
__device__ __forceinline__ int32_t extend_two_hit_keyed(const Q &q, const S &s, int32_t s_left_off, int32_t s_off,
                                                        int32_t q_off, int32_t xdrop, int32_t *hsp_q, int32_t *hsp_s,
                                                        int32_t *hsp_len, int32_t *right_extend,
                                                        int32_t *s_last_off) {
    const int32_t drop = min(xdrop, (1 << (31 - kKeyBits)) - 1) << kKeyBits;
    int32_t k = 0, m = 0;
#pragma unroll
    for (int32_t i = 0; i < kWordSize; ++i) {
        k += key_of(q.at(q_off + i), s.at(s_off + i));
        m = max(m, k);
    }
    const int32_t q_right = q_off + key_length(m), s_right = s_off + key_length(m);
    k = m = 0;
    bool on = true;
    int32_t i = 1, n = min(s_right, q_right);
    auto left = [&](int32_t key) {
        k += key;
        if (on) m = max(m, k);
        on = on && m - k < drop;
    };
    for (; on && i + kWalkStep <= n + 1; i += kWalkStep) {
        int32_t key[kWalkStep];
#pragma unroll
        for (int32_t j = 0; j < kWalkStep; ++j) key[j] = key_of(q.at(q_right - i - j), s.at(s_right - i - j));
#pragma unroll
        for (int32_t j = 0; j < kWalkStep; ++j) left(key[j]);
    }
    for (; on && i <= n; ++i) left(key_of(q.at(q_right - i), s.at(s_right - i)));
    const int32_t left_d = key_length(m);
    int32_t score = key_score(m), right_d = 0;
    *right_extend = 0;
    *s_last_off = s_right;
    if (left_d >= s_right - s_left_off) {
        *right_extend = 1;
        k = m = score << kKeyBits;
        on = true;
        int32_t past = 0;  // positions passed
        auto right = [&](int32_t key) {
            k += key;
            if (on) m = max(m, k);
            on = on && m - k < drop && k > 0;
            past += on ? 1 : 0;
        };
        i = 0;
        n = min(s.len - s_right, q.len - q_right);
        for (; on && i + kWalkStep <= n; i += kWalkStep) {
            int32_t key[kWalkStep];
#pragma unroll
            for (int32_t j = 0; j < kWalkStep; ++j) key[j] = key_of(q.at(q_right + i + j), s.at(s_right + i + j));
#pragma unroll
            for (int32_t j = 0; j < kWalkStep; ++j) right(key[j]);
        }
        for (; on && i < n; ++i) right(key_of(q.at(q_right + i), s.at(s_right + i)));
        right_d = key_length(m);
        score = key_score(m);
        *s_last_off = s_right + past;
    }
    *hsp_q = q_right - left_d;
    *hsp_s = s_right - left_d;
    *hsp_len = left_d + right_d;
    return score;
}

template <typename Q, typename S>
__device__ __forceinline__ int32_t extend_two_hit(const Q &q, const S &s,
                                                  int32_t s_left_off, int32_t s_off, int32_t q_off,
                                                  int32_t xdrop, int32_t *hsp_q, int32_t *hsp_s,
                                                  int32_t *hsp_len, int32_t *right_extend,
                                                  int32_t *s_last_off) {
    int32_t score = 0, left_score = 0, right_d = 0, left_d = 0, right_score = 0;
#pragma unroll
    for (int32_t i = 0; i < kWordSize; ++i) {
        score += score_of(q.at(q_off + i), s.at(s_off + i));
        if (score > left_score) {
            left_score = score;
            right_d = i + 1;
        }
    }
    const int32_t q_right = q_off + right_d, s_right = s_off + right_d;
    left_score = extend_left(q, s, q_right - 1, s_right - 1, xdrop, &left_d);
    right_d = 0;
    *right_extend = 0;
    *s_last_off = s_right;
    if (left_d >= s_right - s_left_off) {
        *right_extend = 1;
        right_score = extend_right(q, s, q_right, s_right, xdrop, left_score, &right_d, s_last_off);
    }
    *hsp_q = q_right - left_d;
    *hsp_s = s_right - left_d;
    *hsp_len = left_d + right_d;
    return max(left_score, right_score);
}

// ------------------------------------------------------------------------
// Word finder state of one warp. A hit is a pair (v, q): v is the position x
// plus `window` for each subject of the group before its own, so that hits of
// different subjects are always more than `window` apart. The diagonal table
// holds, per diagonal (v - q) mod L, either the last recorded hit (v plus a
// running base, so the table never needs clearing between groups), the end of
// a right extension with kFlag, or kPend | seed slot while that diagonal's
// extension is queued. With L >= qlen + window two diagonals that share an
// entry never both matter: all hits of the later one come more than `window`
// positions after every hit of the earlier one and after the end of any
// extension on it; only a seed still queued for an earlier subject makes a hit
// on its entry wait.
//
// Entries are 16 bits wide for the queries kept in shared memory, which
// leaves room for twice the warps with long queries (3,000 residues: 24
// instead of 14 per SM, 18.4 -> 11.7 ms for 139 M residues); the
// values then stay below 2^14: the table is cleared before a group that would
// pass it, and moved down (rebase) inside a long subject. Otherwise 32 bits.
template <bool QS>
struct Tab {
    static constexpr uint32_t kFlag = QS ? 0x8000u : 0x40000000u;
    static constexpr uint32_t kPend = QS ? 0xc000u : 0x60000000u;
    static constexpr uint32_t kMost = QS ? 0x3fffu : 0x1fffffffu;  // the largest value
    static __device__ __forceinline__ uint32_t at(uint32_t w, uint32_t d) { return w + (QS ? 2u : 4u) * d; }
    static __device__ __forceinline__ uint32_t load(uint32_t o) {
        return QS ? lds16(kDiagAt + o) : *reinterpret_cast<const uint32_t *>(smem + kDiagAt + o);
    }
    static __device__ __forceinline__ void store(uint32_t o, uint32_t v) {
        if (QS) *reinterpret_cast<uint16_t *>(smem + kDiagAt + o) = static_cast<uint16_t>(v);
        else *reinterpret_cast<uint32_t *>(smem + kDiagAt + o) = v;
    }
};

struct Finder {
    uint32_t w;  // shared offset of the warp's region
    uint32_t phase, sel;
    int n_defer, n_seed;
    uint32_t base;
    uint32_t n_init;
    uint32_t hits, extensions;  // not yet added to the counters
    uint32_t ns;                // subjects of the group
    uint32_t first, end;        // lane i < ns: subject i's positions [first, end); first is 2^31 - 1 from ns on
    int32_t vb;                 // packed hits count v from here
};

// Per-query parameters of the word finder (one query, or the query of the
// batch at hand).
struct Ctx {
    int32_t qlen;
    const uint32_t *cell_start, *cell_pack;
    const uint16_t *cell_off;
    uint32_t diag_entries, diag_magic, diag_bytes;
    int32_t window, xdrop, cutoff;
    uint32_t seed_span;  // distances from the word size on that trigger an extension
};

// The diagonals of a group that a warp takes: those with v - q + (query length)
// in [first, end). A group is cut into bands where its warp would be the last
// one running, or where a table of the query's whole length plus the window
// would leave few warps on an SM. State is kept per diagonal, so bands are
// independent; a word's hits in a band are one run of its ascending hit list.
struct Band {
    int32_t first, end;
    bool all;  // the only band
};

constexpr int32_t kPackSpan = 1 << 17;
static_assert(kQuerySmemMax <= kKeyedLength, "walks on keys");
static_assert(kGroupMaxBytes + (kGroupMaxSubjects + 2) * kTab16Window <= Tab<true>::kMost, "16-bit entries");
static_assert(kBandQuerySmemMax + kChunk + kTab16Window <= Tab<true>::kMost, "16-bit entries");

// A hit in 32 bits: v (17 bits from vb on) and q (at most 32,000).
__device__ __forceinline__ uint32_t pack_hit(const Finder &f, int32_t v, int32_t q) {
    return (static_cast<uint32_t>(v - f.vb) << 15) | static_cast<uint32_t>(q);
}
__device__ __forceinline__ int32_t hit_v(const Finder &f, uint32_t p) { return static_cast<int32_t>(p >> 15) + f.vb; }
__device__ __forceinline__ int32_t hit_q(uint32_t p) { return static_cast<int32_t>(p & 0x7fffu); }

__device__ __forceinline__ uint32_t defer_at(const Finder &f, uint32_t buf, int i) {
    return f.w + kDeferAt + 4u * (buf * kDeferCap + static_cast<uint32_t>(i));
}
// A seed: the packed hit that triggered it and its distance from the first hit.
__device__ __forceinline__ uint32_t seed_at(const Finder &f, int i) {
    return f.w + kSeedAt + 8u * static_cast<uint32_t>(i);
}
__device__ __forceinline__ uint32_t diag_of(const Ctx &c, int32_t v, int32_t q) {
    return fast_mod(static_cast<uint32_t>(v - q + c.qlen), c.diag_entries, c.diag_magic);
}
__device__ __forceinline__ InitHit *scratch_of(const ScanArgs &a) {
    const unsigned long long gwarp = (static_cast<unsigned long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    return a.scratch + gwarp * a.scratch_cap;
}

// Stores `here` in the entry for the lanes that `act` and returns, for them,
// what the entry then holds: the smallest `here` of the lanes that share it.
// The hardware keeps the lowest lane's store, and lanes are in hit order; the
// loop makes sure of it.
template <bool QS>
__device__ __forceinline__ uint32_t claim(uint32_t entry, uint32_t here, bool act) {
    uint32_t low = here;
    __syncwarp();
    if (act) Tab<QS>::store(entry, here);
    __syncwarp();
    if (act) low = Tab<QS>::load(entry);
    while (__any_sync(kFull, low > here)) {
        if (low > here) Tab<QS>::store(entry, here);
        __syncwarp();
        if (act) low = Tab<QS>::load(entry);
        __syncwarp();
    }
    return low;
}

// Runs up to 32 hits (one per lane, lanes in hit order) through the two-hit
// logic. The entry's distance below a hit decides what it does: a flagged entry
// is further below than any recorded hit, a pending one further still (every
// value stays within Tab::kMost).
//
// About a quarter of a batch's hits share their diagonal with an earlier lane,
// mostly the next word of the same match (1 or 2 positions on). The lanes whose
// hits do something claim their entries; the first of a diagonal does what the
// entry said, and leaves the others one of two cases:
//   it is a seed: they are deferred, as every later hit is until it is extended
//   it starts over: a hit 1 or 2 positions on is ignored, and the first of
//     the others decides by its distance from it: the second claim
// Behind a second hit that starts over as well (rare: it is `window` or more
// from the first) the rest is brought again: true is returned for them.
//
// The kernel is bound by instruction issue (85 % at 300 query residues), and
// this function was nearly half of it. __match_any_sync in place of the claims
// costs few instructions, but 8.4 cycles per distinct value: 270 for a batch of
// 32 diagonals. With the claims and full batches: 139 M residues at 300 / 1,000
// query residues 1.26 -> 1.05 and 3.39 -> 2.70 ms.
template <bool QS>
__device__ __forceinline__ bool two_hit(Finder &f, const Ctx &c, bool valid, int32_t v, int32_t q) {
    const uint32_t entry = Tab<QS>::at(f.w, diag_of(c, v, q));
    const uint32_t here = static_cast<uint32_t>(v) + f.base;
    const uint32_t e = valid ? Tab<QS>::load(entry) : here;  // a lane without a hit does nothing
    int32_t dist = static_cast<int32_t>(here - e);
    // a hit far from the last one starts over, as does the first hit past the
    // end of an extension (the wrapped distances from -kFlag on); one at
    // distance [wordsize, window) triggers an extension; an overlapping one,
    // and one inside the last extension, is ignored
    const bool near = static_cast<uint32_t>(dist - kWordSize) < c.seed_span;
    const bool act = near || dist >= c.window || static_cast<uint32_t>(dist) >= 0u - Tab<QS>::kFlag;
    const uint32_t low = claim<QS>(entry, here, act);
    const bool alone = low == here;
    bool seed = near && alone;
    bool def = valid && e >= Tab<QS>::kPend;  // its diagonal waits for an extension
    bool again = false;
    if (__any_sync(kFull, !alone)) {
        const bool behind_seed = static_cast<uint32_t>(static_cast<int32_t>(low - e) - kWordSize) < c.seed_span;
        const int32_t df = static_cast<int32_t>(here - low);
        def = def || (!alone && behind_seed);
        const bool wait = !behind_seed && df >= kWordSize;
        if (__any_sync(kFull, wait)) {
            const uint32_t low2 = claim<QS>(entry, here, wait);
            const bool second = static_cast<int32_t>(low2 - low) < c.window;  // the second hit is a seed
            if (wait) {
                dist = df;
                seed = second && low2 == here;
                def = second && low2 != here;
                again = !second && low2 != here;
            }
        }
    }
    const unsigned dm = __ballot_sync(kFull, def);
    const unsigned sm = __ballot_sync(kFull, seed);
    if ((dm | sm) != 0u) {
        const unsigned lt = lanemask_lt();
        const uint32_t packed = pack_hit(f, v, q);
        if (def) sts32(defer_at(f, f.sel, f.n_defer + __popc(dm & lt)), packed);
        if (seed) {
            const int slot = f.n_seed + __popc(sm & lt);
            sts64(seed_at(f, slot), make_uint2(packed, static_cast<uint32_t>(dist)));
            Tab<QS>::store(entry, Tab<QS>::kPend | static_cast<uint32_t>(slot));
        }
        f.n_defer += __popc(dm);
        f.n_seed += __popc(sm);
    }
    __syncwarp();
    return again;
}

// Whether the queues may not hold another batch's seeds or deferred hits.
__device__ __forceinline__ bool queues_full(const Finder &f) {
    return f.n_seed >= 32 || f.n_defer > kDeferCap - 32;
}

// Extends every queued seed (one lane each), settles their diagonals, keeps
// those reaching the ungapped cutoff, then replays the deferred hits. The
// seeds that the replay queues wait for the next flush, unless the queues are
// still too full for another batch or (`empty`) have to be emptied: then it
// repeats. Each replay is shorter than the list it replays whenever it queues
// a seed, so the loop ends. Seeds of all the group's subjects share a flush: a
// walk takes as many warp instructions a step whether one lane or 32 take it,
// so what an extension costs falls with the seeds it shares its flush with.
template <bool QS, Words W, bool BANDS, bool ST>
__device__ __forceinline__ void flush(Finder &f, const ScanArgs &a, const Ctx &c, const Query<QS, W> &q,
                                      const Span<ST> &span, bool empty) {
    const uint32_t lane = threadIdx.x & 31;
    const unsigned lt = lanemask_lt();
    // where subject `lane` begins in v (its 16-byte block where there are several)
    const uint32_t v0 = f.ns > 1 ? (f.first & ~15u) + static_cast<uint32_t>(c.window) * lane : f.first;
    do {
        for (int c0 = 0; c0 < f.n_seed; c0 += 32) {
            const int i = c0 + static_cast<int>(lane);
            const uint2 sd = lds64(seed_at(f, min(i, f.n_seed - 1)));
            const int32_t hv = hit_v(f, sd.x), hq = hit_q(sd.x);
            uint32_t subj = 0;  // the last subject that begins at or before the hit
            if (f.ns > 1) {
#pragma unroll
                for (uint32_t step = 16; step >= 1; step >>= 1)
                    if (__shfl_sync(kFull, v0, subj + step) <= static_cast<uint32_t>(hv)) subj += step;
            }
            Subject<ST> sub;
            sub.span = span;
            sub.first = static_cast<int32_t>(__shfl_sync(kFull, f.first, subj));
            sub.len = static_cast<int32_t>(__shfl_sync(kFull, f.end, subj)) - sub.first;
            bool pass = false;
            InitHit h{};
            if (i < f.n_seed) {
                const int32_t to_v = c.window * static_cast<int32_t>(subj) + sub.first;  // from the subject's offsets
                const int32_t so = hv - to_v, left = so - static_cast<int32_t>(sd.y) + kWordSize;
                int32_t rext, slast;
                h.score = (QS && !BANDS) || min(c.qlen, sub.len) <= kKeyedLength
                              ? extend_two_hit_keyed(q, sub, left, so, hq, c.xdrop, &h.q_start, &h.s_start, &h.len,
                                                     &rext, &slast)
                              : extend_two_hit(q, sub, left, so, hq, c.xdrop, &h.q_start, &h.s_start, &h.len, &rext,
                                               &slast);
                Tab<QS>::store(Tab<QS>::at(f.w, diag_of(c, hv, hq)),
                               rext ? Tab<QS>::kFlag | (static_cast<uint32_t>(slast - (kWordSize - 1) + to_v) + f.base)
                                    : static_cast<uint32_t>(hv) + f.base);
                pass = h.score >= c.cutoff;
                h.q_trig = hq;
                h.s_trig = so + sub.first;  // positions until the group is published
                h.s_start += sub.first;
            }
            const unsigned pm = __ballot_sync(kFull, pass);
            const uint32_t at = f.n_init + __popc(pm & lt);
            if (pass && at < a.scratch_cap) scratch_of(a)[at] = h;
            f.n_init += __popc(pm);
        }
        f.extensions += static_cast<uint32_t>(f.n_seed);
        f.n_seed = 0;
        __syncwarp();
        if (f.n_defer > 0) {
            const uint32_t old = f.sel;
            const int n_old = f.n_defer;
            f.sel ^= 1u;
            f.n_defer = 0;
            for (int c0 = 0; c0 < n_old; c0 += 32) {
                const int i = c0 + static_cast<int>(lane);
                const uint32_t p = lds32(defer_at(f, old, min(i, n_old - 1)));
                bool again = i < n_old;
                do again = two_hit<QS>(f, c, again, hit_v(f, p), hit_q(p));
                while (__any_sync(kFull, again));
            }
        }
    } while (queues_full(f) || (empty && (f.n_seed > 0 || f.n_defer > 0)));
}

// Adds the hit and extension counts to the launch's counters.
__device__ __forceinline__ void add_counts(Finder &f, const ScanArgs &a) {
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&a.cnt->word_hits, static_cast<unsigned long long>(f.hits));
        atomicAdd(&a.cnt->extensions, static_cast<unsigned long long>(f.extensions));
    }
    f.hits = f.extensions = 0;
}

// Whether the chunk at cb of a group of one subject (ending at `end`) needs a
// rebase first: the values its hits and extensions can reach, or its packed
// hits, would pass their limits.
template <bool QS>
__device__ __forceinline__ bool needs_rebase(const Finder &f, const Ctx &c, int32_t end, int32_t cb) {
    if (QS) return static_cast<uint32_t>(min(end, cb + kChunk + c.qlen)) + f.base > Tab<QS>::kMost;
    return cb - f.vb > kPackSpan - kChunk;
}

// Lets packed hits count from cb and (16-bit entries) moves the table down so
// that a hit at cb has value `window`; an entry that falls below 0 is more
// than `window` behind cb, or an extension's end behind it, and stays so as 0.
// The queues are empty.
template <bool QS>
__device__ __forceinline__ void rebase(Finder &f, const ScanArgs &a, const Ctx &c, int32_t cb) {
    f.vb = cb;
    add_counts(f, a);
    if (!QS) return;
    const uint32_t delta = static_cast<uint32_t>(cb - c.window) + f.base;
    for (uint32_t i = threadIdx.x & 31; i < c.diag_entries; i += 32) {
        const uint32_t o = Tab<QS>::at(f.w, i), e = Tab<QS>::load(o), v = e & Tab<QS>::kMost;
        Tab<QS>::store(o, (e & Tab<QS>::kFlag) | (v > delta ? v - delta : 0u));
    }
    f.base -= delta;
    __syncwarp();
}

// x << n, 0 from n = 32 on
__device__ __forceinline__ uint32_t shift_left(uint32_t x, uint32_t n) {
    uint32_t r;
    asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(n));
    return r;
}

// Inclusive prefix sum over the warp.
__device__ __forceinline__ uint32_t warp_prefix(uint32_t x) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
        asm volatile("{\n .reg .pred p;\n .reg .u32 t;\n shfl.sync.up.b32 t|p, %0, %1, 0, 0xffffffff;\n @p add.u32 %0, %0, t;\n}"
            : "+r"(x)
            : "r"(o));
    return x;
}

// The parts of the cells at v0 .. v0 + 3 (from cs on, cnt offsets each) on the
// band's diagonals: offsets q with v + qlen - q in [band.first, band.end). The
// eight lower bounds are searched in step, so that their loads overlap.
__device__ __forceinline__ void clip_cells(const Ctx &c, const Band &band, int32_t v0, uint32_t *cs, uint32_t *cnt) {
    const int32_t from = v0 + c.qlen - band.end + 1, to = v0 + c.qlen - band.first + 1;  // q in [from + j, to + j)
    const bool clip = from + 3 > 0 || to < c.qlen;
    const uint32_t most = max(max(cnt[0], cnt[1]), max(cnt[2], cnt[3]));
    const uint32_t all = __reduce_max_sync(kFull, clip ? most : 0u);
    uint32_t lo[4], hi[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        lo[j] = 0u;
        hi[j] = clip ? 0u : cnt[j];
    }
    for (uint32_t step = all ? 0x80000000u >> __clz(static_cast<int>(all)) : 0u; step != 0u; step >>= 1) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint16_t *off = c.cell_off + cs[j];
            if (lo[j] + step <= cnt[j] && static_cast<int32_t>(__ldg(off + (lo[j] + step - 1u))) < from + j) lo[j] += step;
            if (hi[j] + step <= cnt[j] && static_cast<int32_t>(__ldg(off + (hi[j] + step - 1u))) < to + j) hi[j] += step;
        }
    }
    if (all) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            cs[j] += lo[j];
            cnt[j] = hi[j] - lo[j];
        }
    }
}

// Word scan of a group: chunks of 128 positions, four consecutive positions
// per lane. One warp prefix sum per chunk numbers the chunk's hits in (subject
// offset, query offset) order and the words that have any; each such word
// leaves its v and where its hits lie in the warp's list. Lanes then take the
// hits 32 at a time: a bit mask of the hits that start a word gives each lane
// its word by a population count. A chunk's last hits, too few for a batch,
// wait in front of the next chunk's, so batches are full (at 300 query
// residues a chunk brings 79 hits).
template <bool QS, Words W, bool BANDS, bool ST>
__device__ __forceinline__ void scan_span(Finder &f, const ScanArgs &a, const Ctx &c, const Query<QS, W> &q,
                                          const Span<ST> &span, bool long_one, const Band &band) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t list = f.w + kListAt;
    const int32_t end = static_cast<int32_t>(__shfl_sync(kFull, f.end, f.ns - 1u));
    int32_t xend = end - (kWordSize - 1);        // words start below it
    uint32_t before = 0;                         // subjects that begin before the chunk
    uint32_t left = 0;   // hits waiting from the chunks before, fewer than a batch
    uint32_t left_m = 0; // which of them start a word
    uint32_t left_w = 0; // words begun before the chunk whose hits are waiting
    // four positions of a lane lie in one subject's block
    int32_t cb = static_cast<int32_t>(__shfl_sync(kFull, f.first, 0));
    if (f.ns > 1) {
        cb &= ~15;
    } else if (BANDS && !band.all) {  // the positions that have a hit on the band's diagonals
        cb += max(0, band.first - c.qlen - cb) & ~(kChunk - 1);
        xend = min(xend, band.end - 1);
    }
    for (; cb < xend; cb += kChunk) {
        if (long_one && needs_rebase<QS>(f, c, end, cb)) rebase<QS>(f, a, c, cb);
        // the queues are emptied at the group's end and before a rebase
        const bool empty = cb + kChunk >= xend || (long_one && needs_rebase<QS>(f, c, end, cb + kChunk));
        const int32_t p0 = cb + 4 * static_cast<int32_t>(lane);
        uint32_t r[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) r[j] = span.at(ST ? p0 + j : min(p0 + j, end - 1));
        int32_t v0 = p0;
        if (f.ns > 1) {
            const uint32_t begins =
                __reduce_or_sync(kFull, shift_left(1u, ((f.first & ~15u) - static_cast<uint32_t>(cb)) >> 2));
            v0 += c.window * static_cast<int32_t>(before + __popc(begins & lanemask_le()) - 1u);
            before += __popc(begins);
        }
        uint32_t cs[4], cnt[4], has[4], sum = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const bool in = ST || p0 + j < xend;  // (zeros follow the staged residues)
            if (W == Words::kTable) {
                const uint32_t t = kTabOff + (in ? r[j] * 1568u + r[j + 1] * 56u + r[j + 2] * 2u : 0u);
                cs[j] = lds16(t);
                cnt[j] = lds16(t + 2u) - cs[j];
            } else {
                const uint32_t w = in ? r[j] * 784u + r[j + 1] * 28u + r[j + 2] : 0u;
                const bool present = W == Words::kPacked ? in : (lds32(kTabOff + 4u * (w >> 5)) >> (w & 31u)) & 1u;
                const uint32_t pk = present ? __ldg(c.cell_pack + w) : 0u;
                cs[j] = pk >> 8;
                cnt[j] = pk & 0xffu;
                if (cnt[j] == 0xffu) {  // the count or the start does not fit the packed cell
                    cs[j] = __ldg(c.cell_start + w);
                    cnt[j] = __ldg(c.cell_start + w + 1) - cs[j];
                }
            }
        }
        if (BANDS && !band.all) clip_cells(c, band, v0, cs, cnt);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            has[j] = min(cnt[j], 1u);
            sum += cnt[j] * 256u + has[j];  // 24 bits: 128 words of at most 32,000 hits
        }
        const uint32_t incl = warp_prefix(sum);
        const uint32_t all = __shfl_sync(kFull, incl, 31);
        if (all == 0 && !empty) continue;
        f.hits += all >> 8;
        const uint32_t total = left + (all >> 8);  // hits, the waiting ones first
        uint32_t e[4], run = left + ((incl - sum) >> 8), slot = list + 8u * (left_w + ((incl - sum) & 0xffu));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            e[j] = run;  // the word's first hit
            if (cnt[j]) sts64(slot, make_uint2(cs[j] - run, static_cast<uint32_t>(v0 + j)));
            slot += 8u * has[j];
            run += cnt[j];
        }
        __syncwarp();
        // words that begin with one of the hits k0 .. k0 + 31
        auto begins_from = [&](uint32_t k0) {
            return __reduce_or_sync(kFull, shift_left(has[0], e[0] - k0) | shift_left(has[1], e[1] - k0) |
                                               shift_left(has[2], e[2] - k0) | shift_left(has[3], e[3] - k0));
        };
        uint32_t m = begins_from(0) | left_m;
        // the last word begun before the batch: with hits waiting, the first of the list is
        uint32_t word = list - (left > 0 && (left_m & 1u) == 0u ? 0u : 8u);
        uint32_t k0 = 0;  // the first hit not yet taken
        do {
            bool batch = k0 + 32u <= total || (empty && k0 < total);
            if (batch) {
                const uint32_t k = k0 + lane;
                const uint2 wd = lds64(word + 8u * __popc(m & lanemask_le()));
                word += 8u * __popc(m);
                bool go = k < total;
                const int32_t qo = go ? static_cast<int32_t>(__ldg(c.cell_off + (wd.x + k))) : 0;
                do go = two_hit<QS>(f, c, go, static_cast<int32_t>(wd.y), qo);
                while (__any_sync(kFull, go));
                k0 += 32u;
                m = begins_from(k0);
            }
            const bool done = empty && k0 >= total;
            if (queues_full(f) || done) flush<QS, W, BANDS>(f, a, c, q, span, done);
            if (done || !batch) break;
        } while (true);
        // the hits left wait: their words move to the front of the list, counted from k0
        left = k0 < total ? total - k0 : 0u;
        left_m = m;
        left_w = 0;
        if (left > 0) {
            const uint32_t from = (m & 1u) ? word + 8u : word;  // the first hit's word
            left_w = __popc(m | 1u);
            uint2 wd = make_uint2(0u, 0u);
            if (lane < left_w) wd = lds64(from + 8u * lane);
            __syncwarp();
            if (lane < left_w) sts64(list + 8u * lane, make_uint2(wd.x + k0, wd.y));
        }
        __syncwarp();
    }
}

__device__ __forceinline__ uint32_t seed_span(int32_t window) {
    return window > kWordSize ? static_cast<uint32_t>(window - kWordSize) : 0u;
}

// Waits for the stage buffer's copy; false (with kFlagBadState set) if it
// never completes within the spin limit.
__device__ __forceinline__ bool stage_wait(Finder &f, const ScanArgs &a) {
    const uint32_t bar = smem_base() + f.w + kBarAt;
    for (uint32_t i = 0; i < kBulkSpinLimit; ++i) {
        if (mbar_try_wait(bar, f.phase)) {
            f.phase ^= 1u;
            return true;
        }
    }
    if ((threadIdx.x & 31) == 0) atomicOr(&a.cnt->flags, kFlagBadState);
    return false;
}

// Publishes the init hits of the group's subject number `subj` (sorted index
// `subject`, positions [x0, x1)), `n` of the group's, as one contiguous block
// with a work item.
__device__ __forceinline__ void publish_subject(const Finder &f, const ScanArgs &a, uint32_t subject, int32_t x0,
                                                int32_t x1, uint32_t n, uint32_t query_index) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = lanemask_lt();
    unsigned long long first = 0, wi = 0;
    if (lane == 0) {
        first = atomicAdd(&a.cnt->init_count, static_cast<unsigned long long>(n));
        wi = atomicAdd(&a.cnt->work_count, 1ull);
    }
    first = __shfl_sync(kFull, first, 0);
    wi = __shfl_sync(kFull, wi, 0);
    const bool fits = first + n <= a.init_cap && wi < a.work_cap;
    if (!fits && lane == 0) atomicOr(&a.cnt->flags, first + n > a.init_cap ? kFlagInitArrayFull : kFlagWorkArrayFull);
    if (fits) {
        uint32_t done = 0;
        for (uint32_t i0 = 0; i0 < f.n_init; i0 += 32) {
            const bool v = i0 + lane < f.n_init;
            InitHit h{};
            if (v) h = scratch_of(a)[i0 + lane];
            const bool mine = v && h.s_trig >= x0 && h.s_trig < x1;
            const unsigned m = __ballot_sync(kFull, mine);
            if (mine) {
                h.s_start -= x0;
                h.s_trig -= x0;
                a.init_out[first + done + __popc(m & lt)] = h;
            }
            done += __popc(m);
        }
    }
    if (lane == 0 && wi < a.work_cap) {  // a counted slot always holds an item: an empty one if it does not fit
        WorkItem w;
        w.subject = subject;
        w.n_init = fits ? n : 0u;
        w.first = fits ? first : 0u;
        a.work[wi] = w;
        if (a.work_query) a.work_query[wi] = query_index;
    }
}

// Subjects about to be scanned together: the first, its residues (at o0) and
// whether they are on their way to the stage buffer.
struct Group {
    uint32_t lo;
    uint64_t o0;
    bool staged;
};

// Takes the subjects [lo, hi) of a group, or as many as fit the stage buffer,
// and starts their copies there, each lane its subject's; the first one stays in
// global memory when not even it fits or `staging` is off.
__device__ __forceinline__ Group fetch_group(Finder &f, const ScanArgs &a, const Ctx &c, uint32_t lo, uint32_t hi,
                                             bool staging) {
    const uint32_t lane = threadIdx.x & 31;
    Group r;
    r.lo = lo;
    f.ns = hi - lo;  // 1 .. kGroupMaxSubjects
    const uint64_t mine = a.off[lo + min(lane, f.ns)];
    r.o0 = __shfl_sync(kFull, mine, 0);
    const uint64_t next = __shfl_down_sync(kFull, mine, 1);
    const uint32_t lead = static_cast<uint32_t>(mine & 15u);
    uint32_t len = lane < f.ns ? static_cast<uint32_t>(next - mine) : 0u;
    // a subject's block: what precedes it in its first 16 bytes, it, two zeros
    const uint32_t block = lane < f.ns ? (lead + len + 2u + 15u) & ~15u : 0u;
    const uint32_t to = warp_prefix(block);
    const bool fits = lane < f.ns && staging && to <= scan_stage_blocks(a.stage_bytes) &&
                      (lane == 0u || to + static_cast<uint32_t>(c.window) * (lane + 1u) <= kPackSpan - kChunk);
    const uint32_t n = __popc(__ballot_sync(kFull, fits));  // the first n subjects do
    r.staged = n > 0u;
    f.ns = max(n, 1u);
    const bool has = lane < f.ns;
    if (!has) len = 0u;
    f.first = has ? (r.staged ? to - block + lead : 0u) : 0x7fffffffu;
    f.end = f.first + len;
    if (r.staged) {
        const uint32_t bytes = has ? (lead + len + 15u) & ~15u : 0u;  // the database is padded
        const uint32_t all = __reduce_add_sync(kFull, bytes);
        if (lane == 0) stage_expect(all, f.w + kBarAt);
        __syncwarp();
        if (bytes) bulk_stage(f.w + kDiagAt + c.diag_bytes + to - block, a.res + (mine - lead), bytes, f.w + kBarAt);
    }
    return r;
}

// Zeros around the staged subjects, and for a chunk's reads past the last.
__device__ __forceinline__ void clear_margins(const Finder &f, uint32_t stage) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t first = stage + f.first, end = stage + f.end;
    const uint32_t next = (end + 2u + 15u) & ~15u;  // of the block after the subject's
    if (lane < f.ns) {
        // whole words and then bytes up to the subject, bytes and then whole words behind it
        for (uint32_t i = first & ~15u; i + 4u <= first; i += 4u) sts32(i, 0u);
        for (uint32_t i = first & ~3u; i < first; ++i) smem[i] = 0;
        for (uint32_t i = end; (i & 3u) != 0u; ++i) smem[i] = 0;
        for (uint32_t i = (end + 3u) & ~3u; i < next; i += 4u) sts32(i, 0u);
    }
    const uint32_t last = __shfl_sync(kFull, next, f.ns - 1u);
    sts32(last + 4u * lane, 0u);
    if (lane < kScanStageSlack / 4u - 32u) sts32(last + 128u + 4u * lane, 0u);
    __syncwarp();
}

// The diagonal table as empty: every hit to come is `window` or more past 0.
template <bool QS>
__device__ __forceinline__ void clear_table(Finder &f, const Ctx &c) {
    for (uint32_t i = 4u * (threadIdx.x & 31); i < c.diag_bytes; i += 128u) sts32(f.w + kDiagAt + i, 0u);
    f.base = static_cast<uint32_t>(c.window);
    __syncwarp();
}

// Publishes the init hits in this warp's scratch, each subject's as one block.
__device__ __forceinline__ void publish_group(const Finder &f, const ScanArgs &a, uint32_t lo, uint32_t query_index) {
    const uint32_t lane = threadIdx.x & 31;
    __syncwarp();  // the records in scratch were written by several lanes
    for (uint32_t i = 0; i < f.ns; ++i) {
        const int32_t x0 = static_cast<int32_t>(__shfl_sync(kFull, f.first, i));
        const int32_t x1 = static_cast<int32_t>(__shfl_sync(kFull, f.end, i));
        uint32_t n = 0;
        for (uint32_t i0 = 0; i0 < f.n_init; i0 += 32) {
            const int32_t t = i0 + lane < f.n_init ? scratch_of(a)[i0 + lane].s_trig : -1;
            n += __popc(__ballot_sync(kFull, t >= x0 && t < x1));
        }
        if (n) publish_subject(f, a, lo + i, x0, x1, n, query_index);
    }
}

// More init hits than the warp's scratch holds: the run is repeated with more.
__device__ __forceinline__ void scratch_overflow(const ScanArgs &a, uint32_t n) {
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&a.cnt->overflow_subjects, 1u);
        atomicMax(&a.cnt->max_init_needed, n);
    }
}

// A band of group `g` is done: leaves its init hits (positions in the group,
// which every band counts alike) as a fragment -- a record with the next
// fragment and the number of hits, and the hits -- in the group's list. True
// for the group's last band to finish, whose warp then has all of the group's
// hits in its scratch.
__device__ __forceinline__ bool merge_bands(Finder &f, const ScanArgs &a, uint32_t g, uint32_t n_bands) {
    const uint32_t lane = threadIdx.x & 31;
    BandState *st = a.band_state + g;
    if (f.n_init > a.scratch_cap) {
        scratch_overflow(a, f.n_init);
    } else if (f.n_init > 0) {
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(&a.cnt->fragments, static_cast<unsigned long long>(f.n_init + 1u));
        at = __shfl_sync(kFull, at, 0);
        if (at + f.n_init + 1u <= a.fragment_cap) {
            __syncwarp();
            for (uint32_t i = lane; i < f.n_init; i += 32) a.fragments[at + 1u + i] = scratch_of(a)[i];
            __syncwarp();
            if (lane == 0) {
                InitHit head{};
                head.len = static_cast<int32_t>(f.n_init);
                head.q_start = static_cast<int32_t>(atomicExch(&st->head, static_cast<unsigned int>(at + 1u)));
                a.fragments[at] = head;
            }
        } else if (lane == 0) {
            atomicOr(&a.cnt->flags, kFlagInitArrayFull);
            atomicAdd(&a.cnt->init_count, static_cast<unsigned long long>(f.n_init));
        }
    }
    uint32_t done = 0;
    __syncwarp();
    if (lane == 0) {
        __threadfence();  // the fragment before the count
        done = atomicAdd(&st->done, 1u) + 1u;
        __threadfence();
    }
    done = __shfl_sync(kFull, done, 0);
    if (done != n_bands) return false;
    __syncwarp();  // lane 0's fence holds for every lane's reads from here on (a shuffle orders none)
    uint32_t n = 0;
    const InitHit *frag = a.fragments;
    for (uint32_t next = __ldcg(&st->head); next != 0u;) {
        const uint32_t at = next - 1u, m = static_cast<uint32_t>(__ldcg(&frag[at].len));
        for (uint32_t i = lane; i < m && n + i < a.scratch_cap; i += 32) {
            const int32_t *w = reinterpret_cast<const int32_t *>(frag + at + 1u + i);
            scratch_of(a)[n + i] = InitHit{__ldcg(w), __ldcg(w + 1), __ldcg(w + 2), __ldcg(w + 3), __ldcg(w + 4), __ldcg(w + 5)};
        }
        n += m;
        next = static_cast<uint32_t>(__ldcg(&frag[at].q_start));
    }
    f.n_init = n;
    return true;
}

// A launch's item t: its group, which of the group's bands, and of how many.
// Without bands an item is a group. With them group g's items begin at
// pieces[g] + g x extra_bands: one per piece of its residues (ScanArgs::pieces)
// and the extra ones.
struct Item {
    uint32_t group, band, n_bands;
};
template <bool BANDS>
__device__ __forceinline__ Item item_at(const ScanArgs &a, uint32_t t) {
    if (!BANDS) return Item{t, 0u, 1u};
    uint32_t lo = 0, hi = a.n_groups;  // the last group that begins at or before t is in [lo, hi)
    while (hi - lo > 1u) {
        // the lanes try 32 groups spread over [lo, hi), the first of them lo
        const uint32_t step = (hi - lo + 31u) / 32u, g = lo + step * (threadIdx.x & 31u);
        const bool begun = g < hi && a.pieces[g] + g * a.extra_bands <= t;
        const uint32_t k = __popc(__ballot_sync(kFull, begun)) - 1u;
        hi = min(hi, lo + step * (k + 1u));
        lo += step * k;
    }
    return Item{lo, t - (a.pieces[lo] + lo * a.extra_bands), a.pieces[lo + 1u] - a.pieces[lo] + a.extra_bands};
}

// The fetched subjects for the query of `c`: finds the item's init hits and
// publishes each subject's. False when a staging copy never landed.
template <bool QS, Words W, bool BANDS>
__device__ __forceinline__ bool process_group(Finder &f, const ScanArgs &a, const Ctx &c, const Query<QS, W> &q,
                                              const Group &g, uint32_t query_index, const Item &it) {
    f.n_init = 0;
    f.vb = 0;
    // the values the group's hits take, with the distance to the next group's
    const uint32_t extent = __shfl_sync(kFull, f.end, f.ns - 1u) + static_cast<uint32_t>(c.window) * f.ns;
    if (f.base + extent > Tab<QS>::kMost) clear_table<QS>(f, c);
    const bool long_one = QS ? f.base + extent > Tab<QS>::kMost : extent > kPackSpan - kChunk;
    Band b{0, INT32_MAX, !BANDS || it.n_bands == 1u};
    if (!b.all) {  // equal bands over the diagonals, [0, extent + qlen)
        const unsigned long long span = static_cast<unsigned long long>(extent) + static_cast<uint32_t>(c.qlen);
        b.first = static_cast<int32_t>(span * it.band / it.n_bands);
        b.end = static_cast<int32_t>(span * (it.band + 1u) / it.n_bands);
    }
    if (g.staged) {
        if (!stage_wait(f, a)) return false;
        Span<true> span;
        span.off = f.w + kDiagAt + c.diag_bytes;
        span.ptr = nullptr;
        clear_margins(f, span.off);
        scan_span<QS, W, BANDS>(f, a, c, q, span, long_one, b);
    } else {  // one subject
        Span<false> span;
        span.off = 0;
        span.ptr = a.res + g.o0;
        scan_span<QS, W, BANDS>(f, a, c, q, span, long_one, b);
    }
    if (b.all || merge_bands(f, a, it.group, it.n_bands)) {
        if (f.n_init > a.scratch_cap) scratch_overflow(a, f.n_init);
        else if (f.n_init > 0) publish_group(f, a, g.lo, query_index);
    }
    f.base += extent;
    if (f.hits >> 26) add_counts(f, a);
    __syncwarp();
    return true;
}

// Starts a warp's region at shared offset w.
__device__ __forceinline__ void start_region(Finder &f, uint32_t w) {
    f.w = w;
    f.phase = 0u;
    if ((threadIdx.x & 31) == 0) {
        mbar_init(smem_base() + w + kBarAt);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
}

__device__ __forceinline__ void load_matrix() {
    for (int i = threadIdx.x; i < kAlphabet * kAlphabet; i += blockDim.x)
        reinterpret_cast<int32_t *>(smem + kMatOff)[i] = static_cast<int32_t>(g_blosum8[i]) * (1 << kKeyBits) - 1;
}

// A query's tables in shared memory: its word table or word-presence bitset,
// and its residues.
template <bool QS, Words W>
__device__ __forceinline__ void load_query_tables(const uint32_t *cell_start, const uint32_t *presence,
                                                  const uint8_t *q, int32_t qlen) {
    if (W == Words::kTable) {
        uint16_t *tab = reinterpret_cast<uint16_t *>(smem + kTabOff);
        for (uint32_t i = threadIdx.x; i <= kWords; i += blockDim.x) tab[i] = static_cast<uint16_t>(cell_start[i]);
    } else if (W == Words::kBitset) {
        for (uint32_t i = threadIdx.x; i < kPresenceWords; i += blockDim.x) sts32(kTabOff + 4u * i, presence[i]);
    }
    if (QS)
        for (int i = threadIdx.x; i < qlen; i += blockDim.x) smem[kQueryOff<W> + i] = q[i];
}

// One query against the whole database: the query's word table (or its
// word-presence bitset) and the query itself when short enough live in shared
// memory; warps pull groups, longest subjects first.
template <bool QS, Words W, bool BANDS>
__global__ void __launch_bounds__(kScanMaxWarpsPerBlock * 32, 1)
scan_kernel(const ScanArgs a) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Ctx c;
    c.qlen = a.qlen;
    c.cell_start = a.cell_start;
    c.cell_pack = a.cell_pack;
    c.cell_off = a.cell_off;
    c.diag_entries = a.diag_entries;
    c.diag_magic = a.diag_magic;
    c.diag_bytes = a.diag_bytes;
    c.window = a.window;
    c.xdrop = a.xdrop;
    c.cutoff = a.cutoff;
    c.seed_span = seed_span(a.window);
    Finder f{};
    start_region(f, kQueryOff<W> + a.query_smem_bytes + warp * a.warp_smem_bytes);
    // each warp's first group is its own, the longest subjects spread over the
    // blocks; its copy runs while the block fills its tables
    unsigned long long t = static_cast<unsigned long long>(warp) * gridDim.x + blockIdx.x;
    Group g{};
    Item it{};
    uint32_t hi = 0;
    if (t < a.n_items) {
        it = item_at<BANDS>(a, static_cast<uint32_t>(t));
        hi = a.groups[it.group];
        g = fetch_group(f, a, c, a.groups[it.group + 1], hi, true);
    }
    clear_table<QS>(f, c);
    load_matrix();
    load_query_tables<QS, W>(a.cell_start, a.presence, a.q, a.qlen);
    __syncthreads();
    Query<QS, W> q;
    q.ptr = a.q;
    q.len = a.qlen;
    while (t < a.n_items) {
        if (!process_group<QS, W, BANDS>(f, a, c, q, g, a.query_index, it)) return;
        uint32_t lo = g.lo + f.ns;
        if (lo == hi) {
            if (lane == 0) t = atomicAdd(a.cursor, 1ull) + static_cast<unsigned long long>(gridDim.x) * (blockDim.x >> 5);
            t = __shfl_sync(kFull, t, 0);
            if (t >= a.n_items) break;
            it = item_at<BANDS>(a, static_cast<uint32_t>(t));
            lo = a.groups[it.group + 1];
            hi = a.groups[it.group];
        }
        g = fetch_group(f, a, c, lo, hi, true);
    }
    add_counts(f, a);
}

// Many queries against the database, each with its own cursor over the
// database's groups. A block takes a query, stages its tables, and its warps
// pull groups from the query's cursor until none is left; then it goes on to
// the next query that has any. Blocks start at queries spread over the launch
// and meet at the last ones, so only the launch has an end at which warps wait
// for its longest subjects, not each query's pass: 16 queries of 2,000 to 5,000
// residues against 10.5 M residues with subjects of up to 35,000 take 13.1 ms in
// one launch, and in a launch each 112, or 15.4 in bands. The block lays its warps' regions out
// for each query: a warp's diagonal table takes the query's length plus the
// window, so as many warps as fit (at most the block's) work on it.
template <bool QS, Words W>
__global__ void __launch_bounds__(kScanMaxWarpsPerBlock * 32, 1)
scan_batch_kernel(const ScanArgs a) {
    __shared__ uint32_t s_next;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    load_matrix();
    const uint32_t regions = kQueryOff<W> + a.query_smem_bytes;
    const uint32_t start = static_cast<uint32_t>(static_cast<unsigned long long>(blockIdx.x) * a.n_queries / gridDim.x);
    Finder f{};
    bool staging = true;  // false after a bulk copy that never landed (kFlagBadState is set)
    for (uint32_t from = 0;;) {
        __syncwarp();
        __syncthreads();  // the warps are done with the last query's tables
        if (warp == 0) {
            // the first query from `from` on (counted from the block's start)
            // with groups left; one warp looks, so that the block agrees
            uint32_t next = a.n_queries;
            for (uint32_t i0 = from; i0 < a.n_queries; i0 += 32) {
                bool open = false;
                if (i0 + lane < a.n_queries) {
                    const volatile unsigned long long *cursor = a.cursor + (start + i0 + lane) % a.n_queries;
                    open = *cursor < a.n_groups;
                }
                const unsigned m = __ballot_sync(kFull, open);
                if (m != 0u) {
                    next = i0 + static_cast<uint32_t>(__ffs(m)) - 1u;
                    break;
                }
            }
            if (lane == 0) s_next = next;
            __syncwarp();
        }
        __syncthreads();
        from = s_next;
        if (from == a.n_queries) break;
        const uint32_t qi = (start + from) % a.n_queries;
        const BatchQuery bq = a.queries[qi];
        load_query_tables<QS, W>(bq.cell_start, bq.presence, bq.q, bq.qlen);
        __syncthreads();
        const uint32_t warp_bytes = scan_warp_bytes(bq.diag_bytes, a.stage_bytes);
        const uint32_t active = min(blockDim.x >> 5, (a.smem_bytes - regions) / warp_bytes);  // >= 1 (host)
        if (warp < active) {
            Ctx c;
            c.qlen = bq.qlen;
            c.cell_start = bq.cell_start;
            c.cell_pack = bq.cell_pack;
            c.cell_off = bq.cell_off;
            c.diag_entries = bq.diag_entries;
            c.diag_magic = bq.diag_magic;
            c.diag_bytes = bq.diag_bytes;
            c.window = a.window;
            c.xdrop = a.xdrop;
            c.cutoff = bq.ungapped_cutoff;
            c.seed_span = seed_span(a.window);
            start_region(f, regions + warp * warp_bytes);
            clear_table<QS>(f, c);
            Query<QS, W> q;
            q.ptr = bq.q;
            q.len = bq.qlen;
            for (uint32_t lo = 0, hi = 0;;) {
                if (lo == hi) {
                    unsigned long long t = 0;
                    if (lane == 0) t = atomicAdd(a.cursor + qi, 1ull);
                    t = __shfl_sync(kFull, t, 0);
                    if (t >= a.n_groups) break;
                    lo = a.groups[t + 1];
                    hi = a.groups[t];
                }
                // after a copy that never landed: read this and every later
                // subject from global memory (the host reports the run as failed)
                while (!process_group<QS, W, false>(f, a, c, q, fetch_group(f, a, c, lo, hi, staging), bq.index, Item{}))
                    staging = false;
                lo += f.ns;
            }
            __syncwarp();
            if (lane == 0) mbar_inval(smem_base() + f.w + kBarAt);
            __syncwarp();
        }
    }
    add_counts(f, a);
}

}  // namespace

ScanLayout scan_layout(int32_t qlen, int32_t window, uint32_t n_hits, uint32_t stage_bytes, size_t smem_budget,
                       int max_warps, uint32_t band_entries, bool least) {
    ScanLayout l{};
    const bool smem = scan_query_in_smem(qlen, window, band_entries != 0);
    l.diag_entries = band_entries ? band_entries : scan_diag_entries(qlen, window);
    l.diag_magic = static_cast<uint32_t>((1ull << 32) / l.diag_entries + 1);
    l.diag_bytes = (l.diag_entries * (smem ? 2u : 4u) + 15u) & ~15u;
    l.stage_bytes = stage_bytes;
    l.query_smem_bytes = smem ? (static_cast<uint32_t>(qlen) + 15u) & ~15u : 0u;
    l.warp_smem_bytes = scan_warp_bytes(l.diag_bytes, stage_bytes);
    auto fit = [&](size_t tab) {
        const size_t fixed = kScanMatBytes + tab + l.query_smem_bytes;
        int w = std::max(1, std::min(max_warps, kScanMaxWarpsPerBlock));
        while (w > 1 && fixed + static_cast<size_t>(w) * l.warp_smem_bytes > smem_budget) --w;
        l.warps_per_block = w;
        l.smem_bytes = fixed + static_cast<size_t>(w) * l.warp_smem_bytes;
    };
    l.words = least && !smem ? Words::kPacked : Words::kBitset;
    fit(words_bytes(l.words));
    const int w0 = l.warps_per_block;
    // the word table in shared memory where its 16 bits can number the hits and
    // it costs few warps: 139 M residues at 300 query residues 1.43 -> 1.30 ms
    // and at 1,000 (29 warps of 32) 3.56 -> 3.47, but at 1,500 (22 of 28) 5.05
    // -> 5.34 ms
    constexpr int kWordTabWarps = 28;
    if (l.query_smem_bytes && n_hits <= kScanWordTabHits) {
        fit(kScanWordTabBytes);
        if (l.warps_per_block >= std::min(w0, kWordTabWarps)) l.words = Words::kTable;
        else fit(kScanPresenceBytes);
    }
    return l;
}

// Opts a scan kernel in to the device's full dynamic shared memory, once per
// (device, kernel). The attribute is process-wide: setting it per launch to
// that launch's size would let one host thread lower it between another
// thread's setting and launch, and that launch would then fail.
static cudaError_t allow_full_smem(const void *kernel) {
    static std::mutex mu;
    static std::set<std::pair<int, const void *>> done;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    if (done.count({dev, kernel})) return cudaSuccess;
    int optin = 0;
    cudaFuncAttributes fa{};
    e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    // the dynamic allowance plus the kernel's static shared memory may not
    // exceed the opt-in limit
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, kernel);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 optin - static_cast<int>(fa.sharedSizeBytes));
    if (e == cudaSuccess) done.insert({dev, kernel});
    return e;
}

static void (*single_kernel(bool query_in_smem, Words words, bool bands))(ScanArgs) {
    constexpr Words kBitset = Words::kBitset, kTable = Words::kTable;
    if (bands)
        return !query_in_smem ? scan_kernel<false, kBitset, true>
                              : words == kTable ? scan_kernel<true, kTable, true> : scan_kernel<true, kBitset, true>;
    if (words == Words::kPacked) return scan_kernel<false, Words::kPacked, false>;
    return !query_in_smem ? scan_kernel<false, kBitset, false>
                          : words == kTable ? scan_kernel<true, kTable, false> : scan_kernel<true, kBitset, false>;
}

cudaError_t launch_scan(const ScanArgs &a, Words words, int n_blocks, int warps_per_block, size_t smem_bytes,
                        cudaStream_t st) {
    auto kernel = single_kernel(a.query_smem_bytes != 0, words, a.pieces != nullptr);
    cudaError_t e = allow_full_smem(reinterpret_cast<const void *>(kernel));
    if (e != cudaSuccess) return e;
    kernel<<<n_blocks, warps_per_block * 32, smem_bytes, st>>>(a);
    return cudaGetLastError();
}

// Warps of a block as far as registers go (granted per warp in blocks of 256).
static int max_warps_by_registers(const void *kernel) {
    cudaFuncAttributes fa{};
    if (cudaFuncGetAttributes(&fa, kernel) != cudaSuccess) return kScanMaxWarpsPerBlock;
    int dev = 0, regs_per_block = 65536;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&regs_per_block, cudaDevAttrMaxRegistersPerBlock, dev);
    const int per_warp = ((fa.numRegs * 32 + 255) / 256) * 256;
    return per_warp > 0 ? std::max(1, std::min(kScanMaxWarpsPerBlock, std::min(fa.maxThreadsPerBlock / 32, regs_per_block / per_warp))) : kScanMaxWarpsPerBlock;
}

int scan_max_warps_by_registers(bool query_in_smem) {
    int w = kScanMaxWarpsPerBlock;
    for (bool bands : {false, true})
        for (Words words : {Words::kBitset, Words::kTable})
            w = std::min(w, max_warps_by_registers(reinterpret_cast<const void *>(
                                single_kernel(query_in_smem, words, bands))));
    return w;
}

static void (*batch_kernel(bool query_in_smem, Words words))(ScanArgs) {
    constexpr Words kBitset = Words::kBitset, kTable = Words::kTable;
    if (words == Words::kPacked) return scan_batch_kernel<false, Words::kPacked>;
    return !query_in_smem ? scan_batch_kernel<false, kBitset>
                          : words == kTable ? scan_batch_kernel<true, kTable> : scan_batch_kernel<true, kBitset>;
}

cudaError_t launch_scan_batch(const ScanArgs &a, Words words, int n_blocks, int warps_per_block, size_t smem_bytes,
                              cudaStream_t st) {
    auto kernel = batch_kernel(a.query_smem_bytes != 0, words);
    cudaError_t e = allow_full_smem(reinterpret_cast<const void *>(kernel));
    if (e != cudaSuccess) return e;
    kernel<<<n_blocks, warps_per_block * 32, smem_bytes, st>>>(a);
    return cudaGetLastError();
}

cudaError_t scan_batch_occupancy(bool query_in_smem, Words words, int warps_per_block, size_t smem_bytes,
                                 int *blocks_per_sm) {
    auto kernel = batch_kernel(query_in_smem, words);
    cudaError_t e = allow_full_smem(reinterpret_cast<const void *>(kernel));
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kernel, warps_per_block * 32, smem_bytes);
}

int scan_batch_max_warps_by_registers(bool query_in_smem) {
    const int w = max_warps_by_registers(reinterpret_cast<const void *>(batch_kernel(query_in_smem, Words::kBitset)));
    if (!query_in_smem) return w;
    return std::min(w, max_warps_by_registers(reinterpret_cast<const void *>(batch_kernel(true, Words::kTable))));
}

cudaError_t scan_occupancy(bool query_in_smem, Words words, bool bands, int warps_per_block, size_t smem_bytes,
                           int *blocks_per_sm) {
    auto kernel = single_kernel(query_in_smem, words, bands);
    cudaError_t e = allow_full_smem(reinterpret_cast<const void *>(kernel));
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kernel, warps_per_block * 32,
                                                         smem_bytes);
}

}  // namespace blaze
