// scan.cu -- word finder, two-hit seeding and ungapped X-drop extension of
// the BLASTP preliminary search on GB300 (sm_103a). Integer work only.
//
// One warp per group of subjects; persistent warps pull groups, longest
// subjects first, from a device cursor (batched: blocks pull (query, group
// range) tiles, their warps the tile's groups). Per block in shared memory: the BLOSUM62 matrix
// (int8), the query's word-presence bitset and, for queries up to
// kQuerySmemMax, the query residues. Per warp: the diagonal table, the deferred-hit and seed
// queues and a staging buffer that holds the whole group when it fits, so
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
constexpr int kCoopSeeds = 4;  // flushes with at most this many seeds extend warp-cooperatively
__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

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
template <bool WT>
constexpr uint32_t kQueryOff = kTabOff + (WT ? kScanWordTabBytes : kScanPresenceBytes);
// a warp's region, from Finder::w
constexpr uint32_t kBarAt = 0;                                // the stage buffer's mbarrier
constexpr uint32_t kDeferAt = 16;                             // two buffers of deferred hits
constexpr uint32_t kSeedAt = kDeferAt + 2 * kDeferCap * 4;    // queued seeds
constexpr uint32_t kListAt = kSeedAt + kSeedCap * 8;          // the chunk's words with hits
constexpr uint32_t kDiagAt = kListAt + kChunk * 8;            // diagonal table, then the stage buffer
static_assert(kDiagAt == kScanWarpFixedBytes, "a warp's region");

extern __shared__ __align__(16) unsigned char smem[];

__device__ __forceinline__ uint32_t lds16(uint32_t off) { return *reinterpret_cast<const uint16_t *>(smem + off); }
__device__ __forceinline__ uint32_t lds32(uint32_t off) { return reinterpret_cast<const uint32_t *>(smem)[off >> 2]; }
__device__ __forceinline__ void sts32(uint32_t off, uint32_t v) { reinterpret_cast<uint32_t *>(smem)[off >> 2] = v; }
__device__ __forceinline__ uint2 lds64(uint32_t off) { return reinterpret_cast<const uint2 *>(smem)[off >> 3]; }
__device__ __forceinline__ void sts64(uint32_t off, uint2 v) { reinterpret_cast<uint2 *>(smem)[off >> 3] = v; }
__device__ __forceinline__ int32_t score_of(uint32_t qa, uint32_t sb) {
    return static_cast<int32_t>(reinterpret_cast<const int8_t *>(smem)[kMatOff + qa * kAlphabet + sb]);
}

// ------------------------------------------------------------------------
// Subject staging by the bulk-copy (TMA) engine: one elected lane arms the
// warp's mbarrier with the byte count and issues cp.async.bulk
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

// Lane 0 of the calling warp: copies `bytes` (a multiple of 16) from 16-byte
// aligned global `src` to shared offset `dst` and completes the barrier.
__device__ __forceinline__ void bulk_stage(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    const uint32_t d = smem_base() + dst, b = smem_base() + bar;
    // earlier generic reads of this buffer come before the async overwrite
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(d), "l"(src), "r"(bytes), "r"(b)
                 : "memory");
}

// A group's residues, staged in shared memory, or read from global memory
// when they are longer than the staging buffer. Positions (x) count from the
// group's first residue.
template <bool STAGED>
struct Span {
    uint32_t off;        // shared offset of position 0 (staged)
    const uint8_t *ptr;  // global address of position 0 (not staged)
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
template <bool QSMEM, bool WT>
struct Query {
    const uint8_t *ptr;
    int32_t len;
    __device__ __forceinline__ uint32_t at(int32_t i) const {
        if (QSMEM) return smem[kQueryOff<WT> + i];
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
// Warp-cooperative form of extend_two_hit for one seed: the 32 lanes take 32
// consecutive positions of a walk per step. The running score is a prefix sum
// and the running best a prefix maximum (carried between steps); the walk
// stops at the first position whose stop test holds, and the best is the
// first position reaching the final maximum -- exactly the positions and
// scores of the sequential walk. Every lane returns the same values.

// One X-drop walk of up to n positions; score and best start at `start`.
// t(k) gives the score of the k-th position. Returns the best score; *best_k
// is its position (-1 when never above start), *end the position the walk
// stopped at (n when it ran out). right: also stop when the score drops to 0.
template <bool RIGHT, typename F>
__device__ __forceinline__ int32_t walk_warp(F t, int32_t n, int32_t start, int32_t xdrop, int32_t *best_k,
                                             int32_t *end) {
    const int lane = threadIdx.x & 31;
    int32_t carry = start, cmax = start, bk = -1, stop_at = n;
    for (int32_t base = 0; base < n; base += 32) {
        const int32_t k = base + lane;
        const bool valid = k < n;
        int32_t S = valid ? t(k) : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t x = __shfl_up_sync(kFull, S, o);
            if (lane >= o) S += x;
        }
        S += carry;
        int32_t P = S;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t x = __shfl_up_sync(kFull, P, o);
            if (lane >= o) P = max(P, x);
        }
        P = max(P, cmax);
        const bool stop = valid && ((RIGHT && S <= 0) || P - S >= xdrop);
        const unsigned sm = __ballot_sync(kFull, stop);
        const int last = sm ? __ffs(sm) - 1 : min(31, n - 1 - base);
        const int32_t m = __shfl_sync(kFull, P, last);
        if (m > cmax) {
            const unsigned hm = __ballot_sync(kFull, valid && lane <= last && S == m);
            bk = base + __ffs(hm) - 1;
            cmax = m;
        }
        carry = __shfl_sync(kFull, S, last);
        if (sm) {
            stop_at = base + last;
            break;
        }
    }
    *best_k = bk;
    *end = stop_at;
    return cmax;
}

template <typename Q, typename S>
__device__ __forceinline__ int32_t extend_two_hit_warp(const Q &q, const S &s,
                                                       int32_t s_left_off, int32_t s_off, int32_t q_off,
                                                       int32_t xdrop, int32_t *hsp_q, int32_t *hsp_s,
                                                       int32_t *hsp_len, int32_t *right_extend,
                                                       int32_t *s_last_off) {
    int32_t score = 0, left_score = 0, right_d = 0;
#pragma unroll
    for (int32_t i = 0; i < kWordSize; ++i) {
        score += score_of(q.at(q_off + i), s.at(s_off + i));
        if (score > left_score) {
            left_score = score;
            right_d = i + 1;
        }
    }
    const int32_t q_right = q_off + right_d, s_right = s_off + right_d;
    // left: positions k = 0 .. min(s_right, q_right) - 1 backwards from the
    // residue pair before (q_right, s_right)
    int32_t bk, end;
    left_score = walk_warp<false>(
        [&](int32_t k) { return score_of(q.at(q_right - 1 - k), s.at(s_right - 1 - k)); },
        min(s_right, q_right), 0, xdrop, &bk, &end);
    const int32_t left_d = bk + 1;
    int32_t right_score = 0, rd = 0;
    *right_extend = 0;
    *s_last_off = s_right;
    if (left_d >= s_right - s_left_off) {
        *right_extend = 1;
        int32_t bi, iend;
        right_score = walk_warp<true>(
            [&](int32_t i) { return score_of(q.at(q_right + i), s.at(s_right + i)); },
            min(s.len - s_right, q.len - q_right), left_score, xdrop, &bi, &iend);
        rd = bi + 1;
        *s_last_off = s_right + iend;
    }
    *hsp_q = q_right - left_d;
    *hsp_s = s_right - left_d;
    *hsp_len = left_d + rd;
    return max(left_score, right_score);
}

// ------------------------------------------------------------------------
// Word finder state of one warp. The diagonal table holds, per diagonal
// (x - q) mod L, either the last recorded hit (biased by window and by a
// running base so the table never needs clearing between groups), the end of
// a right extension with kFlag, or kPend | seed slot while that diagonal's
// extension is queued. With L >= qlen + window two diagonals that share an
// entry never both matter: all hits of the later one come more than `window`
// positions after every hit of the earlier one and after the end of any
// extension on it. Each subject of a group adds `window` to the bias, so what
// the subjects before it left in the table is likewise out of reach; only a
// seed still queued for an earlier subject makes a hit on its entry wait.
//
// Entries are 16 bits wide for the queries kept in shared memory, which
// leaves room for twice the warps with long queries (3,000 residues: 24
// instead of 14 per SM, 18.4 -> 11.3 ms for 139 M residues); the
// values then stay below 2^14: the table is cleared before a group that would
// pass it, and moved down (rebase) inside a long subject. Otherwise 32 bits.
//
// Deferred hits and seeds are packed: x and the subject's number in the
// group (or, in a group of one subject, 17 bits of x counted from xb), and q.
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
    uint32_t rel;  // lane i: position of the group's subject i (i <= their number)
    int32_t xb;    // packed positions count from here
    uint32_t xs;   // bits of the subject's number in a packed hit
};

// Per-query parameters of the word finder (one query, or the query of the
// current tile in a batch).
struct Ctx {
    int32_t qlen;
    const uint32_t *cell_start, *cell_pack;
    const uint16_t *cell_off;
    uint32_t diag_entries, diag_magic, diag_bytes;
    int32_t window, xdrop, cutoff;
    uint32_t seed_span;  // distances from the word size on that trigger an extension
};

constexpr int kGroupBits = 5;  // of a subject's number in its group
constexpr int32_t kPackSpan = 1 << 17;
static_assert(kGroupMaxSubjects < 32 && (kGroupMaxResidues << kGroupBits) < kPackSpan, "packed hits");
static_assert(kGroupMaxResidues + (kGroupMaxSubjects + 1) * kTab16Window <= Tab<true>::kMost, "16-bit entries");
static_assert(kQuerySmemMax + kChunk + kTab16Window <= Tab<true>::kMost, "16-bit entries");

__device__ __forceinline__ uint32_t pack_hit(const Finder &f, int32_t x, int32_t q, uint32_t subj) {
    return ((static_cast<uint32_t>(x - f.xb) << f.xs | subj) << 15) | static_cast<uint32_t>(q);
}
struct Hit {
    int32_t x, q;
    uint32_t subj;
};
__device__ __forceinline__ Hit unpack_hit(const Finder &f, uint32_t v) {
    Hit h;
    h.q = static_cast<int32_t>(v & 0x7fffu);
    h.subj = (v >> 15) & ((1u << f.xs) - 1u);
    h.x = static_cast<int32_t>(v >> (15u + f.xs)) + f.xb;
    return h;
}

__device__ __forceinline__ uint32_t defer_at(const Finder &f, uint32_t buf, int i) {
    return f.w + kDeferAt + 4u * (buf * kDeferCap + static_cast<uint32_t>(i));
}
// A seed: the packed hit that triggered it and its distance from the first hit.
__device__ __forceinline__ uint32_t seed_at(const Finder &f, int i) {
    return f.w + kSeedAt + 8u * static_cast<uint32_t>(i);
}
__device__ __forceinline__ uint32_t diag_of(const Ctx &c, int32_t x, int32_t q) {
    return fast_mod(static_cast<uint32_t>(x - q + c.qlen), c.diag_entries, c.diag_magic);
}
// What to add to positions of the group's subject number `subj`.
__device__ __forceinline__ uint32_t bias_of(const Finder &f, const Ctx &c, uint32_t subj) {
    return f.base + static_cast<uint32_t>(c.window) * (subj + 1u);
}
__device__ __forceinline__ InitHit *scratch_of(const ScanArgs &a) {
    const unsigned long long gwarp = (static_cast<unsigned long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    return a.scratch + gwarp * a.scratch_cap;
}

// What a hit does on its diagonal, from the entry's distance below it:
// a flagged entry is further below than any recorded hit, a pending one
// further still (`here` and every entry's value stay within Tab::kMost).
struct Outcome {
    bool set, seed, pend;
};
template <bool QS>
__device__ __forceinline__ Outcome outcome(uint32_t here, uint32_t e, const Ctx &c) {
    const int32_t diff = static_cast<int32_t>(here - e);
    Outcome o;
    // a hit far from the last one starts over, as does the first hit past
    // the end of an extension (the wrapped distances from -kFlag on)
    o.set = diff >= c.window || static_cast<uint32_t>(diff) >= 0u - Tab<QS>::kFlag;
    // one at distance [wordsize, window) triggers an extension; an overlapping
    // one, and one inside the last extension, is ignored
    o.seed = static_cast<uint32_t>(diff - kWordSize) < c.seed_span;
    o.pend = e >= Tab<QS>::kPend;
    return o;
}

// Appends the batch's deferred hits and seeds to their queues, in lane order.
template <bool QS>
__device__ __forceinline__ void queue_hits(Finder &f, bool def, bool seed, int32_t x, int32_t q, uint32_t subj,
                                           int32_t dist, uint32_t entry) {
    const unsigned dm = __ballot_sync(kFull, def);
    const unsigned sm = __ballot_sync(kFull, seed);
    if ((dm | sm) != 0u) {
        const unsigned lt = lanemask_lt();
        const uint32_t packed = pack_hit(f, x, q, subj);
        if (def) sts32(defer_at(f, f.sel, f.n_defer + __popc(dm & lt)), packed);
        __syncwarp();  // a seed's entry overwrites the one its diagonal's first hit just recorded
        if (seed) {
            const int slot = f.n_seed + __popc(sm & lt);
            sts64(seed_at(f, slot), make_uint2(packed, static_cast<uint32_t>(dist)));
            Tab<QS>::store(entry, Tab<QS>::kPend | static_cast<uint32_t>(slot));
        }
        f.n_defer += __popc(dm);
        f.n_seed += __popc(sm);
    }
}

// Runs up to 32 hits (one per lane, lanes in hit order) through the two-hit
// logic. A hit whose diagonal waits on an extension is appended to the
// deferred list. About a quarter of a batch's hits share their diagonal with
// an earlier lane, mostly the next word of the same match (1 or 2 positions
// on). What such a hit does follows from the diagonal's first hit in the
// batch, so most are settled here without another pass over the table:
//   first recorded     1-2 positions on: ignored (so are all hits between);
//                      the second hit, 3 to window on: a seed
//   first seeded       deferred
//   first left the entry as it was: the entry decides for the second hit
//                      too, and for later ones that it makes do nothing
// Only the rest (`hard`) reread the table, one per diagonal at a time. The
// kernel is bound by instruction issue, and one pass over the table per hit
// of a diagonal, as before, took 11.4 warp instructions per residue at 300
// query residues, this form 10.5 (139 M residues: 1.64 -> 1.57 ms; at 1,000
// query residues 4.27 -> 4.06 ms).
template <bool QS>
__device__ __forceinline__ void process_batch(Finder &f, const Ctx &c, bool valid, int32_t x, int32_t q,
                                              uint32_t subj, uint32_t bias) {
    const unsigned lt = lanemask_lt();
    const uint32_t entry = Tab<QS>::at(f.w, diag_of(c, x, q));
    const uint32_t here = static_cast<uint32_t>(x) + bias;
    const unsigned peers = __match_any_sync(kFull, valid ? entry : ~(threadIdx.x & 31u));
    const uint32_t e = valid ? Tab<QS>::load(entry) : here;  // a lane without a hit does nothing
    const unsigned lower = peers & lt;
    const Outcome o = outcome<QS>(here, e, c);
    const bool dup = lower != 0u;
    bool set = o.set && !dup, seed = o.seed && !dup, def = o.pend, hard = false;
    int32_t dist = static_cast<int32_t>(here - e);
    const unsigned dupm = __ballot_sync(kFull, dup);
    if (dupm != 0u) {
        const unsigned setm = __ballot_sync(kFull, set), seedm = __ballot_sync(kFull, seed);
        const uint32_t hf = __shfl_sync(kFull, here, __ffs(peers) - 1);
        if (dup) {
            const unsigned first = peers & (0u - peers);
            const bool second = (lower & (lower - 1u)) == 0u;
            const int32_t df = static_cast<int32_t>(here - hf);
            if ((setm & first) != 0u) {
                seed = second && df >= kWordSize && df < c.window;
                hard = !seed && df >= kWordSize;
                dist = df;
            } else if ((seedm & first) != 0u) {
                def = true;
            } else if (o.set || o.seed) {
                set = second && o.set;
                seed = second && o.seed;
                hard = !second;
            }
        }
    }
    if (set) Tab<QS>::store(entry, here);
    queue_hits<QS>(f, def, seed, x, q, subj, dist, entry);
    __syncwarp();
    if (dupm != 0u) {
        for (unsigned hm = __ballot_sync(kFull, hard); hm != 0u;) {
            const bool mine = hard && (lower & hm) == 0u;
            const uint32_t e2 = mine ? Tab<QS>::load(entry) : here;
            const Outcome o2 = outcome<QS>(here, e2, c);
            if (o2.set) Tab<QS>::store(entry, here);
            queue_hits<QS>(f, o2.pend, o2.seed, x, q, subj, static_cast<int32_t>(here - e2), entry);
            hard = hard && !mine;
            hm = __ballot_sync(kFull, hard);
            __syncwarp();
        }
    }
}

// Extends every queued seed (one lane each), settles their diagonals, keeps
// those reaching the ungapped cutoff, then replays the deferred hits; repeats
// until no seed and no deferred hit is left. Each replay is shorter than the
// list it replays whenever it queues a seed, so the loop ends. Seeds of all
// the group's subjects share a flush: a walk takes about 13 warp instructions
// a step whether one lane or 32 take it, so what an extension costs falls with
// the seeds it shares its flush with.
template <bool QS, bool WT, bool ST>
__device__ __forceinline__ void flush(Finder &f, const ScanArgs &a, const Ctx &c, const Query<QS, WT> &q,
                                      const Span<ST> &span) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = lanemask_lt();
    auto settle = [&](const Hit &h, int32_t first, int32_t rext, int32_t slast) {
        const uint32_t bias = bias_of(f, c, h.subj);
        Tab<QS>::store(Tab<QS>::at(f.w, diag_of(c, h.x, h.q)),
                       rext ? (Tab<QS>::kFlag | (static_cast<uint32_t>(first + slast - (kWordSize - 1)) + bias))
                            : (static_cast<uint32_t>(h.x) + bias));
    };
    auto keep = [&](uint32_t at, const Hit &h, int32_t first, int32_t hq, int32_t hs, int32_t hl, int32_t score) {
        if (at >= a.scratch_cap) return;
        InitHit r;
        r.q_start = hq;
        r.s_start = hs + first;  // positions of the span until the group is published
        r.len = hl;
        r.score = score;
        r.q_trig = h.q;
        r.s_trig = h.x;
        scratch_of(a)[at] = r;
    };
    while (f.n_seed > 0 || f.n_defer > 0) {
        // few seeds: one at a time with the whole warp on each walk
        for (int i = 0; f.n_seed <= kCoopSeeds && i < f.n_seed; ++i) {
            const uint2 sd = lds64(seed_at(f, i));
            const Hit h = unpack_hit(f, sd.x);
            Subject<ST> sub;
            sub.span = span;
            sub.first = __shfl_sync(kFull, f.rel, h.subj);
            sub.len = __shfl_sync(kFull, f.rel, h.subj + 1u) - sub.first;
            const int32_t so = h.x - sub.first;
            int32_t hq, hs, hl, rext, slast;
            const int32_t score = extend_two_hit_warp(q, sub, so - static_cast<int32_t>(sd.y) + kWordSize, so, h.q,
                                                      c.xdrop, &hq, &hs, &hl, &rext, &slast);
            if (lane == 0) {
                settle(h, sub.first, rext, slast);
                if (score >= c.cutoff) keep(f.n_init, h, sub.first, hq, hs, hl, score);
            }
            if (score >= c.cutoff) ++f.n_init;
        }
        // many: one lane per seed
        for (int c0 = 0; f.n_seed > kCoopSeeds && c0 < f.n_seed; c0 += 32) {
            const int i = c0 + lane;
            bool pass = false;
            int32_t hq = 0, hs = 0, hl = 0, score = 0;
            const uint2 sd = lds64(seed_at(f, min(i, f.n_seed - 1)));
            const Hit h = unpack_hit(f, sd.x);
            Subject<ST> sub;
            sub.span = span;
            sub.first = __shfl_sync(kFull, f.rel, h.subj);
            sub.len = __shfl_sync(kFull, f.rel, h.subj + 1u) - sub.first;
            if (i < f.n_seed) {
                const int32_t so = h.x - sub.first;
                int32_t rext, slast;
                score = extend_two_hit(q, sub, so - static_cast<int32_t>(sd.y) + kWordSize, so, h.q, c.xdrop, &hq, &hs,
                                       &hl, &rext, &slast);
                settle(h, sub.first, rext, slast);
                pass = score >= c.cutoff;
            }
            const unsigned pm = __ballot_sync(kFull, pass);
            if (pass) keep(f.n_init + __popc(pm & lt), h, sub.first, hq, hs, hl, score);
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
                const int i = c0 + lane;
                const bool v = i < n_old;
                const Hit h = unpack_hit(f, lds32(defer_at(f, old, v ? i : 0)));
                process_batch<QS>(f, c, v, h.x, h.q, h.subj, bias_of(f, c, h.subj));
            }
        }
    }
}

// Adds the hit and extension counts to the launch's counters.
__device__ __forceinline__ void add_counts(Finder &f, const ScanArgs &a) {
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&a.cnt->word_hits, static_cast<unsigned long long>(f.hits));
        atomicAdd(&a.cnt->extensions, static_cast<unsigned long long>(f.extensions));
    }
    f.hits = f.extensions = 0;
}

// Whether the chunk at cb (of a subject ending at x1) needs a rebase first:
// the values its hits and extensions can reach, or its packed positions, would
// pass their limits. Only a group of one subject ever does.
template <bool QS>
__device__ __forceinline__ bool needs_rebase(const Finder &f, const Ctx &c, int32_t x1, int32_t cb, uint32_t bias) {
    if (QS) return static_cast<uint32_t>(min(x1, cb + kChunk + c.qlen)) + bias > Tab<QS>::kMost;
    return cb - f.xb > kPackSpan - kChunk;
}

// Lets packed positions count from cb and (16-bit entries) moves the table
// down so that a hit at cb has value `window`; an entry that falls below 0 is
// more than `window` behind cb, or an extension's end behind it, and stays so
// as 0. The queues are empty.
template <bool QS>
__device__ __forceinline__ void rebase(Finder &f, const ScanArgs &a, const Ctx &c, int32_t cb, uint32_t &bias) {
    f.xb = cb;
    add_counts(f, a);
    if (!QS) return;
    const uint32_t delta = static_cast<uint32_t>(cb) + bias - static_cast<uint32_t>(c.window);
    for (uint32_t i = threadIdx.x & 31; i < c.diag_entries; i += 32) {
        const uint32_t o = Tab<QS>::at(f.w, i), e = Tab<QS>::load(o), v = e & Tab<QS>::kMost;
        Tab<QS>::store(o, (e & Tab<QS>::kFlag) | (v > delta ? v - delta : 0u));
    }
    f.base -= delta;
    bias -= delta;
    __syncwarp();
}

// 1 << n, 0 from n = 32 on
__device__ __forceinline__ uint32_t bit_at(uint32_t n) {
    uint32_t r;
    asm("shl.b32 %0, 1, %1;" : "=r"(r) : "r"(n));
    return r;
}

// Word scan of a group of ns subjects: chunks of 128 positions, four
// consecutive positions per lane. One warp prefix sum per chunk numbers the
// chunk's hits in (subject offset, query offset) order and the words that have
// any; each such word leaves its position and where its hits lie in the warp's
// list. Lanes then take the hits 32 at a time: a bit mask of the hits that
// start a word gives each lane its word by a population count.
template <bool QS, bool WT, bool ST>
__device__ __forceinline__ void scan_span(Finder &f, const ScanArgs &a, const Ctx &c, const Query<QS, WT> &q,
                                          const Span<ST> &span, uint32_t ns) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t subj = 0; subj < ns; ++subj) {
        const int32_t x0 = static_cast<int32_t>(__shfl_sync(kFull, f.rel, subj));
        const int32_t x1 = static_cast<int32_t>(__shfl_sync(kFull, f.rel, subj + 1u));
        const int32_t xend = x1 - (kWordSize - 1);  // words start below it
        uint32_t bias = bias_of(f, c, subj);
        for (int32_t cb = x0; cb < xend; cb += kChunk) {
            if (needs_rebase<QS>(f, c, x1, cb, bias)) rebase<QS>(f, a, c, cb, bias);
            // the queues are emptied at the group's end and before a rebase
            // (the group's last subject is its longest: it has a chunk if any has)
            const int32_t next = cb + kChunk;
            const bool empty = next < xend ? needs_rebase<QS>(f, c, x1, next, bias) : subj + 1u == ns;
            const int32_t p0 = cb + 4 * static_cast<int32_t>(lane);
            uint32_t r[6];
#pragma unroll
            for (int j = 0; j < 6; ++j) r[j] = span.at(ST ? p0 + j : min(p0 + j, x1 - 1));
            uint32_t cs[4], cnt[4], sum = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool v = p0 + j < xend;
                if (WT) {
                    const uint32_t t = kTabOff + r[j] * 1568u + r[j + 1] * 56u + r[j + 2] * 2u;
                    cs[j] = v ? lds16(t) : 0u;
                    cnt[j] = v ? lds16(t + 2u) - cs[j] : 0u;
                } else {
                    const uint32_t w = r[j] * 784u + r[j + 1] * 28u + r[j + 2];
                    const bool present = v && ((lds32(kTabOff + 4u * (v ? w >> 5 : 0u)) >> (w & 31u)) & 1u);
                    const uint32_t pk = present ? __ldg(c.cell_pack + w) : 0u;
                    cs[j] = pk >> 8;
                    cnt[j] = pk & 0xffu;
                    if (cnt[j] == 0xffu) cnt[j] = __ldg(c.cell_start + w + 1) - cs[j];
                }
                sum += (cnt[j] << 8) + (cnt[j] ? 1u : 0u);  // 24 bits: 128 words of at most 32,000 hits
            }
            uint32_t incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl += y;
            }
            const uint32_t total = __shfl_sync(kFull, incl, 31) >> 8;
            if (total == 0 && !empty) continue;
            f.hits += total;
            uint32_t e[4], run = (incl - sum) >> 8, slot = f.w + kListAt + 8u * ((incl - sum) & 0xffu);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                e[j] = cnt[j] ? run : 0x80000000u;  // the word's first hit
                if (cnt[j]) {
                    sts64(slot, make_uint2(cs[j] - run, static_cast<uint32_t>(p0 + j)));
                    slot += 8u;
                }
                run += cnt[j];
            }
            __syncwarp();
            uint32_t word = f.w + kListAt - 8u;  // the last word begun before the batch
            uint32_t kb = 0;
            do {
                if (kb < total) {
                    const uint32_t m = __reduce_or_sync(
                        kFull, bit_at(e[0] - kb) | bit_at(e[1] - kb) | bit_at(e[2] - kb) | bit_at(e[3] - kb));
                    const uint32_t k = kb + lane;
                    const uint2 wd = lds64(word + 8u * __popc(m & (0xffffffffu >> (31u - lane))));
                    word += 8u * __popc(m);
                    const bool hv = k < total;
                    const int32_t qo = hv ? static_cast<int32_t>(__ldg(c.cell_off + (wd.x + k))) : 0;
                    process_batch<QS>(f, c, hv, static_cast<int32_t>(wd.y), qo, subj, bias);
                }
                kb += 32;
                if (f.n_seed >= 32 || f.n_defer > kDeferCap - 32 || (empty && kb >= total)) flush(f, a, c, q, span);
            } while (kb < total);
        }
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

// A group about to be scanned: its subjects [lo, lo + ns), its residues (at
// o0) and whether they are on their way to the stage buffer.
struct Group {
    uint32_t lo, ns;
    uint64_t o0;
    bool staged;
};

// Reads the bounds of group g and, when it fits and `staging` is on, starts
// its copy to the stage buffer.
__device__ __forceinline__ Group fetch_group(Finder &f, const ScanArgs &a, const Ctx &c, uint32_t g, bool staging) {
    const uint32_t lane = threadIdx.x & 31;
    Group r;
    r.lo = a.groups[g + 1];
    r.ns = a.groups[g] - r.lo;  // 1 .. kGroupMaxSubjects
    const uint64_t mine = a.off[r.lo + min(lane, r.ns)];
    r.o0 = __shfl_sync(kFull, mine, 0);
    f.rel = static_cast<uint32_t>(mine - r.o0);
    const uint32_t len = __shfl_sync(kFull, f.rel, r.ns);
    r.staged = staging && len >= static_cast<uint32_t>(kWordSize) && len <= a.stage_bytes;
    if (r.staged && lane == 0) {
        const uint32_t lead = static_cast<uint32_t>(r.o0 & 15u);
        const uint32_t bytes = (lead + len + 15u) & ~15u;  // the database is padded
        bulk_stage(f.w + kDiagAt + c.diag_bytes, a.res + (r.o0 - lead), bytes, f.w + kBarAt);
    }
    return r;
}

// The diagonal table as empty, values from 0 on.
template <bool QS>
__device__ __forceinline__ void clear_table(Finder &f, const Ctx &c) {
    for (uint32_t i = 4u * (threadIdx.x & 31); i < c.diag_bytes; i += 128u) sts32(f.w + kDiagAt + i, 0u);
    f.base = 0;
    __syncwarp();
}

// The subjects of a fetched group for the query of `c`: finds their init hits
// and publishes each subject's. False when the staging copy never landed.
template <bool QS, bool WT>
__device__ __forceinline__ bool process_group(Finder &f, const ScanArgs &a, const Ctx &c, const Query<QS, WT> &q,
                                              const Group &g, uint32_t query_index) {
    const uint32_t lane = threadIdx.x & 31;
    f.n_init = 0;
    f.xb = 0;
    f.xs = g.ns > 1 ? kGroupBits : 0;
    if (f.base + __shfl_sync(kFull, f.rel, g.ns) + static_cast<uint32_t>(c.window) * (g.ns + 1u) > Tab<QS>::kMost)
        clear_table<QS>(f, c);
    if (g.staged) {
        if (!stage_wait(f, a)) return false;
        Span<true> span;
        span.off = f.w + kDiagAt + c.diag_bytes + static_cast<uint32_t>(g.o0 & 15u);
        span.ptr = nullptr;
        scan_span(f, a, c, q, span, g.ns);
    } else {
        Span<false> span;
        span.off = 0;
        span.ptr = a.res + g.o0;
        scan_span(f, a, c, q, span, g.ns);
    }
    if (f.n_init > a.scratch_cap) {
        if (lane == 0) {
            atomicAdd(&a.cnt->overflow_subjects, 1u);
            atomicMax(&a.cnt->max_init_needed, f.n_init);
        }
    } else if (f.n_init > 0) {
        __syncwarp();  // the records in scratch were written by several lanes
        for (uint32_t i = 0; i < g.ns; ++i) {
            const int32_t x0 = static_cast<int32_t>(__shfl_sync(kFull, f.rel, i));
            const int32_t x1 = static_cast<int32_t>(__shfl_sync(kFull, f.rel, i + 1u));
            uint32_t n = 0;
            for (uint32_t i0 = 0; i0 < f.n_init; i0 += 32) {
                const int32_t t = i0 + lane < f.n_init ? scratch_of(a)[i0 + lane].s_trig : -1;
                n += __popc(__ballot_sync(kFull, t >= x0 && t < x1));
            }
            if (n) publish_subject(f, a, g.lo + i, x0, x1, n, query_index);
        }
    }
    f.base += __shfl_sync(kFull, f.rel, g.ns) + static_cast<uint32_t>(c.window) * g.ns;
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

__device__ __forceinline__ void load_matrix8() {
    for (int i = threadIdx.x; i < kAlphabet * kAlphabet; i += blockDim.x)
        reinterpret_cast<int8_t *>(smem)[kMatOff + i] = g_blosum8[i];
}

// One query against the whole database: the query's word table (or its
// word-presence bitset) and the query itself when short enough live in shared
// memory; warps pull groups, longest subjects first.
template <bool QS, bool WT>
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
    start_region(f, kQueryOff<WT> + a.query_smem_bytes + warp * a.warp_smem_bytes);
    // each warp's first group is its own, the longest subjects spread over the
    // blocks; its copy runs while the block fills its tables
    unsigned long long t = static_cast<unsigned long long>(warp) * gridDim.x + blockIdx.x;
    Group g{};
    if (t < a.n_groups) g = fetch_group(f, a, c, static_cast<uint32_t>(t), true);
    clear_table<QS>(f, c);
    load_matrix8();
    if (WT) {
        uint16_t *tab = reinterpret_cast<uint16_t *>(smem + kTabOff);
        for (uint32_t i = threadIdx.x; i <= kWords; i += blockDim.x) tab[i] = static_cast<uint16_t>(a.cell_start[i]);
    } else {
        for (uint32_t i = threadIdx.x; i < kPresenceWords; i += blockDim.x) sts32(kTabOff + 4u * i, a.presence[i]);
    }
    if (QS)
        for (int i = threadIdx.x; i < a.qlen; i += blockDim.x) smem[kQueryOff<WT> + i] = a.q[i];
    __syncthreads();
    Query<QS, WT> q;
    q.ptr = a.q;
    q.len = a.qlen;
    while (t < a.n_groups) {
        if (!process_group(f, a, c, q, g, a.query_index)) return;
        if (lane == 0) t = atomicAdd(a.cursor, 1ull) + static_cast<unsigned long long>(gridDim.x) * (blockDim.x >> 5);
        t = __shfl_sync(kFull, t, 0);
        if (t < a.n_groups) g = fetch_group(f, a, c, static_cast<uint32_t>(t), true);
    }
    add_counts(f, a);
}

// Many queries against the database: blocks pull (query, group range)
// tiles; tile t covers query t mod n_queries and the (t / n_queries)-th
// range counted from the longest subjects down, so every query's long
// subjects come first and queries interleave. Ranges hold about equal
// residues (host-computed bounds, sized for a whole block). A block stages
// its tile's query tables in shared memory -- the word-presence bitset and,
// up to kQuerySmemMax residues, the query -- and lays its warps' regions out
// for that query: each warp's diagonal table takes the query's length plus
// the window, so as many warps as fit (at most the block's) take the range's
// groups, longest subjects first, from a shared cursor; the others sit the
// tile out. The block restages only after every warp has left the tile. Shared
// memory: matrix, presence bitset, query, then the warps' regions.
template <bool QS>
__global__ void __launch_bounds__(kScanMaxWarpsPerBlock * 32, 1)
scan_batch_kernel(const ScanArgs a) {
    __shared__ unsigned long long s_tile;
    __shared__ uint32_t s_next;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t n_warps = blockDim.x >> 5;
    load_matrix8();
    const uint32_t regions = kQueryOff<false> + a.query_smem_bytes;
    Finder f{};
    const unsigned long long n_tiles = static_cast<unsigned long long>(a.n_ranges) * a.n_queries;
    bool staging = true;  // false after a bulk copy that never landed (kFlagBadState is set)
    for (;;) {
        if (threadIdx.x == 0) {
            s_tile = atomicAdd(a.cursor, 1ull);
            s_next = 0u;
        }
        __syncthreads();  // also orders the previous tile's last table reads before the restage
        const unsigned long long t = s_tile;
        if (t >= n_tiles) break;
        const uint32_t qi = static_cast<uint32_t>(t % a.n_queries);
        const uint32_t range = static_cast<uint32_t>(t / a.n_queries);
        const BatchQuery bq = a.queries[qi];
        for (uint32_t i = threadIdx.x; i < kPresenceWords; i += blockDim.x) sts32(kTabOff + 4u * i, bq.presence[i]);
        if (QS)
            for (int i = threadIdx.x; i < bq.qlen; i += blockDim.x) smem[kQueryOff<false> + i] = bq.q[i];
        __syncthreads();
        const uint32_t warp_bytes = scan_warp_bytes(bq.diag_bytes, a.stage_bytes);
        const uint32_t active = min(n_warps, (a.smem_bytes - kScanSlackBytes - regions) / warp_bytes);  // >= 1 (host)
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
            Query<QS, false> q;
            q.ptr = bq.q;
            q.len = bq.qlen;
            const uint32_t g0 = a.tile_bounds[range], g1 = a.tile_bounds[range + 1];
            for (;;) {
                uint32_t k = 0;
                if (lane == 0) k = atomicAdd(&s_next, 1u);
                k = __shfl_sync(kFull, k, 0);
                if (k >= g1 - g0) break;
                // after a copy that never landed: read this and every later
                // group from global memory (the host reports the run as failed)
                while (!process_group(f, a, c, q, fetch_group(f, a, c, g0 + k, staging), bq.index)) staging = false;
            }
            __syncwarp();
            if (lane == 0) mbar_inval(smem_base() + f.w + kBarAt);
        }
        __syncthreads();
    }
    add_counts(f, a);
}

}  // namespace

ScanLayout scan_layout(int32_t qlen, int32_t window, uint32_t n_hits, uint32_t stage_bytes, size_t smem_budget, int max_warps) {
    ScanLayout l{};
    l.diag_entries = scan_diag_entries(qlen, window);
    l.diag_magic = static_cast<uint32_t>((1ull << 32) / l.diag_entries + 1);
    l.diag_bytes = scan_diag_bytes(qlen, window);
    l.stage_bytes = stage_bytes;
    l.query_smem_bytes = scan_query_in_smem(qlen, window) ? (static_cast<uint32_t>(qlen) + 15u) & ~15u : 0u;
    l.warp_smem_bytes = scan_warp_bytes(l.diag_bytes, stage_bytes);
    auto fit = [&](size_t tab) {
        const size_t fixed = kScanMatBytes + tab + l.query_smem_bytes + kScanSlackBytes;
        int w = std::max(1, std::min(max_warps, kScanMaxWarpsPerBlock));
        while (w > 1 && fixed + static_cast<size_t>(w) * l.warp_smem_bytes > smem_budget) --w;
        l.warps_per_block = w;
        l.smem_bytes = fixed + static_cast<size_t>(w) * l.warp_smem_bytes;
    };
    fit(kScanPresenceBytes);
    const int w0 = l.warps_per_block;
    l.word_table = false;
    // the word table in shared memory where its 16 bits can number the hits and
    // it costs few warps: 139 M residues at 300 query residues 1.43 -> 1.30 ms
    // and at 1,000 (29 warps of 32) 3.56 -> 3.47, but at 1,500 (22 of 28) 5.05
    // -> 5.34 ms
    constexpr int kWordTabWarps = 28;
    if (l.query_smem_bytes && n_hits <= kScanWordTabHits) {
        fit(kScanWordTabBytes);
        l.word_table = l.warps_per_block >= std::min(w0, kWordTabWarps);
        if (!l.word_table) fit(kScanPresenceBytes);
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

static void (*single_kernel(bool query_in_smem, bool word_table))(ScanArgs) {
    return !query_in_smem ? scan_kernel<false, false> : word_table ? scan_kernel<true, true> : scan_kernel<true, false>;
}

cudaError_t launch_scan(const ScanArgs &a, bool word_table, int n_blocks, int warps_per_block, size_t smem_bytes,
                        cudaStream_t st) {
    auto kernel = single_kernel(a.query_smem_bytes != 0, word_table);
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
    const int w = max_warps_by_registers(reinterpret_cast<const void *>(single_kernel(query_in_smem, false)));
    if (!query_in_smem) return w;
    return std::min(w, max_warps_by_registers(reinterpret_cast<const void *>(single_kernel(true, true))));
}

static void (*batch_kernel(bool query_in_smem))(ScanArgs) {
    return query_in_smem ? scan_batch_kernel<true> : scan_batch_kernel<false>;
}

cudaError_t launch_scan_batch(const ScanArgs &a, int n_blocks, int warps_per_block, size_t smem_bytes,
                              cudaStream_t st) {
    auto kernel = batch_kernel(a.query_smem_bytes != 0);
    cudaError_t e = allow_full_smem(reinterpret_cast<const void *>(kernel));
    if (e != cudaSuccess) return e;
    kernel<<<n_blocks, warps_per_block * 32, smem_bytes, st>>>(a);
    return cudaGetLastError();
}

cudaError_t scan_batch_occupancy(bool query_in_smem, int warps_per_block, size_t smem_bytes, int *blocks_per_sm) {
    auto kernel = batch_kernel(query_in_smem);
    cudaError_t e = allow_full_smem(reinterpret_cast<const void *>(kernel));
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kernel, warps_per_block * 32, smem_bytes);
}

int scan_batch_max_warps_by_registers(bool query_in_smem) {
    return max_warps_by_registers(reinterpret_cast<const void *>(batch_kernel(query_in_smem)));
}

cudaError_t scan_occupancy(bool query_in_smem, bool word_table, int warps_per_block, size_t smem_bytes,
                           int *blocks_per_sm) {
    auto kernel = single_kernel(query_in_smem, word_table);
    cudaError_t e = allow_full_smem(reinterpret_cast<const void *>(kernel));
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, kernel, warps_per_block * 32,
                                                         smem_bytes);
}

}  // namespace blaze
