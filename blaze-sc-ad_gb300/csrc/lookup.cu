// lookup.cu -- the query's word lookup built on the device: for each of the
// 28^3 words, the query offsets whose word scores at least the threshold
// against it, or equals it (BLAZE_ncbi/prelim_stage.cpp:135-155, :378-386).
//
// A warp takes the 28 words that begin with one pair of letters and walks the
// query or a part of it, a lane per offset: where the pair's score leaves a
// third letter that can reach the threshold the offset is a candidate (about one
// in twenty at the default), and full batches of candidates are tested against
// the 28 letters, a ballot each. So a word's offsets come out ascending and no
// neighbourhood lists are needed. One pass counts, a block per query turns the
// counts into the tables, a second pass writes the offsets.
// One query's passes are bound by the latency of their steps, 32 offsets each: 8
// and 13 us at 300 query residues, 32 and 65 at 12,345, where a thread per word
// that walked the query alone took 0.5 ms a pass; many queries' by issue: 256 of
// 50 to 2,000 residues 0.62 and 1.18 ms (0.86 and 1.74 with a block and eight
// parts for every pair and query).
#include <algorithm>
#include <cstdint>

#include "common.cuh"

namespace blaze {
namespace {

__device__ const int32_t g_blosum_lk[kAlphabet * kAlphabet] = {
#include "blosum62.inc"
};

constexpr unsigned kFull = 0xffffffffu;
constexpr int kLookupWarps = 8;                // per block: pairs of letters times parts of the query
constexpr int kPartLeast = 256;                // offsets of a part: a test of the 28 letters costs the same for
                                               // one candidate and 32, so parts are not cut smaller
constexpr int kPairs = kAlphabet * kAlphabet;  // pairs of letters
constexpr int kRow = kAlphabet + 1;            // of the matrix in shared memory: an odd stride, so that the
                                               // lanes' rows lie in different banks

static_assert(kPairs % kLookupWarps == 0);

// A block's work on a query with `all` offsets: the parts that the query is cut
// in, a warp each, and so how many pairs the block takes.
struct Split {
    int32_t all, parts, part;
    uint32_t pairs;
    __device__ __forceinline__ explicit Split(int32_t qlen) : all(max(qlen - (kWordSize - 1), 0)), parts(1) {
        while (parts < kLookupWarps && all > parts * kPartLeast) parts *= 2;
        part = ((all + parts - 1) / parts + 31) & ~31;
        pairs = kLookupWarps / parts;
    }
    __device__ __forceinline__ bool idle() const { return blockIdx.x * pairs >= kPairs; }
    __device__ __forceinline__ uint32_t pair() const { return blockIdx.x * pairs + (threadIdx.x >> 5) / parts; }
    __device__ __forceinline__ uint32_t mine() const { return (threadIdx.x >> 5) % parts; }  // the warp's part
};

struct WalkShared {
    int32_t mat[kAlphabet * kRow];
    int32_t best[kAlphabet];          // of a row
    uint32_t cand[kLookupWarps][64];  // offset | third letter << 16 | starts with the pair << 31
    int32_t cand_score[kLookupWarps][64];
    uint32_t count[kLookupWarps][32];  // by third letter
};

__device__ __forceinline__ void walk_setup(WalkShared &sh) {
    for (int i = threadIdx.x; i < kPairs; i += blockDim.x)
        sh.mat[i / kAlphabet * kRow + i % kAlphabet] = g_blosum_lk[i];
    __syncthreads();
    if (threadIdx.x < kAlphabet) {
        int32_t m = sh.mat[threadIdx.x * kRow];
        for (int k = 1; k < kAlphabet; ++k) m = max(m, sh.mat[threadIdx.x * kRow + k]);
        sh.best[threadIdx.x] = m;
    }
    __syncthreads();
}

// The warp's part of the query: calls hit(c, mask, i) for each third letter c from 1
// and batch of candidates: the lanes in mask have the word's offset i. Every
// lane makes every call.
template <typename F>
__device__ __forceinline__ void walk_query(WalkShared &sh, const LookupQuery &lq, const Split &sp, int32_t threshold, F hit) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t a = sp.pair() / kAlphabet, b = sp.pair() % kAlphabet;
    const int32_t *mat = sh.mat;
    uint32_t *cand = sh.cand[warp];
    int32_t *cand_score = sh.cand_score[warp];
    const int32_t from = min(sp.part * static_cast<int32_t>(sp.mine()), sp.all);
    const int32_t n = a > 0u && b > 0u ? min(from + sp.part, sp.all) : from;  // no word with the letter 0 has hits
    uint32_t have = 0;
    auto test = [&](uint32_t m) {  // the first m candidates
        const bool in = lane < m;
        const uint32_t w = in ? cand[lane] : 0u;
        const int32_t s = in ? cand_score[lane] : 0;
        const uint32_t z = (w >> 16) & 31u;
        const bool same = (w >> 31) != 0u;
#pragma unroll 4
        for (uint32_t c = 1; c < kAlphabet; ++c) {
            const bool h = in && (s + mat[z * kRow + c] >= threshold || (same && z == c));
            hit(c, __ballot_sync(kFull, h), w & 0xffffu);
        }
    };
    for (int32_t i0 = from; i0 < n; i0 += 32) {
        const int32_t i = i0 + static_cast<int32_t>(lane);
        bool is = false, same = false;
        uint32_t z = 0;
        int32_t s = 0;
        if (i < n) {
            const uint32_t x = lq.q[i], y = lq.q[i + 1];
            z = lq.q[i + 2];
            s = mat[x * kRow + a] + mat[y * kRow + b];
            same = x == a && y == b;
            is = same || s + sh.best[z] >= threshold;
        }
        const uint32_t m = __ballot_sync(kFull, is);
        if (is) {
            const uint32_t at = have + __popc(m & ((1u << lane) - 1u));
            cand[at] = static_cast<uint32_t>(i) | (z << 16) | (same ? 0x80000000u : 0u);
            cand_score[at] = s;
        }
        have += __popc(m);
        __syncwarp();
        if (have >= 32u) {
            test(32u);
            have -= 32u;
            __syncwarp();
            const uint32_t w = cand[32u + lane];
            const int32_t ws = cand_score[32u + lane];
            if (lane < have) {
                cand[lane] = w;
                cand_score[lane] = ws;
            }
            __syncwarp();
        }
    }
    if (have) test(have);
}

// The warps' counts, by third letter.
__device__ __forceinline__ void walk_count(WalkShared &sh, const LookupQuery &lq, const Split &sp, int32_t threshold) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t n = 0;  // lane c: of the word with third letter c
    walk_query(sh, lq, sp, threshold, [&](uint32_t c, uint32_t mask, uint32_t) { n += lane == c ? __popc(mask) : 0; });
    sh.count[threadIdx.x >> 5][lane] = n;
    __syncthreads();
}

// Counts of every word, left in cell_start.
__global__ void __launch_bounds__(kLookupWarps * 32)
lookup_count_kernel(const LookupQuery one, const LookupQuery *many, int32_t threshold) {
    __shared__ WalkShared sh;
    const LookupQuery lq = many ? many[blockIdx.y] : one;
    const Split sp(lq.qlen);
    if (sp.idle()) return;
    walk_setup(sh);
    walk_count(sh, lq, sp, threshold);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (sp.mine() == 0u && lane < kAlphabet) {
        uint32_t n = 0;
        for (int p = 0; p < sp.parts; ++p) n += sh.count[warp + p][lane];
        lq.cell_start[sp.pair() * kAlphabet + lane] = n;
    }
}

// One block per query: starts, packed cells (start << 8 | min(count, 255), or 255
// where the start takes more than 24 bits: 4,900 residues at word threshold 0) and
// the presence bitset from the counts. A warp takes 22 rows of 32 consecutive
// words, so every access is coalesced and a row's presence is a ballot (a run
// of words per thread instead took 38 us for one query).
__global__ void __launch_bounds__(1024) lookup_tables_kernel(const LookupQuery one, const LookupQuery *many) {
    constexpr uint32_t kRows = (kPresenceWords + 31) / 32;
    static_assert(kRows * 1024 >= kWords);
    __shared__ uint32_t warp_sum[32];
    const LookupQuery lq = many ? many[blockIdx.x] : one;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t w0 = warp * kRows * 32u + lane;
    uint32_t n[kRows], sum = 0;
#pragma unroll
    for (uint32_t k = 0; k < kRows; ++k) {
        n[k] = w0 + k * 32u < kWords ? lq.cell_start[w0 + k * 32u] : 0u;
        sum += n[k];
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0u) warp_sum[warp] = sum;
    __syncthreads();  // also: every count is read before a start replaces it
    uint32_t start = __reduce_add_sync(0xffffffffu, lane < warp ? warp_sum[lane] : 0u);
    if (warp == 31u && lane == 0u) lq.cell_start[kWords] = start + sum;
#pragma unroll
    for (uint32_t k = 0; k < kRows; ++k) {
        uint32_t incl = n[k];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= static_cast<uint32_t>(o)) incl += x;
        }
        const uint32_t w = w0 + k * 32u, at = start + incl - n[k];
        const uint32_t bits = __ballot_sync(0xffffffffu, n[k] != 0u);
        if (w < kWords) {
            lq.cell_start[w] = at;
            lq.cell_pack[w] = at < (1u << 24) ? (at << 8) | min(n[k], 255u) : 255u;
        }
        if (lane == 0u && w / 32u < kPresenceWords) lq.presence[w / 32u] = bits;
        start += __shfl_sync(0xffffffffu, incl, 31);
    }
}

// The offsets; where there are several parts a warp counts its own first, for
// where the next one's begin.
__global__ void __launch_bounds__(kLookupWarps * 32)
lookup_write_kernel(const LookupQuery one, const LookupQuery *many, int32_t threshold) {
    __shared__ WalkShared sh;
    const LookupQuery lq = many ? many[blockIdx.y] : one;
    const Split sp(lq.qlen);
    if (sp.idle()) return;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    walk_setup(sh);
    if (sp.parts > 1) walk_count(sh, lq, sp, threshold);
    uint32_t to = 0;  // lane c: where the next offset of its word goes
    if (lane < kAlphabet) {
        to = lq.cell_start[sp.pair() * kAlphabet + lane];
        for (uint32_t w = warp - sp.mine(); w < warp; ++w) to += sh.count[w][lane];
    }
    walk_query(sh, lq, sp, threshold, [&](uint32_t c, uint32_t mask, uint32_t i) {
        const uint32_t at = __shfl_sync(kFull, to, c) + __popc(mask & ((1u << lane) - 1u));
        if ((mask >> lane) & 1u) lq.cell_off[at] = static_cast<uint16_t>(i);
        to += lane == c ? __popc(mask) : 0;
    });
}

}  // namespace

cudaError_t launch_lookup(const LookupQuery &one, const LookupQuery *many, uint32_t n, int32_t threshold,
                          cudaStream_t st) {
    constexpr uint32_t kBlocks = kPairs;
    constexpr uint32_t kMost = 32768;  // queries per launch (the grid's y extent)
    for (uint32_t i = 0; i < n; i += kMost) {
        const LookupQuery *m = many ? many + i : nullptr;
        const uint32_t k = std::min(n - i, kMost);
        lookup_count_kernel<<<dim3(kBlocks, k), kLookupWarps * 32, 0, st>>>(one, m, threshold);
        lookup_tables_kernel<<<k, 1024, 0, st>>>(one, m);
        lookup_write_kernel<<<dim3(kBlocks, k), kLookupWarps * 32, 0, st>>>(one, m, threshold);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace blaze
