// lookup.cu -- the query's word lookup built on the device: for each of the
// 28^3 words, the query offsets whose word scores at least the threshold
// against it, or equals it (BLAZE_ncbi/prelim_stage.cpp:135-155, :378-386).
//
// One thread per word walks the query, so a word's offsets come out ascending
// and no neighbourhood lists are needed: 21,952 threads x the query's length
// x about ten instructions, a few microseconds for a protein. One pass counts,
// a block per query turns the counts into the tables, a second pass writes the
// offsets. Built on the host instead, a 350-residue query's call over a proteome
// took 542 us against 470, and 64 queries arriving at a server 29.8 ms against
// 29.0.
#include <algorithm>
#include <cstdint>

#include "common.cuh"

namespace blaze {
namespace {

__device__ const int32_t g_blosum_lk[kAlphabet * kAlphabet] = {
#include "blosum62.inc"
};

constexpr int kLookupThreads = 256;
constexpr int kLookupTile = 512;  // query offsets staged at a time

// A query offset's word as the walk reads it: its letters' rows in the matrix
// (byte offsets) and the word itself.
struct Pos {
    uint32_t row0, row1, row2, word;
};

// Calls hit(i) for each query offset i whose word is in the thread's cell.
template <typename F>
__device__ __forceinline__ void walk_query(const LookupQuery &lq, int32_t threshold, uint32_t word, F hit) {
    __shared__ int32_t mat[kAlphabet * kAlphabet];
    __shared__ Pos tile[kLookupTile];
    for (int i = threadIdx.x; i < kAlphabet * kAlphabet; i += blockDim.x) mat[i] = g_blosum_lk[i];
    const int32_t n = lq.qlen - (kWordSize - 1);
    const uint32_t a = min(word / 784u, 27u), b = word / 28u % 28u, c = word % 28u;
    const int32_t *m0 = mat + a, *m1 = mat + b, *m2 = mat + c;
    for (int32_t i0 = 0; i0 < n; i0 += kLookupTile) {
        __syncthreads();
        const int32_t m = min(n - i0, kLookupTile);
        for (int32_t i = threadIdx.x; i < m; i += blockDim.x) {
            const uint8_t *q = lq.q + i0 + i;
            const uint32_t x = q[0], y = q[1], z = q[2];
            tile[i] = Pos{x * kAlphabet, y * kAlphabet, z * kAlphabet, x * 784u + y * 28u + z};
        }
        __syncthreads();
#pragma unroll 4
        for (int32_t i = 0; i < m; ++i) {
            const Pos p = tile[i];
            if (m0[p.row0] + m1[p.row1] + m2[p.row2] >= threshold || p.word == word) hit(i0 + i);
        }
    }
}

// Counts of every word, left in cell_start.
__global__ void __launch_bounds__(kLookupThreads)
lookup_count_kernel(const LookupQuery one, const LookupQuery *many, int32_t threshold) {
    const LookupQuery lq = many ? many[blockIdx.y] : one;
    const uint32_t word = blockIdx.x * kLookupThreads + threadIdx.x;
    uint32_t n = 0;
    walk_query(lq, threshold, word, [&](int32_t) { ++n; });
    if (word < static_cast<uint32_t>(kWords)) lq.cell_start[word] = n;
}

// One block per query: starts, packed cells (start << 8 | min(count, 255)) and
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
            lq.cell_pack[w] = (at << 8) | min(n[k], 255u);
        }
        if (lane == 0u && w / 32u < kPresenceWords) lq.presence[w / 32u] = bits;
        start += __shfl_sync(0xffffffffu, incl, 31);
    }
}

__global__ void __launch_bounds__(kLookupThreads)
lookup_write_kernel(const LookupQuery one, const LookupQuery *many, int32_t threshold) {
    const LookupQuery lq = many ? many[blockIdx.y] : one;
    const uint32_t word = blockIdx.x * kLookupThreads + threadIdx.x;
    uint16_t *out = lq.cell_off + (word < static_cast<uint32_t>(kWords) ? lq.cell_start[word] : 0u);
    const bool own = word < static_cast<uint32_t>(kWords);
    walk_query(lq, threshold, word, [&](int32_t i) {
        if (own) *out++ = static_cast<uint16_t>(i);
    });
}

}  // namespace

cudaError_t launch_lookup(const LookupQuery &one, const LookupQuery *many, uint32_t n, int32_t threshold,
                          cudaStream_t st) {
    constexpr uint32_t kBlocks = (kWords + kLookupThreads - 1) / kLookupThreads;
    constexpr uint32_t kMost = 32768;  // queries per launch (the grid's y extent)
    for (uint32_t i = 0; i < n; i += kMost) {
        const LookupQuery *m = many ? many + i : nullptr;
        const uint32_t k = std::min(n - i, kMost);
        lookup_count_kernel<<<dim3(kBlocks, k), kLookupThreads, 0, st>>>(one, m, threshold);
        lookup_tables_kernel<<<k, 1024, 0, st>>>(one, m);
        lookup_write_kernel<<<dim3(kBlocks, k), kLookupThreads, 0, st>>>(one, m, threshold);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace blaze
