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
// the presence bitset from the counts.
__global__ void __launch_bounds__(1024) lookup_tables_kernel(const LookupQuery one, const LookupQuery *many) {
    __shared__ uint16_t count[kWords];  // at most 32,000 offsets
    __shared__ uint32_t warp_sum[32];
    const LookupQuery lq = many ? many[blockIdx.x] : one;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    for (uint32_t w = tid; w < kWords; w += 1024u) count[w] = static_cast<uint16_t>(lq.cell_start[w]);
    __syncthreads();
    constexpr uint32_t kEach = (kWords + 1023) / 1024;
    const uint32_t w0 = min(tid * kEach, static_cast<uint32_t>(kWords)), w1 = min(w0 + kEach, static_cast<uint32_t>(kWords));
    uint32_t sum = 0;
    for (uint32_t w = w0; w < w1; ++w) sum += count[w];
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= static_cast<uint32_t>(o)) incl += x;
    }
    if (lane == 31u) warp_sum[warp] = incl;
    __syncthreads();
    uint32_t start = incl - sum;
    for (uint32_t i = 0; i < warp; ++i) start += warp_sum[i];
    for (uint32_t w = w0; w < w1; ++w) {
        const uint32_t n = count[w];
        lq.cell_start[w] = start;
        lq.cell_pack[w] = (start << 8) | min(n, 255u);
        start += n;
    }
    if (tid == 1023u) lq.cell_start[kWords] = start;
    for (uint32_t p = tid; p < kPresenceWords; p += 1024u) {
        uint32_t bits = 0;
        for (uint32_t k = 0; k < 32u && p * 32u + k < kWords; ++k) bits |= (count[p * 32u + k] ? 1u : 0u) << k;
        lq.presence[p] = bits;
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
