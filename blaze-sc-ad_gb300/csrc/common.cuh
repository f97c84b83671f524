// common.cuh -- internal types shared by the host driver and the kernels of
// libblaze103 (GB300 / sm_103a BLASTP preliminary stage).
#pragma once

#include <cstdint>
#include <climits>

#include <cuda_runtime.h>

#include "blaze_prelim.h"

namespace blaze {

constexpr int kAlphabet = 28;
constexpr int kWords = kAlphabet * kAlphabet * kAlphabet;  // 21952 three-letter words
constexpr int kWordSize = 3;
constexpr int32_t kNeg = INT32_MIN / 2;  // "minus infinity" of the gapped DP
constexpr int kWarp = 32;

// Word-finder tuning (per warp of the scan kernel).
constexpr int kDeferCap = 64;   // deferred hits per buffer (two buffers)
constexpr int kSeedCap = 64;    // queued two-hit seeds (>= kDeferCap)
constexpr int kChunk = 128;     // subject positions a warp looks up at a time
// a warp's region up to its diagonal table: mbarrier, deferred hits (two
// buffers), seeds, words with hits
constexpr uint32_t kScanWarpFixedBytes = 16 + 2 * kDeferCap * 4 + kSeedCap * 8 + (kChunk + 32) * 8;
constexpr uint32_t kScanStageSlack = 144;  // zeros behind the staged subjects: a chunk's reads end there
// A group: consecutive subjects that one warp stages and scans together.
constexpr uint32_t kGroupMaxSubjects = 31;    // their bounds are one per lane, with the end
constexpr uint32_t kGroupSubjectBytes = 32;   // of a subject's block beyond its residues, at most
constexpr uint32_t kGroupMaxBytes = 2240;     // of the blocks of a group of several subjects
__host__ __device__ constexpr uint32_t scan_stage_blocks(uint32_t stage_bytes) { return (stage_bytes + 32u + 15u) & ~15u; }
constexpr int kScanMaxWarpsPerBlock = 32;
constexpr int kGappedWarpsPerBlock = 4;
constexpr int kPresenceWords = (kWords + 31) / 32;                     // 686
constexpr size_t kScanMatBytes = kAlphabet * kAlphabet * 4;           // matrix, 3,136
constexpr size_t kScanPresenceBytes = (kPresenceWords * 4 + 15) & ~15; // 2752
constexpr size_t kScanWordTabBytes = ((kWords + 1) * 2 + 15) & ~15;    // 43,920
// Where the scan looks a word up: in a table of the hit lists' starts in shared
// memory, in the packed cells of words whose bit is set in a bitset there, or in
// the packed cells alone, which leaves the longest diagonal tables the most room.
enum class Words { kBitset, kTable, kPacked };
__host__ __device__ constexpr uint32_t words_bytes(Words w) {
    return static_cast<uint32_t>(w == Words::kTable ? kScanWordTabBytes : w == Words::kBitset ? kScanPresenceBytes : 0);
}
constexpr uint32_t kScanWordTabHits = 65535;  // hit-list entries a 16-bit word table can number
constexpr int32_t kQuerySmemMax = 11776;      // queries up to this length live in shared memory,
constexpr int32_t kBandQuerySmemMax = 14336;  // in bands this one,
constexpr int32_t kTab16Window = 256;        // for windows up to this one: 16-bit diagonal tables
// Diagonals of a band where its table holds no more, by the width of its
// entries: 12,345 residues against 140 M with 16-bit tables of 2,240 / 3,360 /
// 4,480 / 6,720 entries 70.5 / 62.2 / 64.8 / 78.4 ms, 16,000 with 32-bit ones
// 120 / 130 / 147 / 173
constexpr uint32_t kBandEntries16 = 3360, kBandEntries32 = 2240;
static_assert(kBandEntries32 >= kGroupMaxBytes && kBandEntries16 >= kGroupMaxBytes, "a group is one piece");
constexpr uint32_t kPieceLeast = 128, kPieceMost = kGroupMaxBytes;  // residues of a long subject's piece
constexpr int32_t kBandQuery = 7000;         // longer queries take such tables
constexpr int32_t kStageQuery = 1300;        // longer ones stage parts of a group
constexpr uint32_t kScanStageBytes = 1024;   // subjects up to this length are staged

// Whether the register-window DPs of `rows` rows (gapped stage, traceback) stay
// inside int32 and below -inf's distance. They compute the columns behind the
// band as well, up to a window of them: those hold -inf, which an X-drop of 2^30
// would call live, and enter the row gap's prefix maximum as -inf plus gap_extend
// times their column. A band's last column is at most rows + (11 rows + xdrop) /
// gap_extend + 2 (11: the matrix's largest score). Other DPs take the form with
// their rows in memory.
__device__ __forceinline__ bool dp_window_exact(int32_t rows, int32_t gap_open, int32_t gap_extend, int32_t xdrop) {
    constexpr long long kBehind = 256;
    const long long ge = gap_extend, goe = ge + gap_open, drop = xdrop > goe ? xdrop : goe;
    return ge * (rows + kBehind) + 2 * drop + 22ll * rows <= -static_cast<long long>(kNeg);
}

inline bool scan_query_in_smem(int32_t qlen, int32_t window, bool bands = false) {
    return qlen <= (bands ? kBandQuerySmemMax : kQuerySmemMax) && window <= kTab16Window;
}
inline uint32_t scan_band_entries(int32_t qlen) { return qlen <= kBandQuerySmemMax ? kBandEntries16 : kBandEntries32; }
inline uint32_t scan_diag_entries(int32_t qlen, int32_t window) {  // >= qlen + window
    return static_cast<uint32_t>(qlen + window + 3) & ~3u;
}
inline uint32_t scan_diag_bytes(int32_t qlen, int32_t window) {
    return (scan_diag_entries(qlen, window) * (scan_query_in_smem(qlen, window) ? 2u : 4u) + 15u) & ~15u;
}
__host__ __device__ constexpr uint32_t scan_warp_bytes(uint32_t diag_bytes, uint32_t stage_bytes) {
    return kScanWarpFixedBytes + diag_bytes + scan_stage_blocks(stage_bytes) + kScanStageSlack;
}

// An ungapped HSP that reached the ungapped cutoff (NCBI BlastInitHSP analog).
struct InitHit {
    int32_t q_start, s_start, len, score;
    int32_t q_trig, s_trig;  // the second word hit that triggered the extension
};

// One subject with init hits, for the gapped kernel.
struct WorkItem {
    uint32_t subject;  // index into the length-sorted database
    uint32_t n_init;
    uint64_t first;    // first record in the init-hit array
};

// One init hit's gapped extension as a DP task: the subject, the
// query (batched: its index) and the gapped start point. Written by the prep
// kernel at the init hit's slot; valid = 0 for an init hit that is skipped.
struct DpTask {
    uint64_t s_base;  // offset of the subject's residues
    int32_t slen;
    uint32_t query;
    int32_t q_off, s_off;
    int32_t valid;
    int32_t rank;  // of its init hit in its item (0: the best)
    uint64_t item;
};

// A finished gapped HSP as the device writes it (subject = sorted index).
struct DevHsp {
    uint32_t subject;
    int32_t score, q_start, q_end, s_start, s_end, q_gs, s_gs;
};

// The bands of one group of a scan launch: its fragments of init hits (index + 1
// of the last one's record, 0: none) and the bands that are done. Zeroed before
// the launch.
struct BandState {
    unsigned int head, done;
};

// Device counters of one run; zeroed before every run.
struct DevCounters {
    unsigned long long init_count;   // init hits published
    unsigned long long work_count;   // work items published
    unsigned long long out_count;    // HSPs published
    unsigned long long next_gapped;  // gapped-kernel work cursor
    unsigned long long word_hits;
    unsigned long long extensions;
    unsigned long long gapped_ext;
    unsigned long long dp_cells;
    unsigned int overflow_subjects;  // subjects whose init hits exceeded the per-warp scratch
    unsigned int max_init_needed;    // largest init-hit count among those
    unsigned int flags;              // kFlag* bits
    unsigned int pad;
    unsigned long long group_count;  // subject HSP lists published (GroupDesc records)
    unsigned long long next_prep;    // gapped prep-kernel work cursor
    unsigned long long next_dp;      // DP task cursor
    unsigned long long fragments;    // records taken in ScanArgs::fragments
    unsigned long long n_first, n_rest;  // DP tasks: items' best init hits, the others
};

// One subject's HSP list in the gapped stage's output, after the preliminary
// E-value reap and max_hsps: `n` HSPs from `first`, best first. The hit-list
// selection sets n to 0 for a subject outside its query's hitlist_size.
struct GroupDesc {
    unsigned long long first;
    uint32_t query;    // batched runs: the query's position in its batch
    uint32_t subject;  // index into the length-sorted database
    uint32_t oid;
    uint32_t n;
    int32_t best;      // score of the list's first HSP
    uint32_t pad;
};

constexpr unsigned kFlagInitArrayFull = 1u;
constexpr unsigned kFlagWorkArrayFull = 2u;
constexpr unsigned kFlagOutArrayFull = 4u;
constexpr unsigned kFlagSavedFull = 8u;
constexpr unsigned kFlagBadState = 16u;
constexpr unsigned kFlagSubjectTooLong = 32u;  // gapped: a subject longer than its DP rows was skipped
constexpr unsigned kFlagBadInitHit = 64u;      // gapped: an init hit outside its query or subject was skipped

// One query of a batch, as the batched scan kernel reads it.
struct BatchQuery {
    const uint8_t *q;
    int32_t qlen;
    int32_t ungapped_cutoff;
    const uint32_t *cell_start, *cell_pack, *presence;
    const uint16_t *cell_off;
    uint32_t diag_entries, diag_magic, diag_bytes;
    uint32_t index;  // position of the query in its batch
};

// A query's word lookup on the device: where its residues are and its tables
// go (cell_start: kWords + 1 prefix offsets; cell_pack: start << 8 | min(count,
// 255), a count of 255 sends the kernel to cell_start for both, and stands for
// every cell whose start is 2^24 or more; presence: kPresenceWords; cell_off:
// lookup_hits query offsets).
struct LookupQuery {
    const uint8_t *q;
    int32_t qlen;
    uint32_t *cell_start, *cell_pack, *presence;
    uint16_t *cell_off;
};

struct ScanArgs {
    const uint8_t *res;        // residues, length-sorted subjects
    const uint64_t *off;       // n_subj + 1 offsets
    const uint32_t *groups;    // n_groups + 1 subject indices, descending: group g is [groups[g+1], groups[g])
    uint32_t n_groups;
    // a single-query launch in bands (null: without): prefix sums over the groups
    // of their pieces; the bands of a group beyond one per piece; per group
    // state; fragments of init hits
    const uint32_t *pieces;
    uint32_t extra_bands;
    uint32_t n_items;          // groups, or bands
    BandState *band_state;
    InitHit *fragments;
    unsigned long long fragment_cap;
    const uint8_t *q;          // query residues
    int32_t qlen;
    const uint32_t *cell_start;  // kWords + 1
    const uint32_t *cell_pack;   // kWords: as LookupQuery
    const uint32_t *presence;    // kPresenceWords: bit w set when word w has hits
    const uint16_t *cell_off;    // query offsets per cell, ascending
    int32_t window, xdrop, cutoff;
    uint32_t diag_entries;       // >= qlen + window, or the diagonals of a band
    uint32_t diag_magic;         // floor(2^32 / diag_entries) + 1
    uint32_t diag_bytes, stage_bytes, query_smem_bytes, warp_smem_bytes;
    uint32_t smem_bytes;         // batched launches: dynamic shared memory of a block
    // batched launches only
    const BatchQuery *queries;   // n_queries descriptors
    uint32_t n_queries;
    uint32_t *work_query;        // query index of each work item (nullptr: one query)
    uint32_t query_index;        // single-query launches inside a batched pass: the query's index
    InitHit *scratch;          // per warp: scratch_cap records
    uint32_t scratch_cap;
    InitHit *init_out;
    unsigned long long init_cap;
    WorkItem *work;
    unsigned long long work_cap;
    DevCounters *cnt;
    unsigned long long *cursor;  // the launch's work cursor, batched: one per query (zeroed before the pass)
};

struct GappedArgs {
    const uint8_t *res;
    const uint64_t *off;
    const uint8_t *q;
    int32_t qlen;
    // batched launches only: query of each work item and per-query data
    const uint32_t *work_query;
    const uint8_t *const *batch_q;
    const int32_t *batch_qlen;
    const int32_t *batch_cutoff;
    const int32_t *batch_smin;       // per query: lowest score the preliminary reap keeps
    const int32_t *batch_max_hsps;   // per query: HSPs kept per subject (0: all)
    const InitHit *init_in;
    const WorkItem *work;
    unsigned long long work_cap;
    unsigned long long init_cap;  // records in init_in (items beyond it are rejected)
    uint32_t n_subj, n_queries;   // valid subject and query indices of an item
    InitHit *sorted;     // per warp: cap records
    DevHsp *saved;       // per warp: cap records
    uint32_t cap;
    int32_t *dp;         // per warp: 2 * dp_stride ints, 8-byte aligned
    uint32_t dp_stride;  // >= max subject length + 2, even
    int32_t gap_open, gap_extend, xdrop, cutoff;
    int32_t smin, max_hsps;  // single query: as batch_smin / batch_max_hsps
    DevHsp *out;
    unsigned long long out_cap;
    const uint32_t *oid;     // sorted index -> OID
    GroupDesc *groups;       // one per published list (null: none written)
    uint32_t *qkept;         // per query: lists published (null: not counted)
    DevCounters *cnt;
    // the form by DP tasks (launch_gapped_split), per init-hit slot
    InitHit *init_sorted;    // each item's init hits in processing order
    DpTask *dtask;
    int4 *dres;              // per slot: left and right DP (best, row, column, cells; cells -1: not run)
    uint32_t *dorder;        // slots in DP order: items' best from the front, the others from the back
    uint32_t *dleft;         // at an item's first slot: its DPs still to end
    unsigned long long lane_slots;  // from this many slots on one lane per DP, else one warp
};

// Hit-list selection: queries that keep more subjects than their
// hitlist_size keep the hitlist_size best (score of the first HSP
// descending, ties by smaller OID); the others' lists are marked n = 0.
struct HitlistArgs {
    GroupDesc *groups;
    unsigned long long n_groups;
    const uint32_t *seg_off;         // per query: its segment of keys (n_queries + 1; empty if not selecting)
    uint32_t *seg_fill;              // per query: segment cursor, zeroed
    unsigned long long *keys;        // segment storage: ranking key and list index
    uint32_t *idx;
    const uint32_t *sel_queries;     // the selecting queries, one block each
    const int32_t *limit;            // per query: hitlist_size
};

// Shared-memory layout of the scan kernel for one query.
struct ScanLayout {
    uint32_t diag_entries, diag_magic, diag_bytes, stage_bytes, query_smem_bytes, warp_smem_bytes;
    Words words;
    int warps_per_block;
    size_t smem_bytes;
};

// Traceback stage: one preliminary HSP to trace from its gapped start point.
struct TbItem {
    uint32_t subject;  // index into the length-sorted database
    int32_t q_off, s_off;
    uint32_t query;    // batched runs: the query's position in its batch
};

struct TbOut {
    int32_t score, q_start, q_end, s_start, s_end;
    int32_t length, identities, positives, mismatches, gap_opens, gaps;
    int32_t status;  // 0 done, 1 direction buffer too small, 2 inconsistent path
    int32_t cells;   // DP cells computed (left and right)
};

// One side of a traced HSP: the DP's best cell (rows, columns from the start
// point) and the path's counts; last: the kind of its move next to the start
// point (0 a pair, 1 and 2 gaps, -1 none). status as in TbOut.
struct TbPart {
    int32_t score, a, b, pairs, identities, positives, gaps, gap_opens, last, status, cells;
};

struct TracebackArgs {
    const uint8_t *res;
    const uint64_t *off;
    const uint8_t *q;
    int32_t qlen;
    const uint8_t *const *batch_q;  // batched runs: per query (q, qlen unused)
    const int32_t *batch_qlen;
    const TbItem *items;
    uint32_t n_items;
    TbOut *out;
    int32_t gap_open, gap_extend, xdrop;
    int32_t *dp;                // per warp: H and E rows of dp_stride ints each
    uint32_t dp_stride;
    uint8_t *dirs;              // per warp: dir_cap direction bytes
    unsigned long long dir_cap;
    int32_t *rows;              // per warp: 3 ints per DP row
    uint32_t row_cap;
    TbPart *part;               // per item: left and right side
    unsigned int *done;         // per item: sides done (zeroed)
    unsigned long long *cursor;
};

// Launchers (scan.cu, kernels.cu, traceback.cu).
ScanLayout scan_layout(int32_t qlen, int32_t window, uint32_t n_hits, uint32_t stage_bytes, size_t smem_budget,
                       int max_warps, uint32_t band_entries = 0, bool least = false);
cudaError_t launch_scan(const ScanArgs &a, Words words, int n_blocks, int warps_per_block, size_t smem,
                        cudaStream_t st);
cudaError_t scan_occupancy(bool query_in_smem, Words words, bool bands, int warps_per_block, size_t smem, int *blocks_per_sm);
int scan_max_warps_by_registers(bool query_in_smem);
cudaError_t launch_gapped(const GappedArgs &a, int n_blocks, cudaStream_t st,
                          int warps_per_block = kGappedWarpsPerBlock);
cudaError_t launch_hitlist(const HitlistArgs &a, uint32_t n_select, int n_sm, cudaStream_t st);
constexpr int kTracebackWarpsPerBlock = 4;
constexpr int kTracebackBlocksPerSm = 5;      // with the band in registers
constexpr int kTracebackRowsBlocksPerSm = 8;  // with the rows in memory
constexpr int32_t kTbParts = 3, kTbWindow = 64 * kTbParts;  // columns that the registers hold
// Whether an X-drop's bands fit the registers: they reach about three times the
// columns of their first row's gap. Of 4,000 alignments of 300 residues at gap
// costs 11/1 none outgrows them at X-drop 68 (0.47 ms, 0.82 with the rows in
// memory), at 72 so many do that the other form is no slower, and from 95 on it is
// the faster (1.03 and 1.01, at 140 2.54 and 2.24); of 2,300 of 450 residues with
// subjects of up to 20,000 1.54 and 1.04 ms at 75. A band has one column more than
// its subject at most.
inline bool traceback_in_window(int32_t gap_open, int32_t gap_extend, int32_t xdrop, uint32_t longest) {
    const int64_t first_gap = (static_cast<int64_t>(xdrop) - gap_open - gap_extend) / gap_extend;
    return 3 * first_gap + 16 <= kTbWindow || longest + 1u <= static_cast<uint32_t>(kTbWindow);
}
cudaError_t launch_traceback(const TracebackArgs &a, bool window, int n_blocks, cudaStream_t st);
cudaError_t launch_scan_batch(const ScanArgs &a, Words words, int n_blocks, int warps_per_block, size_t smem,
                              cudaStream_t st);
cudaError_t scan_batch_occupancy(bool query_in_smem, Words words, int warps_per_block, size_t smem,
                                 int *blocks_per_sm);
int scan_batch_max_warps_by_registers(bool query_in_smem);
cudaError_t gapped_occupancy(int *blocks_per_sm);
// The gapped stage as DP tasks; n_blocks as for launch_gapped, the lane DP
// kernel fills n_sm SMs. Results equal launch_gapped's.
cudaError_t launch_gapped_split(const GappedArgs &a, int n_blocks, int n_sm, cudaStream_t st);

// The lookups of n queries: `many` (a device array), or `one` when it is null.
constexpr uint32_t kLookupKernels = 3;  // of a launch
cudaError_t launch_lookup(const LookupQuery &one, const LookupQuery *many, uint32_t n, int32_t threshold,
                          cudaStream_t st);

// Host helpers (host.cpp).
extern const int32_t kBlosum62[kAlphabet][kAlphabet];
// Entries of a query's hit lists (its word lookup's size), without building it.
uint32_t lookup_hits(const uint8_t *query, int32_t qlen, int32_t threshold);
int default_params(int32_t qlen, uint64_t db_len, uint32_t db_n, double evalue,
                   blaze_params *out);

}  // namespace blaze

#define BLAZE_CUDA_TRY(expr)                                  \
    do {                                                      \
        cudaError_t err__ = (expr);                           \
        if (err__ != cudaSuccess) {                           \
            last_cuda_error(err__);                           \
            return err__ == cudaErrorMemoryAllocation         \
                       ? BLAZE_ERR_OUT_OF_MEMORY              \
                       : BLAZE_ERR_CUDA;                      \
        }                                                     \
    } while (0)

void last_cuda_error(cudaError_t e);
