// api.cu -- C ABI of libblaze103: resident database, query tables, and the
// search driver that runs the two device stages and finishes each subject's
// HSP list (E-values, preliminary E-value reap, OID order) on the host.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <numeric>
#include <type_traits>
#include <utility>
#include <vector>

#include "handles.h"
#include "internal.h"

namespace {
thread_local cudaError_t g_last_cuda = cudaSuccess;
}  // namespace

void last_cuda_error(cudaError_t e) { g_last_cuda = e; }
int last_cuda_error_code() { return static_cast<int>(g_last_cuda); }
void set_last_cuda_error_code(int code) { g_last_cuda = static_cast<cudaError_t>(code); }

extern "C" const char *blaze_last_cuda_error(void) { return cudaGetErrorString(g_last_cuda); }

extern "C" int blaze_device_count(int *count) {
    if (!count) return BLAZE_ERR_INVALID_ARG;
    *count = 0;
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return BLAZE_OK;
    }
    *count = n;
    return BLAZE_OK;
}

extern "C" int blaze_db_create(int device, const uint8_t *residues, const uint64_t *offsets,
                               uint32_t n_subjects, blaze_db **out) try {
    if (!out || !offsets || (n_subjects > 0 && !residues)) return BLAZE_ERR_INVALID_ARG;
    *out = nullptr;
    int ndev = 0;
    blaze_device_count(&ndev);
    if (ndev == 0) return BLAZE_ERR_NO_DEVICE;
    if (device < 0 || device >= ndev) return BLAZE_ERR_INVALID_ARG;
    for (uint32_t i = 0; i < n_subjects; ++i) {
        if (offsets[i + 1] < offsets[i]) return BLAZE_ERR_INVALID_ARG;
        if (offsets[i + 1] - offsets[i] > kMaxSubjectLength) return BLAZE_ERR_LIMIT;
    }
    const uint64_t base = offsets[0], total = offsets[n_subjects] - base;
    if (!valid_residues(residues + base, total)) return BLAZE_ERR_INVALID_ARG;
    BLAZE_CUDA_TRY(cudaSetDevice(device));
    auto *db = new blaze_db();
    db->device = device;
    db->n = n_subjects;
    db->total = total;
    // length-sorted order (stable: equal lengths keep OID order)
    std::vector<uint32_t> order(n_subjects);
    std::iota(order.begin(), order.end(), 0u);
    auto len = [&](uint32_t i) { return offsets[i + 1] - offsets[i]; };
    bool sorted = true;
    for (uint32_t i = 1; i < n_subjects && sorted; ++i) sorted = len(i - 1) <= len(i);
    if (!sorted) std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return len(a) < len(b); });
    db->oid_of = order;
    db->sorted_of.resize(n_subjects);
    for (uint32_t k = 0; k < n_subjects; ++k) db->sorted_of[order[k]] = k;
    std::vector<uint64_t> off(n_subjects + 1);
    off[0] = 0;
    for (uint32_t k = 0; k < n_subjects; ++k) {
        off[k + 1] = off[k] + len(order[k]);
        db->max_len = std::max<uint32_t>(db->max_len, static_cast<uint32_t>(len(order[k])));
    }
    int rc = BLAZE_OK;
    do {
        cudaError_t e = cudaMalloc(&db->d_res, total + 64);
        if (e == cudaSuccess) e = cudaMalloc(&db->d_off, sizeof(uint64_t) * (n_subjects + 1));
        if (e == cudaSuccess) e = cudaMalloc(&db->d_oid, sizeof(uint32_t) * std::max<uint32_t>(n_subjects, 1));
        if (e != cudaSuccess) {
            last_cuda_error(e);
            rc = e == cudaErrorMemoryAllocation ? BLAZE_ERR_OUT_OF_MEMORY : BLAZE_ERR_CUDA;
            break;
        }
        if (sorted) {
            e = cudaMemcpy(db->d_res, residues + base, total, cudaMemcpyHostToDevice);
        } else {
            std::vector<uint8_t> tmp(total);
            for (uint32_t k = 0; k < n_subjects; ++k)
                std::memcpy(tmp.data() + off[k], residues + offsets[order[k]], len(order[k]));
            e = cudaMemcpy(db->d_res, tmp.data(), total, cudaMemcpyHostToDevice);
        }
        if (e == cudaSuccess) e = cudaMemset(db->d_res + total, 0, 64);
        if (e == cudaSuccess) e = cudaMemcpy(db->d_off, off.data(), sizeof(uint64_t) * (n_subjects + 1), cudaMemcpyHostToDevice);
        if (e == cudaSuccess && n_subjects)
            e = cudaMemcpy(db->d_oid, order.data(), sizeof(uint32_t) * n_subjects, cudaMemcpyHostToDevice);
        if (e != cudaSuccess) {
            last_cuda_error(e);
            rc = BLAZE_ERR_CUDA;
        }
    } while (false);
    if (rc == BLAZE_OK) {
        db->h_off.swap(off);
        rc = db_make_groups(db);
    }
    if (rc != BLAZE_OK) {
        blaze_db_free(db);
        return rc;
    }
    *out = db;
    return BLAZE_OK;
} BLAZE_ABI_CATCH

int db_make_groups(blaze_db *db) {
    const std::vector<uint64_t> &off = db->h_off;
    // A group holds twice a warp's share of the residues that are left (32 warps
    // an SM), at most what a warp stages: what a group costs beyond its residues
    // -- fetching it, its last partial batches and extensions -- is spread over
    // more of them, and the last groups are small, so that the warps end about
    // together. 300 query residues against 14 / 35 / 140 M: 0.183 / 0.329 / 1.013
    // ms with 1/16 of a warp's share of all residues, 0.140 / 0.261 / 0.983 so.
    constexpr uint64_t kLeast = 512;
    int n_sm = 0;
    BLAZE_CUDA_TRY(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, db->device));
    const uint64_t warps = static_cast<uint64_t>(n_sm) * kScanMaxWarpsPerBlock;
    const uint64_t least = std::min<uint64_t>(kLeast, db->total / warps);
    auto cut = [&](uint64_t at_least, std::vector<uint32_t> &b) {  // returns the bytes of the largest group of several
        uint32_t largest = 0;
        b.assign(1, db->n);
        for (uint32_t hi = db->n; hi > 0;) {
            const uint64_t most = std::min<uint64_t>(std::max<uint64_t>(2 * off[hi] / warps, at_least), kGroupMaxBytes);
            uint32_t lo = hi - 1;
            while (lo > 0 && hi - lo < kGroupMaxSubjects &&
                   off[hi] - off[lo - 1] + kGroupSubjectBytes * (hi - lo + 1) <= most)
                --lo;
            if (hi - lo > 1)
                largest = std::max(largest, static_cast<uint32_t>(off[hi] - off[lo] + kGroupSubjectBytes * (hi - lo)));
            b.push_back(lo);
            hi = lo;
        }
        return largest;
    };
    std::vector<uint32_t> &b = db->h_groups, batch;
    db->group_bytes = cut(least, b);
    if (least < kLeast) cut(kLeast, batch);
    // A subject alone in its group is cut in pieces of a warp's share of the
    // residues (with what precedes it in its first 16 bytes), other groups are
    // one piece. (4,000 residues against 500 subjects: 0.21 ms with pieces of
    // 128, 0.35 of 512, 0.52 of 2,240.)
    const uint64_t piece = std::min<uint64_t>(std::max<uint64_t>(db->total / warps, kPieceLeast), kPieceMost);
    std::vector<uint32_t> pieces(1, 0u);
    for (size_t g = 0; g + 1 < b.size(); ++g) {
        const uint64_t len = b[g] - b[g + 1] == 1 ? off[b[g]] - off[b[g + 1]] : 0;
        pieces.push_back(pieces.back() + std::max<uint32_t>(1u, static_cast<uint32_t>((len + 15 + piece - 1) / piece)));
    }
    db->n_pieces = pieces.back();
    std::vector<uint32_t> both(b);
    both.insert(both.end(), batch.begin(), batch.end());
    BLAZE_CUDA_TRY(cudaMalloc(&db->d_groups, sizeof(uint32_t) * both.size()));
    BLAZE_CUDA_TRY(cudaMemcpy(db->d_groups, both.data(), sizeof(uint32_t) * both.size(), cudaMemcpyHostToDevice));
    if (!batch.empty()) {
        db->d_batch_groups = db->d_groups + b.size();
        db->n_batch_groups = static_cast<uint32_t>(batch.size() - 1);
    }
    BLAZE_CUDA_TRY(cudaMalloc(&db->d_pieces, sizeof(uint32_t) * pieces.size()));
    BLAZE_CUDA_TRY(cudaMemcpy(db->d_pieces, pieces.data(), sizeof(uint32_t) * pieces.size(), cudaMemcpyHostToDevice));
    return BLAZE_OK;
}

extern "C" int blaze_db_free(blaze_db *db) {
    if (!db) return BLAZE_OK;
    cudaSetDevice(db->device);
    if (db->d_res) cudaFree(db->d_res);
    if (db->d_off) cudaFree(db->d_off);
    if (db->d_oid) cudaFree(db->d_oid);
    if (db->d_groups) cudaFree(db->d_groups);
    if (db->d_pieces) cudaFree(db->d_pieces);
    delete db;
    return BLAZE_OK;
}

extern "C" int blaze_db_info(const blaze_db *db, uint64_t *total, uint32_t *n, uint32_t *max_len) {
    if (!db) return BLAZE_ERR_INVALID_ARG;
    if (total) *total = db->total;
    if (n) *n = db->n;
    if (max_len) *max_len = db->max_len;
    return BLAZE_OK;
}

// Where a query's residues (with 64 zero bytes behind them) and its lookup's
// tables lie in one device buffer.
struct QueryTables {
    size_t res_bytes, cs, pack, pres, off, bytes;
    QueryTables(int32_t length, uint32_t n_off) {
        auto up = [](size_t x) { return (x + 15) & ~size_t{15}; };
        res_bytes = up(static_cast<size_t>(length) + 64);
        cs = res_bytes;
        pack = up(cs + sizeof(uint32_t) * (kWords + 1));
        pres = up(pack + sizeof(uint32_t) * kWords);
        off = up(pres + sizeof(uint32_t) * kPresenceWords);
        bytes = off + sizeof(uint16_t) * std::max<uint32_t>(n_off, 1);
    }
    void point(blaze_query &q, unsigned char *p) const {
        q.d_q = p;
        q.d_cell_start = reinterpret_cast<uint32_t *>(p + cs);
        q.d_cell_pack = reinterpret_cast<uint32_t *>(p + pack);
        q.d_presence = reinterpret_cast<uint32_t *>(p + pres);
        q.d_cell_off = reinterpret_cast<uint16_t *>(p + off);
    }
};

// The query's lookup, built on the device from its residues.
static cudaError_t build_lookup(const blaze_query &q, cudaStream_t st) {
    return launch_lookup(LookupQuery{q.d_q, q.qlen, q.d_cell_start, q.d_cell_pack, q.d_presence, q.d_cell_off}, nullptr,
                         1, q.threshold, st);
}

extern "C" int blaze_query_create(const blaze_db *db, const uint8_t *query, int32_t length,
                                  int32_t word_threshold, blaze_query **out) try {
    if (!db || !query || !out || length <= 0) return BLAZE_ERR_INVALID_ARG;
    *out = nullptr;
    if (length > kMaxQueryLength) return BLAZE_ERR_LIMIT;
    if (!valid_residues(query, static_cast<uint64_t>(length))) return BLAZE_ERR_INVALID_ARG;
    BLAZE_CUDA_TRY(cudaSetDevice(db->device));
    const uint32_t n_off = lookup_hits(query, length, word_threshold);
    const QueryTables t(length, n_off);
    std::vector<uint8_t> res(t.res_bytes, 0);
    std::memcpy(res.data(), query, length);
    auto *q = new blaze_query();
    q->device = db->device;
    q->qlen = length;
    q->threshold = word_threshold;
    q->n_off = n_off;
    q->upload_bytes = t.res_bytes;
    cudaError_t e = cudaMalloc(&q->d_tables, t.bytes);
    if (e == cudaSuccess) {
        t.point(*q, q->d_tables);
        e = cudaMemcpy(q->d_q, res.data(), t.res_bytes, cudaMemcpyHostToDevice);
    }
    if (e == cudaSuccess) e = build_lookup(*q, nullptr);
    if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);  // searches run on streams of their own
    if (e != cudaSuccess) {
        last_cuda_error(e);
        blaze_query_free(q);
        return e == cudaErrorMemoryAllocation ? BLAZE_ERR_OUT_OF_MEMORY : BLAZE_ERR_CUDA;
    }
    *out = q;
    return BLAZE_OK;
} BLAZE_ABI_CATCH

extern "C" int blaze_query_free(blaze_query *q) {
    if (!q) return BLAZE_OK;
    cudaSetDevice(q->device);
    if (q->d_tables) cudaFree(q->d_tables);
    delete q;
    return BLAZE_OK;
}

extern "C" int blaze_search_create(blaze_db *db, blaze_search **out) try {
    if (!db || !out) return BLAZE_ERR_INVALID_ARG;
    *out = nullptr;
    BLAZE_CUDA_TRY(cudaSetDevice(db->device));
    auto *s = new blaze_search();
    s->db = db;
    cudaError_t e = cudaDeviceGetAttribute(&s->n_sm, cudaDevAttrMultiProcessorCount, db->device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMalloc(&s->d_cnt, sizeof(DevCounters));
    if (e == cudaSuccess) e = cudaMallocHost(&s->h_cnt, sizeof(DevCounters));
    for (int i = 0; i < 4 && e == cudaSuccess; ++i) e = cudaEventCreate(&s->ev[i]);
    int per_sm = 0;
    if (e == cudaSuccess) e = gapped_occupancy(&per_sm);
    if (e != cudaSuccess) {
        last_cuda_error(e);
        blaze_search_free(s);
        return BLAZE_ERR_CUDA;
    }
    s->gapped_blocks = s->n_sm * std::min(std::max(per_sm, 1), 8);
    for (int smem = 0; smem < 2; ++smem) s->reg_warps[smem] = scan_max_warps_by_registers(smem != 0);
    s->batch_reg_warps = std::min(scan_batch_max_warps_by_registers(true), scan_batch_max_warps_by_registers(false));
    s->init_cap = std::max<unsigned long long>(1ull << 20, db->n / 8);
    s->work_cap = std::max<unsigned long long>(1ull << 20, db->n / 4);
    s->out_cap = std::max<unsigned long long>(1ull << 20, db->n / 16);
    // Starting capacities can be lowered (e.g. to exercise the grow-and-repeat
    // path); they grow on demand either way.
    if (const char *v = std::getenv("BLAZE_INITIAL_SCRATCH_CAP")) s->scratch_cap = std::max(1, std::atoi(v));
    if (const char *v = std::getenv("BLAZE_INITIAL_INIT_CAP")) s->init_cap = std::max(1, std::atoi(v));
    if (const char *v = std::getenv("BLAZE_INITIAL_OUT_CAP")) s->out_cap = std::max(1, std::atoi(v));
    if (const char *v = std::getenv("BLAZE_INITIAL_WORK_CAP")) s->work_cap = std::max(1, std::atoi(v));
    // likewise the pass size from which the gapped stage runs one lane per DP
    if (const char *v = std::getenv("BLAZE_LANE_DP_SLOTS")) s->lane_dp_slots = std::strtoull(v, nullptr, 10);
    if (const char *v = std::getenv("BLAZE_INITIAL_TRACEBACK_CAP")) s->tb_dir_cap = std::max(64, std::atoi(v));
    *out = s;
    return BLAZE_OK;
} BLAZE_ABI_CATCH

extern "C" int blaze_search_free(blaze_search *s) {
    if (!s) return BLAZE_OK;
    cudaSetDevice(s->db->device);
    if (s->stream) cudaStreamSynchronize(s->stream);
    if (s->graph_exec) cudaGraphExecDestroy(s->graph_exec);
    s->scratch.release();
    s->init_out.release();
    s->band_state.release();
    s->gapped_ws.release();
    s->work.release();
    s->saved.release();
    s->out.release();
    s->dp.release();
    s->bq.release();
    s->bqptr.release();
    s->bqlen.release();
    s->bcut.release();
    s->work_query.release();
    s->cursors.release();
    s->bsmin.release();
    s->bmaxh.release();
    s->sel_limit.release();
    s->groups.release();
    s->qkept.release();
    s->seg_off.release();
    s->seg_fill.release();
    s->seg_idx.release();
    s->sel_q.release();
    s->seg_keys.release();
    s->qt.release();
    if (s->h_stage) cudaFreeHost(s->h_stage);
    s->tb_items.release();
    s->tb_out.release();
    s->tb_part.release();
    s->tb_done.release();
    s->tb_dirs.release();
    s->tb_rows.release();
    s->tb_dp.release();
    s->tb_cursor.release();
    if (s->h_groups) cudaFreeHost(s->h_groups);
    if (s->d_cnt) cudaFree(s->d_cnt);
    if (s->h_cnt) cudaFreeHost(s->h_cnt);
    if (s->h_out) cudaFreeHost(s->h_out);
    for (cudaEvent_t ev : s->ev)
        if (ev) cudaEventDestroy(ev);
    if (s->stream) cudaStreamDestroy(s->stream);
    delete s;
    return BLAZE_OK;
}

int check_params(const blaze_params *p) {
    if (!p) return BLAZE_ERR_INVALID_ARG;
    if (p->window <= 0 || p->window > (1 << 20) || p->ungapped_xdrop <= 0 || p->gap_open < 0 ||
        p->gap_extend <= 0 || p->gapped_xdrop <= 0 || p->gapped_cutoff <= 0 || p->ungapped_cutoff <= 0)
        return BLAZE_ERR_INVALID_ARG;
    // E-value statistics: E must fall with the score (the reap is a score threshold)
    if (!(p->lambda > 0.0) || !std::isfinite(p->lambda) || !(p->K > 0.0) || !std::isfinite(p->K) ||
        !(p->eff_searchsp >= 0.0) || !std::isfinite(p->eff_searchsp) || std::isnan(p->prelim_evalue))
        return BLAZE_ERR_INVALID_ARG;
    return BLAZE_OK;
}

// The preliminary reap drops an HSP when eff_searchsp * K * exp(-lambda * S)
// exceeds prelim_evalue. E falls with S, so on the scores a gapped HSP can
// have (1 and up) it keeps exactly those from the smallest passing S, found
// by bisection over the same expression.
static int32_t reap_min_score(const blaze_params &p) {
    auto keeps = [&p](int64_t S) {
        return !(p.eff_searchsp * p.K * std::exp(-p.lambda * static_cast<double>(S)) > p.prelim_evalue);
    };
    int64_t lo = 1, hi = INT32_MAX;  // keeps(hi) or no score passes
    if (keeps(lo)) return 1;
    if (!keeps(hi)) return INT32_MAX;
    while (hi - lo > 1) {  // !keeps(lo), keeps(hi)
        const int64_t mid = lo + (hi - lo) / 2;
        (keeps(mid) ? hi : lo) = mid;
    }
    return static_cast<int32_t>(hi);
}

// What one run searches: one query, or a batch with one parameter set per
// query.
struct RunSpec {
    const blaze_query *q = nullptr;
    const blaze_batch *b = nullptr;
    const blaze_params *p = nullptr;
    std::vector<int32_t> smin;  // per query: the reap's lowest kept score
    std::vector<uint32_t> border;  // batched: query indices in launch (length) order
};

// One pass's launch sequence: counter reset, scan kernel, gapped kernel and
// the counter read-back, with the timing events between them.
struct ScanLaunch {
    ScanArgs sa;
    int blocks, warps_per_block;
    size_t smem_bytes;
    bool queue;  // the batched kernel, else the single-query one
    Words words;
};

struct PassLaunch {
    std::vector<ScanLaunch> scans;
    uint32_t n_cursors;
    const GappedArgs *ga;
    bool batched;
};

// Batched passes of at least this many queries may hold so many init hits
// (kLaneDpSlots) that one lane per DP is the faster; only the device knows.
constexpr uint32_t kLaneDpMinQueries = 16;

static cudaError_t enqueue_pass(blaze_search *s, const PassLaunch &pl, unsigned event_flags) {
    cudaError_t e = cudaMemsetAsync(s->d_cnt, 0, sizeof(DevCounters), s->stream);
    if (e == cudaSuccess)
        e = cudaMemsetAsync(s->cursors.p, 0, sizeof(unsigned long long) * pl.n_cursors, s->stream);
    if (e == cudaSuccess) e = cudaEventRecordWithFlags(s->ev[1], s->stream, event_flags);
    for (const ScanLaunch &l : pl.scans) {
        if (e == cudaSuccess && l.sa.pieces)
            e = cudaMemsetAsync(s->band_state.p, 0, sizeof(BandState) * l.sa.n_groups, s->stream);
        if (e != cudaSuccess) break;
        e = l.queue ? launch_scan_batch(l.sa, l.words, l.blocks, l.warps_per_block, l.smem_bytes, s->stream)
                       : launch_scan(l.sa, l.words, l.blocks, l.warps_per_block, l.smem_bytes, s->stream);
    }
    if (e == cudaSuccess) e = cudaEventRecordWithFlags(s->ev[2], s->stream, event_flags);
    if (e == cudaSuccess) e = launch_gapped_split(*pl.ga, s->gapped_blocks, s->n_sm, s->stream);
    if (e == cudaSuccess) e = cudaEventRecordWithFlags(s->ev[3], s->stream, event_flags);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(s->h_cnt, s->d_cnt, sizeof(DevCounters), cudaMemcpyDeviceToHost, s->stream);
    return e;
}

static int launch_pass_direct(blaze_search *s, const PassLaunch &pl) {
    BLAZE_CUDA_TRY(enqueue_pass(s, pl, cudaEventRecordDefault));
    return BLAZE_OK;
}

// Replays the pass from a CUDA graph. The graph's kernel arguments are the
// ScanArgs/GappedArgs values themselves (every buffer they point to keeps its
// address while it is not regrown), so a pass whose arguments and launch
// shapes equal those of the captured one replays it; otherwise the sequence
// is captured again and the executable graph updated in place (or rebuilt
// when the update is refused). Capture is thread-local, so other host
// threads may allocate meanwhile.
static int launch_pass_graph(blaze_search *s, const PassLaunch &pl) {
    std::vector<unsigned char> key;
    auto put = [&key](const void *p, size_t n) {
        const auto *c = static_cast<const unsigned char *>(p);
        key.insert(key.end(), c, c + n);
    };
    const int64_t head[2] = {pl.batched, s->gapped_blocks};
    put(head, sizeof(head));
    for (const ScanLaunch &l : pl.scans) {
        put(&l.sa, sizeof(ScanArgs));
        const int64_t shape[4] = {l.blocks, l.warps_per_block, static_cast<int64_t>(l.smem_bytes),
                                  static_cast<int64_t>(l.words)};
        put(shape, sizeof(shape));
    }
    put(pl.ga, sizeof(GappedArgs));
    if (s->graph_exec && key == s->graph_key) {
        BLAZE_CUDA_TRY(cudaGraphLaunch(s->graph_exec, s->stream));
        s->stats.graph_replays++;
        return BLAZE_OK;
    }
    BLAZE_CUDA_TRY(cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
    const cudaError_t e = enqueue_pass(s, pl, cudaEventRecordExternal);
    cudaGraph_t g = nullptr;
    const cudaError_t ec = cudaStreamEndCapture(s->stream, &g);
    if (e != cudaSuccess || ec != cudaSuccess) {
        if (g) cudaGraphDestroy(g);
        s->graph_key.clear();
        BLAZE_CUDA_TRY(e != cudaSuccess ? e : ec);
    }
    bool updated = false;
    if (s->graph_exec) {
        cudaGraphExecUpdateResultInfo info;
        if (cudaGraphExecUpdate(s->graph_exec, g, &info) == cudaSuccess) {
            updated = true;
        } else {
            cudaGetLastError();  // a refused update is not an error: rebuild
            cudaGraphExecDestroy(s->graph_exec);
            s->graph_exec = nullptr;
        }
    }
    cudaError_t ei = cudaSuccess;
    if (!updated) ei = cudaGraphInstantiate(&s->graph_exec, g, 0);
    cudaGraphDestroy(g);
    if (ei != cudaSuccess) {
        s->graph_exec = nullptr;
        s->graph_key.clear();
        BLAZE_CUDA_TRY(ei);
    }
    s->graph_key.swap(key);
    s->stats.graph_builds++;
    BLAZE_CUDA_TRY(cudaGraphLaunch(s->graph_exec, s->stream));
    return BLAZE_OK;
}

// One scan launch of a pass: the single-query kernel (a single-query run, or
// one query of a batch), or the batched kernel over a group of a batch's
// queries (queries [first, first + n) of the length-ordered descriptors),
// each with its own shared-memory layout.
struct ScanPlan {
    ScanLayout lay;
    int blocks = 0;
    uint32_t first = 0, n = 1;
    bool queue = false;  // the batched kernel over the plan's queries; else one query's launch
    bool batch_groups = false;  // with blaze_db::d_batch_groups
    bool bands = false;  // one query's launch in bands
    uint32_t extra_bands = 0;
};

// One pass of both stages; fills s->h_cnt.
static int run_pass(blaze_search *s, const RunSpec &r, const std::vector<ScanPlan> &plans) {
    blaze_db *db = s->db;
    const blaze_params *p = r.p;
    const bool batched = r.b != nullptr;
    size_t scan_warps = 0;
    for (const ScanPlan &pl : plans)
        scan_warps = std::max(scan_warps, static_cast<size_t>(pl.blocks) * pl.lay.warps_per_block);
    const size_t gapped_warps = static_cast<size_t>(s->gapped_blocks) * kGappedWarpsPerBlock;
    const size_t work_cap = batched ? s->work_cap : std::max<uint32_t>(db->n, 1);
    int rc;
    if ((rc = s->scratch.ensure(scan_warps * s->scratch_cap)) != BLAZE_OK) return rc;
    if ((rc = s->saved.ensure(gapped_warps * s->scratch_cap)) != BLAZE_OK) return rc;
    if ((rc = s->init_out.ensure(s->init_cap)) != BLAZE_OK) return rc;
    if ((rc = s->work.ensure(work_cap)) != BLAZE_OK) return rc;
    if ((rc = s->out.ensure(s->out_cap)) != BLAZE_OK) return rc;
    const uint32_t nq = batched ? r.b->n : 1u;
    // the gapped stage's arrays, per init-hit slot: ordered init hit, DP task,
    // two DP results, DP order, DPs left
    constexpr size_t slot_bytes = sizeof(InitHit) + sizeof(DpTask) + 2 * sizeof(int4) + 2 * sizeof(uint32_t);
    if ((rc = s->gapped_ws.ensure(s->init_cap * slot_bytes)) != BLAZE_OK) return rc;
    const size_t n_groups = db->h_groups.size() - 1;
    for (const ScanPlan &plan : plans)
        if (plan.bands && (rc = s->band_state.ensure(n_groups)) != BLAZE_OK) return rc;
    if ((rc = s->groups.ensure(s->out_cap)) != BLAZE_OK) return rc;  // a published list holds >= 1 HSP
    if ((rc = s->qkept.ensure(nq)) != BLAZE_OK) return rc;
    if (batched && (rc = s->work_query.ensure(work_cap)) != BLAZE_OK) return rc;
    // DP rows of the longest subject plus 2, even so that each warp's H and E
    // rows start 8-byte aligned (the DP reads and writes column pairs)
    const size_t dp_stride = (static_cast<size_t>(std::max<uint32_t>(db->max_len, 1)) + 3) & ~size_t{1};
    if ((rc = s->dp.ensure(gapped_warps * 2 * dp_stride)) != BLAZE_OK) return rc;
    if ((rc = s->cursors.ensure(nq)) != BLAZE_OK) return rc;

    PassLaunch pl;
    pl.batched = batched;
    pl.n_cursors = nq;
    for (const ScanPlan &plan : plans) {
        const ScanLayout &lay = plan.lay;
        ScanLaunch l;
        ScanArgs &sa = l.sa;
        std::memset(&sa, 0, sizeof(sa));  // whole bytes: the graph key compares them
        l.words = lay.words;
        l.blocks = plan.blocks;
        l.warps_per_block = lay.warps_per_block;
        l.smem_bytes = lay.smem_bytes;
        sa.res = db->d_res;
        sa.off = db->d_off;
        sa.groups = plan.batch_groups ? db->d_batch_groups : db->d_groups;
        sa.n_groups = plan.batch_groups ? db->n_batch_groups : static_cast<uint32_t>(n_groups);
        sa.n_items = sa.n_groups;
        if (plan.bands) {
            sa.pieces = db->d_pieces;
            sa.extra_bands = plan.extra_bands;
            sa.n_items = db->n_pieces + sa.n_groups * plan.extra_bands;
            sa.band_state = s->band_state.p;
            // a hit takes two records at most; the gapped stage's arrays lie idle
            // meanwhile
            static_assert(slot_bytes >= 2 * sizeof(InitHit));
            sa.fragments = reinterpret_cast<InitHit *>(s->gapped_ws.p);
            sa.fragment_cap = std::min<unsigned long long>(2 * s->init_cap, UINT32_MAX - 1);
        }
        sa.window = p->window;
        sa.xdrop = p->ungapped_xdrop;
        sa.diag_entries = lay.diag_entries;
        sa.diag_magic = lay.diag_magic;
        sa.diag_bytes = lay.diag_bytes;
        sa.stage_bytes = lay.stage_bytes;
        sa.query_smem_bytes = lay.query_smem_bytes;
        sa.warp_smem_bytes = lay.warp_smem_bytes;
        sa.smem_bytes = static_cast<uint32_t>(lay.smem_bytes);
        sa.scratch = s->scratch.p;
        sa.scratch_cap = s->scratch_cap;
        sa.init_out = s->init_out.p;
        sa.init_cap = s->init_cap;
        sa.work = s->work.p;
        sa.work_cap = work_cap;
        sa.cnt = s->d_cnt;
        sa.cursor = s->cursors.p + plan.first;
        l.queue = plan.queue;
        if (batched && !plan.queue) {
            // one query of the batch with the single-query kernel; its work
            // items carry the query's batch index
            const uint32_t i = r.border[plan.first];
            const blaze_batch *b = r.b;
            sa.q = b->d_res + b->res_off[i];
            sa.qlen = b->qlen[i];
            sa.cell_start = b->d_cell_start + static_cast<size_t>(i) * (kWords + 1);
            sa.cell_pack = b->d_cell_pack + static_cast<size_t>(i) * kWords;
            sa.presence = b->d_presence + static_cast<size_t>(i) * kPresenceWords;
            sa.cell_off = b->d_cell_off + b->off_off[i];
            sa.cutoff = r.p[i].ungapped_cutoff;
            sa.n_queries = 1;
            sa.query_index = i;
            sa.work_query = s->work_query.p;
        } else if (batched) {
            sa.queries = s->bq.p + plan.first;
            sa.n_queries = plan.n;
            sa.work_query = s->work_query.p;
        } else {
            const blaze_query *q = r.q;
            sa.q = q->d_q;
            sa.qlen = q->qlen;
            sa.cell_start = q->d_cell_start;
            sa.cell_pack = q->d_cell_pack;
            sa.presence = q->d_presence;
            sa.cell_off = q->d_cell_off;
            sa.cutoff = p->ungapped_cutoff;
            sa.n_queries = 1;
        }
        pl.scans.push_back(l);
    }

    GappedArgs ga;
    std::memset(&ga, 0, sizeof(ga));
    ga.res = db->d_res;
    ga.off = db->d_off;
    ga.init_in = s->init_out.p;
    ga.work = s->work.p;
    ga.work_cap = work_cap;
    ga.init_cap = s->init_cap;
    ga.n_subj = db->n;
    ga.n_queries = nq;
    ga.saved = s->saved.p;
    ga.cap = s->scratch_cap;
    ga.dp = s->dp.p;
    ga.dp_stride = static_cast<uint32_t>(dp_stride);
    ga.gap_open = p->gap_open;
    ga.gap_extend = p->gap_extend;
    ga.xdrop = p->gapped_xdrop;
    ga.out = s->out.p;
    ga.out_cap = s->out_cap;
    ga.oid = db->d_oid;
    ga.groups = s->groups.p;
    ga.qkept = s->qkept.p;
    ga.cnt = s->d_cnt;
    unsigned char *ws = s->gapped_ws.p;
    auto take = [&](auto *&p, size_t n) {
        p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(ws);
        ws += n * sizeof(*p);
    };
    take(ga.dres, 2 * s->init_cap);
    take(ga.dtask, s->init_cap);
    take(ga.init_sorted, s->init_cap);
    take(ga.dorder, s->init_cap);
    take(ga.dleft, s->init_cap);
    ga.lane_slots = batched && nq >= kLaneDpMinQueries ? s->lane_dp_slots : ~0ull;
    if (batched) {
        ga.work_query = s->work_query.p;
        ga.batch_q = s->bqptr.p;
        ga.batch_qlen = s->bqlen.p;
        ga.batch_cutoff = s->bcut.p;
        ga.batch_smin = s->bsmin.p;
        ga.batch_max_hsps = s->bmaxh.p;
    } else {
        ga.q = r.q->d_q;
        ga.qlen = r.q->qlen;
        ga.cutoff = p->gapped_cutoff;
        ga.smin = r.smin[0];
        ga.max_hsps = p->max_hsps;
    }
    pl.ga = &ga;
    BLAZE_CUDA_TRY(cudaMemsetAsync(s->qkept.p, 0, sizeof(uint32_t) * nq, s->stream));
    const bool graph = s->launch_mode == 2 || (s->launch_mode == 0 && batched);
    if ((rc = graph ? launch_pass_graph(s, pl) : launch_pass_direct(s, pl)) != BLAZE_OK) return rc;
    s->stats.kernel_launches += static_cast<uint32_t>(pl.scans.size()) + (ga.lane_slots == ~0ull ? 2u : 4u);
    s->stats.d2h_bytes += sizeof(DevCounters);
    BLAZE_CUDA_TRY(cudaStreamSynchronize(s->stream));
    return BLAZE_OK;
}

template <typename T>
static int ensure_pinned(T *&p, size_t &n, size_t want) {
    if (want <= n) return BLAZE_OK;
    if (p) cudaFreeHost(p);
    p = nullptr;
    n = 0;
    BLAZE_CUDA_TRY(cudaMallocHost(&p, sizeof(T) * want));
    n = want;
    return BLAZE_OK;
}

// The published lists that hold HSPs, by (query, OID), in s->order[0]: keys of
// as many bits as queries and subjects need, sorted by radix passes of 11 bits,
// few lists by comparisons. (A comparison sort of the descriptors took 0.6 of
// the 0.9 ms that the host spent on 12,312 HSPs.)
static void order_lists(blaze_search *s, size_t n_groups, uint32_t nq) {
    constexpr size_t kRadixFrom = 256;
    constexpr unsigned kDigit = 11;
    auto bits = [](uint32_t n) {  // of the numbers below n
        unsigned b = 0;
        while (b < 32 && (n - 1) >> b) ++b;
        return b;
    };
    const unsigned oid_bits = bits(std::max<uint32_t>(s->db->n, 1)), key_bits = oid_bits + bits(nq);
    std::vector<ListKey> &a = s->order[0], &b = s->order[1];
    a.clear();
    for (size_t i = 0; i < n_groups; ++i) {
        const GroupDesc &g = s->h_groups[i];
        if (g.n > 0) a.push_back(ListKey{(static_cast<uint64_t>(g.query) << oid_bits) | g.oid, static_cast<uint32_t>(i)});
    }
    if (a.size() < kRadixFrom) {
        std::sort(a.begin(), a.end(), [](const ListKey &x, const ListKey &y) { return x.key < y.key; });
        return;
    }
    b.resize(a.size());
    for (unsigned shift = 0; shift < key_bits; shift += kDigit) {
        uint32_t at[1u << kDigit] = {};
        auto digit = [shift](const ListKey &x) { return (x.key >> shift) & ((1u << kDigit) - 1); };
        for (const ListKey &x : a) ++at[digit(x)];
        uint32_t sum = 0;
        for (uint32_t &n : at) sum += std::exchange(n, sum);
        for (const ListKey &x : a) b[at[digit(x)]++] = x;
        a.swap(b);
    }
}

// E-values of one query's scores, each score's computed once while it stays in
// the table (12,312 HSPs of 4,999 residues: a few hundred scores).
class EvalueTable {
public:
    void query(const blaze_params &p, uint32_t q) {
        p_ = &p;
        tag_ = (static_cast<uint64_t>(q) + 1) << 32;
    }
    double of(int32_t score) {
        const uint64_t tag = tag_ | static_cast<uint32_t>(score);
        Slot &s = slots_[static_cast<uint32_t>(score) % kSlots];
        if (s.tag != tag) {
            s.tag = tag;
            s.e = p_->eff_searchsp * p_->K * std::exp(-p_->lambda * static_cast<double>(score));
        }
        return s.e;
    }

private:
    static constexpr uint32_t kSlots = 512;
    struct Slot {
        uint64_t tag = 0;
        double e = 0.0;
    };
    Slot slots_[kSlots];
    const blaze_params *p_ = nullptr;
    uint64_t tag_ = 0;
};

// Runs both stages (growing buffers and repeating a pass that overflowed),
// copies the HSPs back and finishes them: E-values, preliminary reap, order
// by (query, OID).
static int run_search(blaze_search *s, const RunSpec &spec, uint64_t *n_hsps) {
    blaze_db *db = s->db;
    const blaze_params *p0 = spec.p;
    const bool batched = spec.b != nullptr;
    const uint32_t nq = batched ? spec.b->n : 1;
    RunSpec r = spec;
    r.smin.resize(nq);
    for (uint32_t i = 0; i < nq; ++i) r.smin[i] = reap_min_score(r.p[i]);
    s->results.clear();
    s->batch_results.clear();
    s->stats = blaze_stats{};
    if (n_hsps) *n_hsps = 0;

    constexpr size_t kSmemBudget = 220 * 1024;
    const int reg_cap = batched ? s->batch_reg_warps : s->reg_warps[scan_query_in_smem(r.q->qlen, p0->window)];
    const int warp_cap = s->max_warps ? std::min(reg_cap, static_cast<int>(s->max_warps)) : reg_cap;
    // layout of one single-query scan launch
    const uint64_t share = db->total / (static_cast<uint64_t>(s->n_sm) * kScanMaxWarpsPerBlock);
    constexpr size_t kSmemMost = 227 * 1024 - 64;  // the opt-in limit less static shared memory
    auto layout_for = [&](int32_t qlen, uint32_t n_hits, int warps, bool queue, uint32_t band_entries = 0) {
        // A warp stages a whole group, but a part of one next to a long query's
        // table, where more warps on an SM are worth more (1,500 / 3,000 residues
        // against 140 M: 3.79 -> 3.61 and 8.16 -> 7.81 ms) -- unless there is no
        // more than a group for each warp (1,500 against 7 M: 0.35 -> 0.40)
        const bool part = band_entries == 0 && qlen > kStageQuery && (queue || share > kGroupMaxBytes);
        const uint32_t stage_bytes = part ? s->stage_bytes : std::max(s->stage_bytes, db->group_bytes);
        ScanLayout l = scan_layout(qlen, p0->window, n_hits, stage_bytes, kSmemBudget, warps, band_entries);
        // next to the longest tables only smaller groups are staged
        if (l.smem_bytes > kSmemMost)
            l = scan_layout(qlen, p0->window, n_hits, std::max(s->stage_bytes, 576u) - 576u, kSmemBudget, warps,
                            band_entries);
        // and next to the very longest only the shortest subjects, and no bitset:
        // query and window may have 56,688 residues together, with the bitset
        // 55,888 to 56,000
        if (l.smem_bytes > kSmemMost) l = scan_layout(qlen, p0->window, n_hits, 0, kSmemBudget, warps, band_entries, true);
        return l;
    };
    // layout of one batched scan launch over queries of up to `longest`
    // residues: shared memory for all the block's warps at the longest query
    // when that fits the budget, else the whole budget (at least one warp);
    // the block runs as many warps as fit for each query
    auto batch_layout_for = [&](int32_t longest, Words words) {
        ScanLayout l = layout_for(longest, UINT32_MAX, 1, true);
        const size_t regions = l.smem_bytes - l.warp_smem_bytes - words_bytes(l.words) + words_bytes(words);
        l.words = words;
        l.warps_per_block = std::max(1, std::min(warp_cap, kScanMaxWarpsPerBlock));
        l.smem_bytes = std::max(std::min(kSmemBudget, regions + static_cast<size_t>(l.warps_per_block) * l.warp_smem_bytes),
                                regions + l.warp_smem_bytes);
        return l;
    };
    // Batched: the queries in length order, one scan launch for those that
    // take the same kernel (the query in shared memory or not, its word table
    // or not).
    std::vector<uint32_t> order(nq);
    std::iota(order.begin(), order.end(), 0u);
    if (batched)
        std::stable_sort(order.begin(), order.end(),
                         [&](uint32_t a, uint32_t b) { return r.b->qlen[a] < r.b->qlen[b]; });
    auto qlen_at = [&](uint32_t k) { return batched ? r.b->qlen[order[k]] : r.q->qlen; };
    std::vector<ScanPlan> plans;
    auto query_layout = [&](uint32_t k, bool queue, uint32_t band_entries = 0) {
        return layout_for(qlen_at(k), batched ? r.b->n_off[order[k]] : r.q->n_off, warp_cap, queue, band_entries);
    };
    // One query's launch runs in bands of diagonals
    // - where a subject is so long that the launch would end in a wait for it:
    //   such subjects are cut in pieces. A warp alone on its SM takes a residue in
    //   4 ns plus 0.05 per query residue, 2.5 times as fast as next to 31 others,
    //   so the wait is for what a subject has beyond 2.5 shares of the residues (a
    //   share: all of them over 152 x 32 warps); bands cost 10 to 15 us (a buffer
    //   to clear, merging) and look words up again. 300 and 4,999 residues against
    //   17.5 M with subjects of up to 35,000: 0.81 -> 0.29 and 10.46 -> 2.83 ms; of
    //   uniform lengths up to 35,000, 100 residues against 34 / 85 / 131 M (5 / 2 /
    //   1.3 shares): 0.50 -> 0.32, 0.61 -> 0.58, 0.72 -> 0.83, 3,000 residues 6.4 ->
    //   4.5, 8.1 -> 10.2, 10.1 -> 15.3; up to 1,000, 31 residues against 0.25 / 1.6 M
    //   84 -> 86 and 80 -> 95 us;
    // - for the longest queries, with a table of one band's diagonals: tables of
    //   a whole query would leave few warps an SM. 8,000 / 12,345 / 30,000
    //   residues against 140 M: 42.0 -> 37.5, 172 -> 62 and 1,520 -> 230 ms; at
    //   5,000 (14 warps without) 19.9 -> 24.0, since every band looks up its
    //   words again. Such queries of a batch have launches of their own too.
    // A batch runs as one launch whose blocks go from query to query
    // - where a query's own pass would end in a wait for its longest subjects,
    //   that is where one of them is more than a warp's share of the residues: 16
    //   queries of 2,000 to 5,000 residues against 10.5 M residues with subjects
    //   of up to 35,000 scan in 13.1 ms, with a banded launch each in 15.4;
    // - where a query's own pass is mostly its start and its end: against fewer
    //   than 2^23 residues. 64 queries of 20 to 60 residues against 0.3 / 3 / 8 M
    //   residues of peptides in one launch 0.50 / 1.21 / 2.60 ms, in one each 1.11
    //   / 1.71 / 3.04; 64 of 50 to 500 against 3 / 8 M of proteins up to 300 2.02 /
    //   4.84 and 2.64 / 5.30.
    // Otherwise one launch per query is the faster (4 queries of 50 to 500 residues
    // against 12 M 0.593 and 0.604 ms, 17 of 1,000 to 5,000 18.2 and 18.6, 256 against
    // 35 M 100.9 and 103.9).
    constexpr uint64_t kOneLaunchResidues = 1ull << 23;
    const bool per_query = batched && (s->batch_launch == 2 ||
                                       (s->batch_launch == 0 &&
                                        (nq == 1 || (db->max_len < share && db->total >= kOneLaunchResidues))));
    const bool has_pieces = db->n_pieces + 1 > db->h_groups.size();
    auto waits_for_longest = [&](int32_t qlen) {
        const uint64_t passed = share * 5 / 2;
        return db->max_len > passed && (db->max_len - passed) * (static_cast<uint64_t>(qlen) + 80) >= 240000;
    };
    auto narrow_layout = [&](uint32_t k) { return query_layout(k, false, scan_band_entries(qlen_at(k))); };
    auto is_narrow = [&](uint32_t k) {  // (a group's bands have to be staged as one)
        return qlen_at(k) > kBandQuery && p0->window <= kTab16Window && db->n > 0 &&
               narrow_layout(k).stage_bytes >= db->group_bytes;
    };
    r.border = order;
    for (uint32_t i = 0; i < nq;) {
        uint32_t j = i + 1;
        ScanPlan pl;
        const bool narrow = is_narrow(i);
        pl.queue = batched && !per_query && (!narrow || s->batch_launch == 1);
        pl.lay = query_layout(i, pl.queue);
        const bool banded = narrow || (has_pieces && waits_for_longest(qlen_at(i)) && p0->window <= kTab16Window);
        if (pl.queue) {
            const bool smem = pl.lay.query_smem_bytes != 0;
            const Words words = pl.lay.words;
            for (; j < nq; ++j) {
                const ScanLayout l = query_layout(j, true);
                if ((l.query_smem_bytes != 0) != smem || l.words != words || is_narrow(j) != narrow) break;
            }
            pl.lay = batch_layout_for(qlen_at(j - 1), words);
        } else if (banded) {
            if (narrow) {
                pl.lay = narrow_layout(i);
                // a group's diagonals: its positions, the windows between its
                // subjects and the query
                const uint32_t reach = static_cast<uint32_t>(qlen_at(i) + p0->window * static_cast<int32_t>(kGroupMaxSubjects));
                pl.extra_bands = (reach + pl.lay.diag_entries - 1) / pl.lay.diag_entries;
            }
            pl.bands = true;
        }
        pl.first = i;
        pl.n = j - i;
        // On a small database a group holds a warp's share of one query's pass,
        // down to a subject each; a launch of many queries has groups for all its
        // warps without. 256 queries of 20 to 60 residues against 0.3 M residues of
        // peptides 1.59 -> 0.72 ms, but 17 of 1,000 to 4,000 against 0.1 M of
        // proteins up to 300 (one group for each warp) 0.387 -> 0.426.
        constexpr uint64_t kGroupsEach = 4;
        pl.batch_groups = pl.queue && db->d_batch_groups &&
                          static_cast<uint64_t>(pl.n) * db->n_batch_groups >=
                              kGroupsEach * static_cast<uint64_t>(s->n_sm) * kScanMaxWarpsPerBlock;
        if (pl.lay.smem_bytes > kSmemMost) return BLAZE_ERR_LIMIT;
        int per_sm = 0;
        if (pl.queue) {
            BLAZE_CUDA_TRY(scan_batch_occupancy(pl.lay.query_smem_bytes != 0, pl.lay.words, pl.lay.warps_per_block,
                                                pl.lay.smem_bytes, &per_sm));
        } else {
            BLAZE_CUDA_TRY(scan_occupancy(pl.lay.query_smem_bytes != 0, pl.lay.words, pl.bands,
                                          pl.lay.warps_per_block, pl.lay.smem_bytes, &per_sm));
        }
        if (per_sm < 1) return BLAZE_ERR_LIMIT;
        pl.blocks = s->n_sm * per_sm;
        plans.push_back(pl);
        i = j;
    }

    if (batched) {
        // per-query descriptors of this run in length order (cutoffs come from
        // the parameters); the per-query arrays of the gapped stage stay in
        // batch order
        std::vector<BatchQuery> bq(nq);
        std::vector<const uint8_t *> qp(nq);
        std::vector<int32_t> ql(nq), cut(nq), mh(nq);
        for (uint32_t k = 0; k < nq; ++k) {
            const uint32_t i = order[k];
            const blaze_params &pi = r.p[i];
            BatchQuery &d = bq[k];
            d.q = r.b->d_res + r.b->res_off[i];
            d.qlen = r.b->qlen[i];
            d.ungapped_cutoff = pi.ungapped_cutoff;
            d.cell_start = r.b->d_cell_start + static_cast<size_t>(i) * (kWords + 1);
            d.cell_pack = r.b->d_cell_pack + static_cast<size_t>(i) * kWords;
            d.presence = r.b->d_presence + static_cast<size_t>(i) * kPresenceWords;
            d.cell_off = r.b->d_cell_off + r.b->off_off[i];
            d.diag_entries = scan_diag_entries(d.qlen, pi.window);
            d.diag_magic = static_cast<uint32_t>((1ull << 32) / d.diag_entries + 1);
            d.diag_bytes = scan_diag_bytes(d.qlen, pi.window);
            d.index = i;
            qp[i] = d.q;
            ql[i] = d.qlen;
            cut[i] = pi.gapped_cutoff;
            mh[i] = pi.max_hsps;
        }
        int rc;
        if ((rc = s->bq.ensure(nq)) != BLAZE_OK) return rc;
        if ((rc = s->bqptr.ensure(nq)) != BLAZE_OK) return rc;
        if ((rc = s->bqlen.ensure(nq)) != BLAZE_OK) return rc;
        if ((rc = s->bcut.ensure(nq)) != BLAZE_OK) return rc;
        if ((rc = s->bsmin.ensure(nq)) != BLAZE_OK) return rc;
        if ((rc = s->bmaxh.ensure(nq)) != BLAZE_OK) return rc;
        BLAZE_CUDA_TRY(cudaMemcpyAsync(s->bq.p, bq.data(), sizeof(BatchQuery) * nq, cudaMemcpyHostToDevice, s->stream));
        BLAZE_CUDA_TRY(cudaMemcpyAsync(s->bqptr.p, qp.data(), sizeof(const uint8_t *) * nq, cudaMemcpyHostToDevice, s->stream));
        BLAZE_CUDA_TRY(cudaMemcpyAsync(s->bqlen.p, ql.data(), sizeof(int32_t) * nq, cudaMemcpyHostToDevice, s->stream));
        BLAZE_CUDA_TRY(cudaMemcpyAsync(s->bcut.p, cut.data(), sizeof(int32_t) * nq, cudaMemcpyHostToDevice, s->stream));
        BLAZE_CUDA_TRY(cudaMemcpyAsync(s->bsmin.p, r.smin.data(), sizeof(int32_t) * nq, cudaMemcpyHostToDevice, s->stream));
        BLAZE_CUDA_TRY(cudaMemcpyAsync(s->bmaxh.p, mh.data(), sizeof(int32_t) * nq, cudaMemcpyHostToDevice, s->stream));
        BLAZE_CUDA_TRY(cudaStreamSynchronize(s->stream));
        s->stats.h2d_bytes += (sizeof(BatchQuery) + sizeof(const uint8_t *) + 4 * sizeof(int32_t)) * nq;
    }

    DevCounters c{};
    int rc;
    BLAZE_CUDA_TRY(cudaEventRecord(s->ev[0], s->stream));
    for (int attempt = 0;; ++attempt) {
        if ((rc = run_pass(s, r, plans)) != BLAZE_OK) return rc;
        c = *s->h_cnt;
        {
            float ms = 0.f;
            BLAZE_CUDA_TRY(cudaEventElapsedTime(&ms, s->ev[2], s->ev[3]));
            s->stats.gapped_ms = ms;
        }
        // the DP rows fit the longest subject and the scan's init hits lie in
        // their sequences, so these two are consistency failures here
        if (c.flags & (kFlagBadState | kFlagSubjectTooLong | kFlagBadInitHit)) return BLAZE_ERR_INTERNAL;
        bool again = false;
        if (c.overflow_subjects > 0) {
            s->scratch_cap = std::max<uint32_t>(s->scratch_cap * 2, c.max_init_needed + 64);
            again = true;
        }
        if (c.flags & kFlagInitArrayFull) {
            s->init_cap = std::max<unsigned long long>(s->init_cap * 2, c.init_count + c.init_count / 4 + 1024);
            again = true;
        }
        if (c.flags & kFlagOutArrayFull) {
            s->out_cap = std::max<unsigned long long>(s->out_cap * 2, c.out_count + c.out_count / 4 + 1024);
            again = true;
        }
        if (c.flags & kFlagWorkArrayFull) {
            if (!batched) return BLAZE_ERR_INTERNAL;  // one item per subject at most
            s->work_cap = std::max<unsigned long long>(s->work_cap * 2, c.work_count + c.work_count / 4 + 1024);
            again = true;
        }
        if (!again) break;
        if (attempt >= 8) return BLAZE_ERR_INTERNAL;
        s->stats.reruns++;
    }

    // hit lists: a query keeping more subjects than its hitlist_size keeps
    // the hitlist_size best on the device (the others' lists get n = 0)
    const size_t n_groups = static_cast<size_t>(c.group_count);
    bool limited = false;
    for (uint32_t i = 0; i < nq; ++i) limited |= r.p[i].hitlist_size > 0;
    if (limited && n_groups) {
        std::vector<uint32_t> kept_per_query(nq);
        BLAZE_CUDA_TRY(cudaMemcpyAsync(kept_per_query.data(), s->qkept.p, sizeof(uint32_t) * nq,
                                       cudaMemcpyDeviceToHost, s->stream));
        BLAZE_CUDA_TRY(cudaStreamSynchronize(s->stream));
        s->stats.d2h_bytes += sizeof(uint32_t) * nq;
        std::vector<uint32_t> seg(nq + 1, 0), sel;
        std::vector<int32_t> limit(nq);
        for (uint32_t i = 0; i < nq; ++i) {
            limit[i] = r.p[i].hitlist_size;
            const bool selects = limit[i] > 0 && kept_per_query[i] > static_cast<uint32_t>(limit[i]);
            seg[i + 1] = seg[i] + (selects ? kept_per_query[i] : 0u);
            if (selects) sel.push_back(i);
        }
        if (!sel.empty()) {
            int rc2;
            if ((rc2 = s->seg_off.ensure(nq + 1)) != BLAZE_OK) return rc2;
            if ((rc2 = s->seg_fill.ensure(nq)) != BLAZE_OK) return rc2;
            if ((rc2 = s->sel_limit.ensure(nq)) != BLAZE_OK) return rc2;
            if ((rc2 = s->sel_q.ensure(sel.size())) != BLAZE_OK) return rc2;
            if ((rc2 = s->seg_keys.ensure(seg[nq])) != BLAZE_OK) return rc2;
            if ((rc2 = s->seg_idx.ensure(seg[nq])) != BLAZE_OK) return rc2;
            BLAZE_CUDA_TRY(cudaMemcpyAsync(s->seg_off.p, seg.data(), sizeof(uint32_t) * (nq + 1),
                                           cudaMemcpyHostToDevice, s->stream));
            BLAZE_CUDA_TRY(cudaMemcpyAsync(s->sel_limit.p, limit.data(), sizeof(int32_t) * nq,
                                           cudaMemcpyHostToDevice, s->stream));
            BLAZE_CUDA_TRY(cudaMemcpyAsync(s->sel_q.p, sel.data(), sizeof(uint32_t) * sel.size(),
                                           cudaMemcpyHostToDevice, s->stream));
            BLAZE_CUDA_TRY(cudaMemsetAsync(s->seg_fill.p, 0, sizeof(uint32_t) * nq, s->stream));
            s->stats.h2d_bytes += sizeof(uint32_t) * (nq + 1) + sizeof(int32_t) * nq + sizeof(uint32_t) * sel.size();
            HitlistArgs ha{};
            ha.groups = s->groups.p;
            ha.n_groups = n_groups;
            ha.seg_off = s->seg_off.p;
            ha.seg_fill = s->seg_fill.p;
            ha.keys = s->seg_keys.p;
            ha.idx = s->seg_idx.p;
            ha.sel_queries = s->sel_q.p;
            ha.limit = s->sel_limit.p;
            BLAZE_CUDA_TRY(launch_hitlist(ha, static_cast<uint32_t>(sel.size()), s->n_sm, s->stream));
            s->stats.kernel_launches += 2;
        }
    }

    // copy back: the kept HSPs and one descriptor per subject list
    const size_t n_out = static_cast<size_t>(c.out_count);
    if ((rc = ensure_pinned(s->h_out, s->h_out_n, n_out)) != BLAZE_OK) return rc;
    if ((rc = ensure_pinned(s->h_groups, s->h_groups_n, n_groups)) != BLAZE_OK) return rc;
    if (n_out) {
        BLAZE_CUDA_TRY(cudaMemcpyAsync(s->h_out, s->out.p, sizeof(DevHsp) * n_out, cudaMemcpyDeviceToHost, s->stream));
        BLAZE_CUDA_TRY(cudaMemcpyAsync(s->h_groups, s->groups.p, sizeof(GroupDesc) * n_groups,
                                       cudaMemcpyDeviceToHost, s->stream));
        s->stats.d2h_bytes += sizeof(DevHsp) * n_out + sizeof(GroupDesc) * n_groups;
    }
    BLAZE_CUDA_TRY(cudaEventRecord(s->ev[3], s->stream));
    BLAZE_CUDA_TRY(cudaStreamSynchronize(s->stream));
    {
        float ms = 0.f;
        BLAZE_CUDA_TRY(cudaEventElapsedTime(&ms, s->ev[1], s->ev[2]));
        s->stats.scan_ms = ms;
        BLAZE_CUDA_TRY(cudaEventElapsedTime(&ms, s->ev[0], s->ev[3]));
        s->stats.device_ms = ms;
    }
    // the lists by (query, OID); E-values of the kept HSPs (the reap,
    // max_hsps and the hit list already applied on the device)
    order_lists(s, n_groups, nq);
    const std::vector<ListKey> &lists = s->order[0];
    size_t n_keep = 0;
    for (const ListKey &l : lists) n_keep += s->h_groups[l.at].n;
    if (batched) s->batch_results.resize(n_keep);
    else s->results.resize(n_keep);
    EvalueTable evalues;
    size_t to = 0;
    for (const ListKey &l : lists) {
        const GroupDesc &g = s->h_groups[l.at];
        evalues.query(r.p[g.query], g.query);
        for (uint32_t k = 0; k < g.n; ++k, ++to) {
            const DevHsp &d = s->h_out[g.first + k];
            blaze_hsp &h = batched ? s->batch_results[to].hsp : s->results[to];
            if (batched) {
                s->batch_results[to].query = g.query;
                s->batch_results[to].reserved = 0;
            }
            h.oid = g.oid;
            h.score = d.score;
            h.q_start = d.q_start;
            h.q_end = d.q_end;
            h.s_start = d.s_start;
            h.s_end = d.s_end;
            h.q_gapped_start = d.q_gs;
            h.s_gapped_start = d.s_gs;
            h.evalue = evalues.of(d.score);
        }
    }
    const uint32_t subjects = static_cast<uint32_t>(lists.size());
    const size_t n_res = batched ? s->batch_results.size() : s->results.size();
    s->last_init_count = c.init_count;
    s->last_work_count = c.work_count;
    s->last_batched = batched;
    s->last_batch = r.b;
    s->stats.residues_scanned = db->total * nq;
    s->stats.word_hits = c.word_hits;
    s->stats.ungapped_extensions = c.extensions;
    s->stats.init_hsps = c.init_count;
    s->stats.gapped_extensions = c.gapped_ext;
    s->stats.dp_cells = c.dp_cells;
    s->stats.hsps = n_res;
    s->stats.subjects_with_hsps = subjects;
    if (n_hsps) *n_hsps = n_res;
    return BLAZE_OK;
}

extern "C" int blaze_search_run(blaze_search *s, const blaze_query *q, const blaze_params *p,
                                uint64_t *n_hsps) try {
    if (!s || !q || q->device != s->db->device) return BLAZE_ERR_INVALID_ARG;
    int rc = check_params(p);
    if (rc != BLAZE_OK) return rc;
    if (p->word_threshold != q->threshold) return BLAZE_ERR_INVALID_ARG;
    BLAZE_CUDA_TRY(cudaSetDevice(s->db->device));
    RunSpec r;
    r.q = q;
    r.p = p;
    rc = run_search(s, r, n_hsps);
    s->stats.h2d_bytes += q->upload_bytes;
    return rc;
} BLAZE_ABI_CATCH

extern "C" int blaze_search_run_batch(blaze_search *s, const blaze_batch *b, const blaze_params *params,
                                      uint64_t *n_hsps) try {
    if (!s || !b || !params || b->device != s->db->device || b->n == 0) return BLAZE_ERR_INVALID_ARG;
    for (uint32_t i = 0; i < b->n; ++i) {
        int rc = check_params(&params[i]);
        if (rc != BLAZE_OK) return rc;
        const blaze_params &a = params[0], &c = params[i];
        if (c.word_threshold != b->threshold || c.window != a.window || c.ungapped_xdrop != a.ungapped_xdrop ||
            c.gap_open != a.gap_open || c.gap_extend != a.gap_extend || c.gapped_xdrop != a.gapped_xdrop)
            return BLAZE_ERR_INVALID_ARG;
    }
    BLAZE_CUDA_TRY(cudaSetDevice(s->db->device));
    RunSpec r;
    r.b = b;
    r.p = params;
    int rc = run_search(s, r, n_hsps);
    s->stats.h2d_bytes += b->upload_bytes;
    return rc;
} BLAZE_ABI_CATCH

extern "C" int blaze_search_batch_results(const blaze_search *s, blaze_batch_hsp *out, uint64_t capacity,
                                          uint64_t *n_hsps) try {
    if (!s) return BLAZE_ERR_INVALID_ARG;
    if (n_hsps) *n_hsps = s->batch_results.size();
    if (capacity < s->batch_results.size()) return BLAZE_ERR_OUTPUT_TOO_SMALL;
    if (!s->batch_results.empty()) {
        if (!out) return BLAZE_ERR_INVALID_ARG;
        std::memcpy(out, s->batch_results.data(), sizeof(blaze_batch_hsp) * s->batch_results.size());
    }
    return BLAZE_OK;
} BLAZE_ABI_CATCH

extern "C" int blaze_search_set_tuning(blaze_search *s, const blaze_tuning *t) try {
    if (!s || !t) return BLAZE_ERR_INVALID_ARG;
    if (t->stage_bytes > 16384 || t->max_warps_per_block > static_cast<uint32_t>(kScanMaxWarpsPerBlock))
        return BLAZE_ERR_LIMIT;
    if (t->launch_mode > 2 || t->batch_launch > 2) return BLAZE_ERR_INVALID_ARG;
    s->launch_mode = t->launch_mode;
    s->batch_launch = t->batch_launch;
    s->stage_bytes = t->stage_bytes ? t->stage_bytes : kScanStageBytes;
    s->max_warps = t->max_warps_per_block;
    return BLAZE_OK;
} BLAZE_ABI_CATCH

extern "C" int blaze_search_results(const blaze_search *s, blaze_hsp *out, uint64_t capacity,
                                    uint64_t *n_hsps) try {
    if (!s) return BLAZE_ERR_INVALID_ARG;
    if (n_hsps) *n_hsps = s->results.size();
    if (capacity < s->results.size()) return BLAZE_ERR_OUTPUT_TOO_SMALL;
    if (!s->results.empty()) {
        if (!out) return BLAZE_ERR_INVALID_ARG;
        std::memcpy(out, s->results.data(), sizeof(blaze_hsp) * s->results.size());
    }
    return BLAZE_OK;
} BLAZE_ABI_CATCH

extern "C" int blaze_search_stats(const blaze_search *s, blaze_stats *out) {
    if (!s || !out) return BLAZE_ERR_INVALID_ARG;
    *out = s->stats;
    return BLAZE_OK;
}

extern "C" int blaze_search_init_hits(blaze_search *s, blaze_init_hit *out, uint64_t capacity,
                                      uint64_t *n_hits) try {
    if (!s || s->last_batched) return BLAZE_ERR_INVALID_ARG;  // single-query runs only
    const size_t n_init = static_cast<size_t>(s->last_init_count);
    const size_t n_work = static_cast<size_t>(s->last_work_count);
    if (n_hits) *n_hits = n_init;
    if (capacity < n_init) return BLAZE_ERR_OUTPUT_TOO_SMALL;
    if (n_init == 0) return BLAZE_OK;
    if (!out) return BLAZE_ERR_INVALID_ARG;
    BLAZE_CUDA_TRY(cudaSetDevice(s->db->device));
    std::vector<InitHit> hits(n_init);
    std::vector<WorkItem> work(n_work);
    BLAZE_CUDA_TRY(cudaMemcpy(hits.data(), s->init_out.p, sizeof(InitHit) * n_init, cudaMemcpyDeviceToHost));
    BLAZE_CUDA_TRY(cudaMemcpy(work.data(), s->work.p, sizeof(WorkItem) * n_work, cudaMemcpyDeviceToHost));
    std::sort(work.begin(), work.end(), [&](const WorkItem &a, const WorkItem &b) {
        return s->db->oid_of[a.subject] < s->db->oid_of[b.subject];
    });
    size_t k = 0;
    for (const WorkItem &w : work) {
        std::vector<InitHit> sub(hits.begin() + w.first, hits.begin() + w.first + w.n_init);
        std::sort(sub.begin(), sub.end(), [](const InitHit &x, const InitHit &y) {
            if (x.score != y.score) return x.score > y.score;
            if (x.s_trig != y.s_trig) return x.s_trig < y.s_trig;
            return x.q_trig < y.q_trig;
        });
        for (const InitHit &h : sub) {
            blaze_init_hit &o = out[k++];
            o.oid = s->db->oid_of[w.subject];
            o.q_start = h.q_start;
            o.s_start = h.s_start;
            o.length = h.len;
            o.score = h.score;
            o.q_trigger = h.q_trig;
            o.s_trigger = h.s_trig;
        }
    }
    if (n_hits) *n_hits = k;
    return k == n_init ? BLAZE_OK : BLAZE_ERR_INTERNAL;
} BLAZE_ABI_CATCH

// One call with host buffers: the query's residues go through pinned staging
// into a buffer the search context keeps (grown on demand), and its lookup is
// built there on the search's stream ahead of the kernels -- no allocation and
// no device-wide synchronisation per query once warm.
extern "C" int blaze_prelim_search(blaze_search *s, const uint8_t *query, int32_t length,
                                   const blaze_params *p, blaze_hsp *out, uint64_t capacity,
                                   uint64_t *n_hsps) try {
    if (!s || !p || !query || length <= 0) return BLAZE_ERR_INVALID_ARG;
    if (length > kMaxQueryLength) return BLAZE_ERR_LIMIT;
    if (!valid_residues(query, static_cast<uint64_t>(length))) return BLAZE_ERR_INVALID_ARG;
    int rc = check_params(p);
    if (rc != BLAZE_OK) return rc;
    BLAZE_CUDA_TRY(cudaSetDevice(s->db->device));
    blaze_query q;  // a view of the search's buffer; not freed
    q.device = s->db->device;
    q.qlen = length;
    q.threshold = p->word_threshold;
    q.n_off = lookup_hits(query, length, p->word_threshold);
    const QueryTables t(length, q.n_off);
    q.upload_bytes = t.res_bytes;
    if ((rc = ensure_pinned(s->h_stage, s->h_stage_n, t.res_bytes)) != BLAZE_OK) return rc;
    std::memcpy(s->h_stage, query, length);
    std::memset(s->h_stage + length, 0, t.res_bytes - static_cast<size_t>(length));
    if ((rc = s->qt.ensure(t.bytes)) != BLAZE_OK) return rc;
    t.point(q, s->qt.p);
    // A search that is refused waits for nothing: then the copy has to end here,
    // since the next call overwrites the staging, and other residues under the
    // lookup's kernels could have more hits than the tables have room for.
    struct StreamWait {
        cudaStream_t st;
        bool on = true;
        ~StreamWait() {
            if (on) cudaStreamSynchronize(st);
        }
    } wait{s->stream};
    BLAZE_CUDA_TRY(cudaMemcpyAsync(q.d_q, s->h_stage, t.res_bytes, cudaMemcpyHostToDevice, s->stream));
    BLAZE_CUDA_TRY(build_lookup(q, s->stream));
    RunSpec r;
    r.q = &q;
    r.p = p;
    rc = run_search(s, r, n_hsps);
    s->stats.h2d_bytes += q.upload_bytes;
    s->stats.kernel_launches += kLookupKernels;
    if (rc != BLAZE_OK) return rc;
    wait.on = false;  // the search has waited
    return blaze_search_results(s, out, capacity, n_hsps);
} BLAZE_ABI_CATCH
