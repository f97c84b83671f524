// batch.cu -- query batches of the batched form: every query's residues and
// word tables in one set of device arrays (refilled in place by the serving
// loop).
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "handles.h"
#include "internal.h"

static int check_batch_input(const uint8_t *residues, const uint64_t *offsets, uint32_t n_queries) {
    if (!residues || !offsets || n_queries == 0) return BLAZE_ERR_INVALID_ARG;
    for (uint32_t i = 0; i < n_queries; ++i) {
        if (offsets[i + 1] <= offsets[i]) return BLAZE_ERR_INVALID_ARG;
        if (offsets[i + 1] - offsets[i] > static_cast<uint64_t>(kMaxQueryLength)) return BLAZE_ERR_LIMIT;
        if (!valid_residues(residues + offsets[i], offsets[i + 1] - offsets[i])) return BLAZE_ERR_INVALID_ARG;
    }
    return BLAZE_OK;
}

// Uploads every query's residues and builds their lookups on the device, in
// the batch's buffers, growing those only when they are too small (so that a
// refilled batch allocates nothing once it has seen its largest load). The work
// goes on `stream` (null: the default one) and is done on return.
static int batch_fill(blaze_batch *b, const uint8_t *residues, const uint64_t *offsets, uint32_t n_queries,
                      int32_t word_threshold, cudaStream_t stream) {
    b->n = n_queries;
    b->threshold = word_threshold;
    b->qlen.clear();
    b->res_off.clear();
    b->off_off.clear();
    b->n_off.clear();
    std::vector<uint8_t> res;
    uint64_t n_offs = 0;
    for (uint32_t i = 0; i < n_queries; ++i) {
        const int32_t len = static_cast<int32_t>(offsets[i + 1] - offsets[i]);
        const uint8_t *q = residues + offsets[i];
        b->qlen.push_back(len);
        b->res_off.push_back(res.size());
        res.insert(res.end(), q, q + len);
        res.resize((res.size() + 63) & ~static_cast<size_t>(63), 0);  // 64-byte separation
        b->off_off.push_back(n_offs);
        b->n_off.push_back(lookup_hits(q, len, word_threshold));
        n_offs += b->n_off.back();
    }
    res.resize(res.size() + 64, 0);
    // a refill grows by half again so that slowly rising loads settle
    const size_t slack = stream ? 2 : 1;
    auto grow = [&](auto &buf, size_t want) {
        return want <= buf.n ? BLAZE_OK : buf.ensure(want + (slack - 1) * want / 2);
    };
    int rc = grow(b->res, res.size());
    if (rc == BLAZE_OK) rc = grow(b->cell_start, static_cast<size_t>(n_queries) * (kWords + 1));
    if (rc == BLAZE_OK) rc = grow(b->cell_pack, static_cast<size_t>(n_queries) * kWords);
    if (rc == BLAZE_OK) rc = grow(b->presence, static_cast<size_t>(n_queries) * kPresenceWords);
    if (rc == BLAZE_OK) rc = grow(b->cell_off, std::max<uint64_t>(n_offs, 1));
    if (rc == BLAZE_OK) rc = grow(b->lookups, n_queries);
    if (rc != BLAZE_OK) return rc;
    b->d_res = b->res.p;
    b->d_cell_start = b->cell_start.p;
    b->d_cell_pack = b->cell_pack.p;
    b->d_presence = b->presence.p;
    b->d_cell_off = b->cell_off.p;
    std::vector<LookupQuery> lookups(n_queries);
    for (uint32_t i = 0; i < n_queries; ++i)
        lookups[i] = LookupQuery{b->d_res + b->res_off[i], b->qlen[i],
                                 b->d_cell_start + static_cast<size_t>(i) * (kWords + 1),
                                 b->d_cell_pack + static_cast<size_t>(i) * kWords,
                                 b->d_presence + static_cast<size_t>(i) * kPresenceWords, b->d_cell_off + b->off_off[i]};
    cudaError_t e = cudaMemcpyAsync(b->d_res, res.data(), res.size(), cudaMemcpyHostToDevice, stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(b->lookups.p, lookups.data(), sizeof(LookupQuery) * n_queries, cudaMemcpyHostToDevice,
                            stream);
    if (e == cudaSuccess) e = launch_lookup(LookupQuery{}, b->lookups.p, n_queries, word_threshold, stream);
    // the host arrays die with this frame, and searches run on other streams
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    b->upload_bytes = res.size() + sizeof(LookupQuery) * n_queries;
    b->device_bytes = b->res.n + sizeof(uint32_t) * (b->cell_start.n + b->cell_pack.n + b->presence.n) +
                      sizeof(uint16_t) * b->cell_off.n + sizeof(LookupQuery) * b->lookups.n;
    if (e != cudaSuccess) {
        last_cuda_error(e);
        return e == cudaErrorMemoryAllocation ? BLAZE_ERR_OUT_OF_MEMORY : BLAZE_ERR_CUDA;
    }
    return BLAZE_OK;
}

extern "C" int blaze_batch_create(const blaze_db *db, const uint8_t *residues, const uint64_t *offsets,
                                  uint32_t n_queries, int32_t word_threshold, blaze_batch **out) try {
    if (!db || !out) return BLAZE_ERR_INVALID_ARG;
    *out = nullptr;
    const int vrc = check_batch_input(residues, offsets, n_queries);
    if (vrc != BLAZE_OK) return vrc;
    BLAZE_CUDA_TRY(cudaSetDevice(db->device));
    auto *b = new blaze_batch();
    b->device = db->device;
    const int rc = batch_fill(b, residues, offsets, n_queries, word_threshold, nullptr);
    if (rc != BLAZE_OK) {
        blaze_batch_free(b);
        return rc;
    }
    *out = b;
    return BLAZE_OK;
} BLAZE_ABI_CATCH

int batch_refill(blaze_search *s, blaze_batch **inout, const uint8_t *residues, const uint64_t *offsets,
                 uint32_t n_queries, int32_t word_threshold) {
    if (!s || !inout) return BLAZE_ERR_INVALID_ARG;
    const int vrc = check_batch_input(residues, offsets, n_queries);
    if (vrc != BLAZE_OK) return vrc;
    BLAZE_CUDA_TRY(cudaSetDevice(s->db->device));
    if (!*inout) {
        *inout = new blaze_batch();
        (*inout)->device = s->db->device;
    }
    return batch_fill(*inout, residues, offsets, n_queries, word_threshold, s->stream);
}

extern "C" int blaze_batch_free(blaze_batch *b) {
    if (!b) return BLAZE_OK;
    cudaSetDevice(b->device);
    b->res.release();
    b->cell_start.release();
    b->cell_pack.release();
    b->presence.release();
    b->cell_off.release();
    b->lookups.release();
    delete b;
    return BLAZE_OK;
}

extern "C" int blaze_batch_info(const blaze_batch *b, uint32_t *n_queries, uint64_t *device_bytes) {
    if (!b) return BLAZE_ERR_INVALID_ARG;
    if (n_queries) *n_queries = b->n;
    if (device_bytes) *device_bytes = b->device_bytes;
    return BLAZE_OK;
}
