// host.cpp -- host-side pieces of libblaze103 that need no GPU: the BLOSUM62
// table, the size of a query's word lookup and the NCBI-default search parameters.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <vector>

#include "common.cuh"

namespace blaze {

const int32_t kBlosum62[kAlphabet][kAlphabet] = {
#include "blosum62.inc"
};

namespace {

// Size of every three-letter word's neighbourhood for one threshold: the words
// v with score(w, v) >= threshold, and w itself (BLAZE_ncbi/
// prelim_stage.cpp:135-155 enumerates the same set; :378-383 keeps the exact
// word). No v has the letter 0, whatever the threshold: residues are 1 and up,
// and the scan takes zeros around its subjects for words without hits. Computed
// once per threshold and kept (44 KB) for a few of them.
std::mutex g_nb_mutex;
using NeighbourhoodSizes = std::shared_ptr<const std::vector<uint16_t>>;
std::map<int32_t, NeighbourhoodSizes> g_nb_cache;
constexpr size_t kNbCacheMost = 32;

NeighbourhoodSizes neighbourhood_sizes(int32_t threshold) {
    std::lock_guard<std::mutex> lock(g_nb_mutex);
    auto it = g_nb_cache.find(threshold);
    if (it != g_nb_cache.end()) return it->second;
    auto sizes = std::make_shared<std::vector<uint16_t>>(kWords);
    std::vector<uint16_t> &size = *sizes;
    int32_t row_max[kAlphabet];
    for (int a = 0; a < kAlphabet; ++a)
        row_max[a] = *std::max_element(kBlosum62[a], kBlosum62[a] + kAlphabet);
    for (int w = 0; w < kWords; ++w) {
        const int x = w / 784, y = (w / 28) % 28, z = w % 28;
        uint32_t n = kBlosum62[x][x] + kBlosum62[y][y] + kBlosum62[z][z] < threshold ? 1 : 0;
        for (int a = 1; a < kAlphabet; ++a) {
            const int32_t s0 = kBlosum62[x][a];
            if (s0 + row_max[y] + row_max[z] < threshold) continue;
            for (int b = 1; b < kAlphabet; ++b) {
                const int32_t s1 = s0 + kBlosum62[y][b];
                if (s1 + row_max[z] < threshold) continue;
                for (int c = 1; c < kAlphabet; ++c) n += s1 + kBlosum62[z][c] >= threshold ? 1u : 0u;
            }
        }
        size[w] = static_cast<uint16_t>(n);  // at most 27^3
    }
    if (g_nb_cache.size() >= kNbCacheMost) g_nb_cache.clear();
    return g_nb_cache.emplace(threshold, std::move(sizes)).first->second;
}

}  // namespace

uint32_t lookup_hits(const uint8_t *query, int32_t qlen, int32_t threshold) {
    const NeighbourhoodSizes sizes = neighbourhood_sizes(threshold);
    const std::vector<uint16_t> &size = *sizes;
    uint32_t n = 0;
    for (int32_t i = 0; i + kWordSize <= qlen; ++i) n += size[query[i] * 784 + query[i + 1] * 28 + query[i + 2]];
    return n;
}

// Karlin-Altschul constants of BLOSUM62 (published NCBI table values).
namespace ka {
constexpr double kUngappedLambda = 0.3176, kUngappedK = 0.134;
constexpr double kGappedLambda = 0.267, kGappedK = 0.041;  // gap open 11, extend 1
constexpr double kGappedAlpha = 1.9, kGappedBeta = -30.0;
constexpr double kLn2 = 0.69314718055994530942;
constexpr double kGapTriggerBits = 22.0;        // blastp default gap trigger
constexpr double kUngappedXdropBits = 7.0;      // blastp default ungapped X-drop
constexpr double kGappedXdropBits = 15.0;       // blastp default preliminary gapped X-drop
}  // namespace ka

// Edge-effect length adjustment: the largest integer ell >= 0 strictly below
// the fixed point of beta + (alpha/lambda)(ln K + ln((m-ell)(n-N ell))) that
// keeps K(m-ell)(n-N ell) above max(m, n) (Altschul & Gish 1996).
static int32_t length_adjustment(double K, double alpha_d_lambda, double beta, int32_t m_len,
                                 uint64_t n_len, uint32_t n_seqs) {
    const double m = m_len, n = static_cast<double>(n_len), N = n_seqs;
    const double logK = std::log(K), floor_sp = std::max(m, n);
    auto feasible = [&](int32_t ell) {
        const double mm = m - ell, nn = n - N * ell;
        if (mm <= 0 || nn <= 0 || K * mm * nn <= floor_sp) return false;
        return beta + alpha_d_lambda * (logK + std::log(mm) + std::log(nn)) > ell;
    };
    int32_t lo = 0, hi = std::max(m_len - 1, 0), best = 0;
    while (lo <= hi) {  // feasible() is true up to the answer and false after it
        const int32_t mid = lo + (hi - lo) / 2;
        if (feasible(mid)) {
            best = mid;
            lo = mid + 1;
        } else {
            hi = mid - 1;
        }
    }
    return best;
}

int default_params(int32_t qlen, uint64_t db_len, uint32_t db_n, double evalue, blaze_params *p) {
    if (!p || qlen <= 0 || evalue <= 0) return BLAZE_ERR_INVALID_ARG;
    using namespace ka;
    std::memset(p, 0, sizeof(*p));
    p->word_threshold = 11;
    p->window = 40;
    p->gap_open = 11;
    p->gap_extend = 1;
    p->ungapped_xdrop = static_cast<int32_t>(std::ceil(kUngappedXdropBits * kLn2 / kUngappedLambda));
    p->gapped_xdrop = static_cast<int32_t>(kGappedXdropBits * kLn2 / kGappedLambda);
    p->lambda = kGappedLambda;
    p->K = kGappedK;
    const int32_t ell = length_adjustment(kGappedK, kGappedAlpha / kGappedLambda, kGappedBeta, qlen,
                                          db_len, db_n);
    const double eff_q = std::max<double>(qlen - ell, 1.0);
    const double eff_db = std::max<double>(static_cast<double>(db_len) - static_cast<double>(db_n) * ell, 1.0);
    p->eff_searchsp = eff_q * eff_db;
    // smallest raw score whose E-value over the search space is <= evalue
    const double s = std::log(kGappedK * p->eff_searchsp / evalue) / kGappedLambda;
    p->gapped_cutoff = std::max<int32_t>(static_cast<int32_t>(std::ceil(s)), 1);
    const int32_t gap_trigger = static_cast<int32_t>(
        (kGapTriggerBits * kLn2 + std::log(kUngappedK)) / kUngappedLambda);
    p->ungapped_cutoff = std::min(gap_trigger, p->gapped_cutoff);
    p->prelim_evalue = evalue;
    p->hitlist_size = 0;
    p->max_hsps = 0;
    return BLAZE_OK;
}

}  // namespace blaze

extern "C" const char *blaze_status_string(int status) {
    switch (status) {
        case BLAZE_OK: return "ok";
        case BLAZE_ERR_INVALID_ARG: return "invalid argument";
        case BLAZE_ERR_CUDA: return "CUDA runtime error";
        case BLAZE_ERR_NO_DEVICE: return "no usable CUDA device";
        case BLAZE_ERR_OUT_OF_MEMORY: return "out of memory";
        case BLAZE_ERR_OUTPUT_TOO_SMALL: return "output buffer too small";
        case BLAZE_ERR_LIMIT: return "request exceeds a library limit";
        case BLAZE_ERR_INTERNAL: return "internal consistency check failed";
        default: return "unknown status";
    }
}

extern "C" int blaze_params_default(int32_t query_length, uint64_t db_residues, uint32_t db_subjects,
                                    double evalue, blaze_params *out) {
    return blaze::default_params(query_length, db_residues, db_subjects, evalue, out);
}
