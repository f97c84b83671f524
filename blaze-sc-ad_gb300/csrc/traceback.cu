// traceback.cu -- the traceback stage on GB300 (sm_103a): every HSP of a
// preliminary result is aligned again from its gapped start point with the
// final X-drop, keeping the path, and its identities, mismatches and gaps are
// counted from that path (the published gapped-BLAST traceback; in the
// reference this is NCBI's traceback stage after the preliminary search,
// BLAZE_ncbi/prelim_stage.cpp:1462-1498).
//
// One warp per side of an HSP. The X-drop DP runs row by row with its band in
// registers, as in the gapped stage; every row's direction bytes go to the
// warp's buffer. The warp then walks the path back from the best cell, 32 cells
// of a diagonal at a time. Where the band outgrows the registers, or the gap
// costs or the X-drop are too large for them, the rows are kept in memory and
// one lane walks; X-drops with such bands go there at once.
#include <cstdint>

#include "common.cuh"

namespace blaze {
namespace {

__device__ const int32_t g_blosum_tb[kAlphabet * kAlphabet] = {
#include "blosum62.inc"
};

constexpr unsigned kFull = 0xffffffffu;
// direction byte: bits 0-1 where H came from (diagonal, vertical gap E,
// horizontal gap F); the E handed down extends; the F handed right extends;
// the cell is dead
constexpr uint8_t kTbDiag = 0, kTbE = 1, kTbF = 2, kTbEExt = 4, kTbFExt = 8, kTbDead = 128;

struct DirRows {
    uint8_t *dir;
    int32_t *rows;  // first, end, offset per row
    unsigned long long cap;
    uint32_t row_cap;
    bool overflow;
};

// The gapped stage's row-parallel X-drop DP with each computed cell's
// direction recorded. The sources follow the sequential recurrence: H takes
// the diagonal unless the vertical gap is larger, and either unless the
// horizontal gap is larger; a gap state handed on extends unless opening from
// H is strictly larger. (Values of dead cells may differ from the sequential
// DP's; a path never passes through one.)
template <bool REV>
__device__ int32_t xdrop_dp_dirs(const uint8_t *__restrict__ A, const uint8_t *__restrict__ B, int32_t M,
                                 int32_t N, int32_t gap_open, int32_t gap_extend, int32_t xdrop, const int32_t *mat,
                                 int32_t *Hb, int32_t *Eb, int32_t *a_best, int32_t *b_best, DirRows &d,
                                 int32_t *rows_used, int32_t *cells) {
    const int lane = threadIdx.x & 31;
    const int32_t goe = gap_open + gap_extend, ge = gap_extend;
    if (xdrop < goe) xdrop = goe;
    *a_best = 0;
    *b_best = 0;
    *rows_used = 0;
    if (M <= 0 || N <= 0) return 0;
    if (static_cast<uint32_t>(M) + 1 > d.row_cap || static_cast<unsigned long long>(N) + 2 > d.cap) {
        d.overflow = true;
        return 0;
    }
    int32_t bsize = 1 + min(N, (xdrop - goe) / ge + 1);
    for (int32_t i = lane; i < bsize; i += 32) {
        const int32_t h = i == 0 ? 0 : -goe - (i - 1) * ge;
        Hb[i] = h;
        Eb[i] = h - goe;
        d.dir[i] = i == 0 ? kTbDiag : static_cast<uint8_t>(kTbF | kTbFExt);  // row 0: gap from the origin
    }
    if (lane == 0) {
        d.rows[0] = 0;
        d.rows[1] = bsize;
        d.rows[2] = 0;
    }
    unsigned long long at = static_cast<unsigned long long>(bsize);
    __syncwarp();
    int32_t best = 0, first = 0, ab = 0, bb = 0, a = 1;
    for (; a <= M; ++a) {
        if (at + static_cast<unsigned long long>(N + 2 - first) > d.cap) {
            d.overflow = true;
            break;
        }
        const int32_t *row = mat + kAlphabet * (REV ? A[M - a] : A[a]);
        const int32_t row_first = first;
        *cells += bsize - first;
        int32_t carry_p = kNeg, carry_best = best, carry_hold = kNeg;
        int32_t first_alive = -1, last_alive = -1, row_best = best, row_best_b = -1;
        for (int32_t c0 = first; c0 < bsize; c0 += 32) {
            const int32_t b = c0 + lane;
            const bool act = b < bsize;
            const int32_t hold = act ? Hb[b] : kNeg;
            const int32_t ein = act ? Eb[b] : kNeg;
            int32_t hprev = __shfl_up_sync(kFull, hold, 1);
            if (lane == 0) hprev = carry_hold;
            const int32_t diag = (act && b > first) ? hprev + row[REV ? B[N - b] : B[b]] : kNeg;
            const int32_t D = max(ein, diag);
            const int32_t P = act ? max(D, kNeg) + ge * b : kNeg;
            int32_t incl = P;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int32_t x = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl = max(incl, x);
            }
            int32_t excl = __shfl_up_sync(kFull, incl, 1);
            if (lane == 0) excl = kNeg;
            excl = max(excl, carry_p);
            const int32_t G = excl - goe + ge - ge * b;
            const int32_t H = max(D, G);
            // the best so far in row-major order: only a segment whose largest
            // H beats the carried best needs the prefix maximum
            const int32_t hv = act ? H : INT32_MIN;
            const int32_t cm = __reduce_max_sync(kFull, hv);
            int32_t cur_best = carry_best;
            if (cm > carry_best) {
                int32_t inclh = hv;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int32_t x = __shfl_up_sync(kFull, inclh, o);
                    if (lane >= o) inclh = max(inclh, x);
                }
                int32_t exclh = __shfl_up_sync(kFull, inclh, 1);
                if (lane == 0) exclh = INT32_MIN;
                cur_best = max(carry_best, exclh);
                const unsigned mm = __ballot_sync(kFull, act && H == cm);
                row_best = cm;
                row_best_b = c0 + __ffs(mm) - 1;
                carry_best = cm;
            }
            const bool alive = act && (cur_best - H <= xdrop);
            const unsigned am = __ballot_sync(kFull, alive);
            if (am) {
                if (first_alive < 0) first_alive = c0 + __ffs(am) - 1;
                last_alive = c0 + 31 - __clz(am);
            }
            carry_hold = __shfl_sync(kFull, hold, 31);
            carry_p = max(carry_p, __shfl_sync(kFull, incl, 31));
            __syncwarp();
            if (act) {
                uint8_t dv = kTbDead;
                if (alive) {
                    dv = max(diag, ein) < G ? kTbF : (diag < ein ? kTbE : kTbDiag);
                    if (!(H - goe > ein - ge)) dv |= kTbEExt;
                    if (!(H - goe > G - ge)) dv |= kTbFExt;
                    Eb[b] = max(H - goe, ein - ge);
                    Hb[b] = H;
                } else if (first_alive >= 0 && b > first_alive) {
                    Hb[b] = kNeg;
                }
                d.dir[at + static_cast<unsigned long long>(b - row_first)] = dv;
            }
            __syncwarp();
        }
        int32_t row_end = bsize;
        if (first_alive < 0) {
            if (lane == 0) {
                d.rows[3 * a] = row_first;
                d.rows[3 * a + 1] = row_end;
                d.rows[3 * a + 2] = static_cast<int32_t>(at);
            }
            at += static_cast<unsigned long long>(row_end - row_first);
            ++a;
            break;
        }
        if (row_best_b >= 0) {
            best = row_best;
            ab = a;
            bb = row_best_b;
        }
        first = first_alive;
        if (last_alive < bsize - 1) {
            bsize = last_alive + 1;
        } else {
            const int32_t F = carry_p - goe + ge - ge * bsize;
            const int32_t thr = best - xdrop;
            if (F >= thr && bsize <= N) {
                const int32_t n_ext = min(N - bsize + 1, (F - thr) / ge + 1);
                for (int32_t t = lane; t < n_ext; t += 32) {
                    Hb[bsize + t] = F - t * ge;
                    Eb[bsize + t] = F - t * ge - goe;
                    d.dir[at + static_cast<unsigned long long>(bsize + t - row_first)] =
                        static_cast<uint8_t>(kTbF | kTbFExt);  // the row gap continues
                }
                bsize += n_ext;
            }
            row_end = bsize;
        }
        if (bsize <= N) {
            if (lane == 0) {
                Hb[bsize] = kNeg;
                Eb[bsize] = kNeg;
                d.dir[at + static_cast<unsigned long long>(bsize - row_first)] = kTbDead;  // sentinel column
            }
            ++bsize;
            row_end = bsize;
        }
        if (lane == 0) {
            d.rows[3 * a] = row_first;
            d.rows[3 * a + 1] = row_end;
            d.rows[3 * a + 2] = static_cast<int32_t>(at);
        }
        at += static_cast<unsigned long long>(row_end - row_first);
        __syncwarp();
    }
    *rows_used = a;
    *a_best = ab;
    *b_best = bb;
    __syncwarp();
    return best;
}

struct Walk {
    int32_t pairs, identities, positives, gaps, gap_opens;
    int last_move;
    bool ok;
};

__device__ __forceinline__ bool dir_at(const DirRows &d, int32_t rows, int32_t a, int32_t b, uint8_t *v) {
    if (a < 0 || a >= rows) return false;
    const int32_t f = d.rows[3 * a], e = d.rows[3 * a + 1];
    if (b < f || b >= e) return false;
    *v = d.dir[static_cast<unsigned long long>(d.rows[3 * a + 2]) + static_cast<unsigned long long>(b - f)];
    return true;
}

// Lane 0: the path from (a, b) back to the origin.
template <bool REV>
__device__ Walk walk_back(const DirRows &d, int32_t rows, const uint8_t *A, const uint8_t *B, int32_t M, int32_t N,
                          int32_t a, int32_t b, const int32_t *mat) {
    Walk w{0, 0, 0, 0, 0, -1, true};
    int state = 0, prev = -1;
    long long guard = 2ll * (M + N) + 8;
    while ((a > 0 || b > 0) && guard-- > 0) {
        int move;
        uint8_t v = 0;
        if (state == 0) {
            if (a == 0) {
                state = 2;
                continue;
            }
            if (!dir_at(d, rows, a, b, &v) || (v & kTbDead)) {
                w.ok = false;
                return w;
            }
            const int src = v & 3;
            if (src == kTbDiag) {
                const uint32_t x = REV ? A[M - a] : A[a], y = REV ? B[N - b] : B[b];
                ++w.pairs;
                w.identities += x == y;
                w.positives += mat[x * kAlphabet + y] > 0;
                move = 0;
                --a;
                --b;
            } else {
                state = src == kTbE ? 1 : 2;
                continue;
            }
        } else if (state == 1) {
            if (a - 1 > 0 && !dir_at(d, rows, a - 1, b, &v)) {
                w.ok = false;
                return w;
            }
            move = 1;
            ++w.gaps;
            if (a - 1 == 0 || !(v & kTbEExt)) state = 0;
            --a;
        } else {
            if (!dir_at(d, rows, a, b - 1, &v)) {
                w.ok = false;
                return w;
            }
            move = 2;
            ++w.gaps;
            if (!(v & kTbFExt) || (a == 0 && b - 1 == 0)) state = 0;
            --b;
        }
        if (move != 0 && move != prev) ++w.gap_opens;
        prev = move;
        w.last_move = move;
    }
    w.ok = w.ok && a == 0 && b == 0;
    return w;
}

// The same DP with the band in registers: a window of 192 columns, parts of 64,
// lane i holding H and E of columns w0 + 2i and w0 + 2i + 1 of each. A part is
// computed only in rows whose band reaches it; the window moves right when the
// band outgrows its first part. A row's direction bytes begin at its own w0:
// d.rows holds w0 and where they are. H of every dead cell is -inf, and E of a
// dead cell is at most its H was, so neither changes a live cell's direction.
// Row letter k is Q[dir * k], column letter k is S[dir * k]. Returns false when
// the band does not fit the window.
//
// Bound by instruction issue and by the chain of a row's steps. 7,756 sides of
// 500 query residues: 1.20 ms with the rows in memory, both sides on one warp and
// one lane walking back; 1.06 with 128 columns (many bands outgrow them), 0.62
// with 192 and 20 warps an SM, 0.70 with 192 or 256 and 16 warps.
constexpr int kTbRowMost = kTbWindow + 64;  // bytes of a row: the window, moved by less than 64, holds its end
__device__ __forceinline__ bool xdrop_dp_window_dirs(const uint8_t *__restrict__ Q, const uint8_t *__restrict__ S,
                                                     int32_t dir, int32_t M, int32_t N, int32_t gap_open,
                                                     int32_t gap_extend, int32_t xdrop, const int32_t *mat, DirRows &d,
                                                     TbPart &out) {
    const int lane = threadIdx.x & 31;
    const int32_t goe = gap_open + gap_extend, ge = gap_extend;
    if (xdrop < goe) xdrop = goe;
    if (M <= 0 || N <= 0) return true;
    int32_t bsize = 1 + min(N, (xdrop - goe) / ge + 1);
    if (bsize > kTbWindow) return false;
    if (static_cast<uint32_t>(M) + 1 > d.row_cap) {
        d.overflow = true;
        return true;
    }
    int2 *rows_out = reinterpret_cast<int2 *>(d.rows);
    int32_t w0 = 0, at = 0;
    auto letter = [&](int32_t b) { return b >= 1 && b <= N ? static_cast<int32_t>(S[dir * b]) : 0; };
    int32_t h[2 * kTbParts], e[2 * kTbParts], l[2 * kTbParts];  // per part: the lane's two columns
#pragma unroll
    for (int j = 0; j < 2 * kTbParts; ++j) {
        const int32_t b = 64 * (j >> 1) + 2 * lane + (j & 1);
        l[j] = letter(b);
        h[j] = b >= bsize ? kNeg : b == 0 ? 0 : -goe - (b - 1) * ge;
        e[j] = b >= bsize ? kNeg : h[j] - goe;
    }
    int32_t best = 0, first = 0, ab = 0, bb = 0, n_cells = 0;
    int32_t rows = 0;  // lane i: the matrix row of row letter (a - 1) rounded down to 32, plus i + 1
    for (int32_t a = 1; a <= M; ++a) {
        if (static_cast<unsigned long long>(at) + kTbRowMost > d.cap) {
            d.overflow = true;
            return true;
        }
        const int32_t ai = (a - 1) & 31;
        if (ai == 0) rows = a + lane <= M ? kAlphabet * static_cast<int32_t>(Q[dir * (a + lane)]) : 0;
        const int32_t *row = mat + __shfl_sync(kFull, rows, ai);
        if (lane == 0) rows_out[a] = make_int2(w0, at);
        uint8_t *dirs = d.dir + at - w0;  // a column's byte
        n_cells += bsize - first;
        int32_t carry_p = kNeg, carry_h = kNeg;  // into the next part
        int32_t lo = INT32_MAX, hi = -1;         // the first and last live column
        int32_t row_end = w0;                    // of the parts computed
        auto part = [&](int s, int32_t &h0, int32_t &h1, int32_t &e0, int32_t &e1, int32_t l0, int32_t l1) {
            const int32_t b0 = w0 + 64 * s + 2 * lane, b1 = b0 + 1, gb = ge * b0;
            const bool in0 = b0 < bsize, in1 = b1 < bsize;
            int32_t hprev = __shfl_up_sync(kFull, h1, 1);
            if (lane == 0) hprev = carry_h;
            const int32_t g0 = hprev + row[l0], g1 = h0 + row[l1];  // by the diagonal
            const int32_t d0 = in0 ? max(g0, e0) : kNeg, d1 = in1 ? max(g1, e1) : kNeg;
            // row gap: prefix maximum of D + ge * column over the columns before each
            const int32_t p0 = d0 + gb, p1 = d1 + gb + ge;
            int32_t incl = max(p0, p1);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) incl = max(incl, __shfl_up_sync(kFull, incl, o));  // lanes < o get their own
            int32_t excl = __shfl_up_sync(kFull, incl, 1);
            if (lane == 0) excl = kNeg;
            excl = max(excl, carry_p);
            const int32_t open = ge - goe - gb;
            const int32_t f0 = excl + open, f1 = max(excl, p0) + open - ge;
            const int32_t H0 = in0 ? max(f0, d0) : kNeg, H1 = in1 ? max(f1, d1) : kNeg;
            const int32_t top = max(H0, H1), cm = __reduce_max_sync(kFull, top);
            int32_t thr0 = best - xdrop, thr1 = thr0;  // live from there on
            if (cm > best) {
                int32_t t = top;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) t = max(t, __shfl_up_sync(kFull, t, o));
                t = __shfl_up_sync(kFull, t, 1);
                if (lane > 0) thr0 = max(thr0, t - xdrop);
                thr1 = max(thr0, H0 - xdrop);
                const unsigned m0 = __ballot_sync(kFull, H0 == cm), m1 = __ballot_sync(kFull, H1 == cm);
                const int fl = __ffs(m0 | m1) - 1;
                ab = a;
                bb = w0 + 64 * s + 2 * fl + ((m0 >> fl) & 1u ? 0 : 1);
                best = cm;
            }
            const bool alive0 = H0 >= thr0, alive1 = H1 >= thr1;
            lo = min(lo, __reduce_min_sync(kFull, alive0 ? b0 : alive1 ? b1 : INT32_MAX));
            hi = max(hi, __reduce_max_sync(kFull, alive1 ? b1 : alive0 ? b0 : -1));
            auto direction = [&](bool alive, int32_t g, int32_t ein, int32_t f, int32_t H) {
                uint32_t v = max(g, ein) < f ? kTbF : g < ein ? kTbE : kTbDiag;
                if (H - goe <= ein - ge) v |= kTbEExt;
                if (H - goe <= f - ge) v |= kTbFExt;
                return alive ? v : static_cast<uint32_t>(kTbDead);
            };
            const uint32_t v0 = direction(alive0, g0, e0, f0, H0), v1 = direction(alive1, g1, e1, f1, H1);
            *reinterpret_cast<uint16_t *>(dirs + b0) = static_cast<uint16_t>(v0 | (v1 << 8));
            if (s + 1 < kTbParts) carry_h = __shfl_sync(kFull, h1, 31);
            // live cells hand on; dead ones keep their E
            if (alive0) e0 = max(H0 - goe, e0 - ge);
            if (alive1) e1 = max(H1 - goe, e1 - ge);
            h0 = alive0 ? H0 : kNeg;
            h1 = alive1 ? H1 : kNeg;
            carry_p = max(carry_p, __shfl_sync(kFull, incl, 31));
            row_end = w0 + 64 * (s + 1);
        };
#pragma unroll
        for (int s = 0; s < kTbParts; ++s)
            if (s == 0 || bsize > w0 + 64 * s) part(s, h[2 * s], h[2 * s + 1], e[2 * s], e[2 * s + 1], l[2 * s], l[2 * s + 1]);
        if (hi < 0) break;
        first = lo;
        const int32_t from = hi + 1;  // columns from here on are outside, or the row gap's
        int32_t n_ext = 0, F = 0;
        if (from == bsize && bsize <= N) {
            F = carry_p - goe + ge - ge * bsize;
            const int32_t room = F - (best - xdrop);
            if (room >= 0) n_ext = min(N - bsize + 1, room / ge + 1);
        }
        bsize = from + n_ext;
        if (bsize <= N) ++bsize;  // the next column, -inf so far
        // move the window when the band leaves its first part (unless that
        // gains little) or the window itself
        const int32_t behind = first - w0, reach = bsize - w0, w_row = w0;
        if (reach > 64 && (behind >= 16 || reach > kTbWindow || (behind >= 4 && reach - behind < 64))) {
            const int32_t by = min(behind >> 1, 31);
            w0 += 2 * by;
            if (bsize - w0 > kTbWindow) return false;
            const int src = (lane + by) & 31;
            const bool same = lane + by < 32;
#pragma unroll
            for (int j = 0; j < 2 * kTbParts; ++j) {
                const int32_t hn = j + 2 < 2 * kTbParts ? h[j + 2 < 2 * kTbParts ? j + 2 : j] : kNeg;
                const int32_t en = j + 2 < 2 * kTbParts ? e[j + 2 < 2 * kTbParts ? j + 2 : j] : kNeg;
                const int32_t ha = __shfl_sync(kFull, h[j], src), hb = __shfl_sync(kFull, hn, src);
                const int32_t ea = __shfl_sync(kFull, e[j], src), eb = __shfl_sync(kFull, en, src);
                h[j] = same ? ha : hb;
                e[j] = same ? ea : eb;
            }
#pragma unroll
            for (int j = 0; j < 2 * kTbParts; ++j) l[j] = letter(w0 + 64 * (j >> 1) + 2 * lane + (j & 1));
        }
        if (n_ext > 0) {
#pragma unroll
            for (int j = 0; j < 2 * kTbParts; ++j) {
                const int32_t t = w0 + 64 * (j >> 1) + 2 * lane + (j & 1) - from;
                if (t >= 0 && t < n_ext) {
                    h[j] = F - t * ge;
                    e[j] = h[j] - goe;
                }
            }
            __syncwarp();  // the last part's bytes are there
            for (int32_t t = lane; t < n_ext; t += 32) dirs[from + t] = static_cast<uint8_t>(kTbF | kTbFExt);
        }
        at += (max(row_end, bsize) - w_row + 63) & ~63;
    }
    out.score = best;
    out.a = ab;
    out.b = bb;
    out.cells += n_cells;
    __syncwarp();
    return true;
}

// The path from the best cell of xdrop_dp_window_dirs back to the origin, by
// the whole warp: lane i looks at the cell i steps up the diagonal, and the
// leading cells that came from their diagonal are passed at once.
__device__ __forceinline__ void walk_window(const DirRows &d, const uint8_t *__restrict__ Q,
                                            const uint8_t *__restrict__ S, int32_t dir, const int32_t *mat,
                                            TbPart &p) {
    const int32_t lane = threadIdx.x & 31;
    const int2 *rows = reinterpret_cast<const int2 *>(d.rows);
    int32_t a = p.a, b = p.b;
    auto byte_at = [&](int32_t ra, int32_t cb) {  // -1: not in the row
        const int2 r = rows[ra];
        const int32_t k = cb - r.x;
        return k >= 0 && k < kTbRowMost ? static_cast<int32_t>(d.dir[r.y + k]) : -1;
    };
    p.status = 2;
    while (a > 0) {
        const int32_t ra = a - lane, cb = b - lane;
        const int32_t v = ra > 0 && cb >= 0 ? byte_at(ra, cb) : -1;
        const bool diag = cb > 0 && v >= 0 && (v & (kTbDead | 3)) == kTbDiag;
        const unsigned m = __ballot_sync(kFull, diag);
        const int32_t n = m == kFull ? 32 : __ffs(~m) - 1;
        if (n > 0) {
            const bool in = lane < n;
            const uint32_t x = in ? Q[dir * ra] : 0u, y = in ? S[dir * cb] : 0u;
            p.pairs += n;
            p.identities += __popc(__ballot_sync(kFull, in && x == y));
            p.positives += __popc(__ballot_sync(kFull, in && mat[x * kAlphabet + y] > 0));
            p.last = 0;
            a -= n;
            b -= n;
            if (n == 32 || a == 0) continue;
        }
        const int32_t here = __shfl_sync(kFull, v, n);
        if (here < 0 || (here & kTbDead)) return;
        const int32_t kind = (here & 3) == kTbE ? 1 : 2;  // a gap: down the rows, or along this row
        if (p.last != kind) ++p.gap_opens;
        p.last = kind;
        for (bool on = true; on;) {
            ++p.gaps;
            if (kind == 1) {
                --a;
                const int32_t w = a > 0 ? byte_at(a, b) : 0;
                if (w < 0) return;
                on = (w & kTbEExt) != 0;
            } else {
                --b;
                const int32_t w = b >= 0 ? byte_at(a, b) : -1;
                if (w < 0) return;
                on = (w & kTbFExt) != 0;
            }
        }
    }
    if (b > 0) {  // along row 0
        if (p.last != 2) ++p.gap_opens;
        p.last = 2;
        p.gaps += b;
    }
    p.status = 0;
}

// Sides whose bands are expected to outgrow the registers (traceback_in_window)
// have a kernel without them: it needs fewer and runs more warps. 2,300 alignments
// of 450 residues at X-drop 105 / 215: 3.02 / 5.08 ms as the other form's way out,
// 2.36 / 4.11 so (2.40 / 4.35 with both sides on one warp).
template <bool WINDOW>
__global__ void
__launch_bounds__(kTracebackWarpsPerBlock * 32, WINDOW ? kTracebackBlocksPerSm : kTracebackRowsBlocksPerSm)
traceback_kernel(const TracebackArgs a) {
    __shared__ int32_t mat[kAlphabet * kAlphabet];
    for (int i = threadIdx.x; i < kAlphabet * kAlphabet; i += blockDim.x) mat[i] = g_blosum_tb[i];
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const unsigned long long gwarp = (static_cast<unsigned long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    int32_t *Hb = a.dp + gwarp * 2ull * a.dp_stride;
    int32_t *Eb = Hb + a.dp_stride;
    DirRows d;
    d.dir = a.dirs + gwarp * a.dir_cap;
    d.rows = a.rows + gwarp * 3ull * a.row_cap;
    d.cap = a.dir_cap;
    d.row_cap = a.row_cap;
    for (;;) {
        unsigned long long t = 0;
        if (lane == 0) t = atomicAdd(a.cursor, 1ull);
        t = __shfl_sync(kFull, t, 0);
        if (t >= 2ull * a.n_items) break;
        const bool is_left = (t & 1ull) == 0;
        const unsigned long long ti = t >> 1;
        const TbItem it = a.items[ti];
        const uint64_t o0 = a.off[it.subject];
        const uint8_t *sub = a.res + o0;
        const int32_t slen = static_cast<int32_t>(a.off[it.subject + 1] - o0);
        const int32_t q_off = it.q_off, s_off = it.s_off;
        const uint8_t *qres = a.batch_q ? a.batch_q[it.query] : a.q;
        const int32_t qlen = a.batch_q ? a.batch_qlen[it.query] : a.qlen;
        // row and column letter k at Q[dir * k] and S[dir * k]
        const int32_t dir = is_left ? -1 : 1;
        const uint8_t *Q = qres + q_off + (is_left ? 1 : 0), *S = sub + s_off + (is_left ? 1 : 0);
        const int32_t M = is_left ? q_off + 1 : qlen - q_off - 1, N = is_left ? s_off + 1 : slen - s_off - 1;
        d.overflow = false;
        TbPart p{};
        p.last = -1;
        if (WINDOW && dp_window_exact(M, a.gap_open, a.gap_extend, a.xdrop) &&
            xdrop_dp_window_dirs(Q, S, dir, M, N, a.gap_open, a.gap_extend, a.xdrop, mat, d, p)) {
            if (!d.overflow) walk_window(d, Q, S, dir, mat, p);
        } else {
            __syncwarp();
            int32_t rows;
            Walk w{0, 0, 0, 0, 0, -1, true};
            if (is_left) {
                p.score = xdrop_dp_dirs<true>(qres, sub, M, N, a.gap_open, a.gap_extend, a.xdrop, mat, Hb, Eb, &p.a,
                                              &p.b, d, &rows, &p.cells);
                if (!d.overflow && lane == 0) w = walk_back<true>(d, rows, qres, sub, M, N, p.a, p.b, mat);
            } else {
                p.score = xdrop_dp_dirs<false>(Q, S, M, N, a.gap_open, a.gap_extend, a.xdrop, mat, Hb, Eb, &p.a, &p.b,
                                               d, &rows, &p.cells);
                if (!d.overflow && lane == 0) w = walk_back<false>(d, rows, Q, S, M, N, p.a, p.b, mat);
            }
            p.pairs = w.pairs;
            p.identities = w.identities;
            p.positives = w.positives;
            p.gaps = w.gaps;
            p.gap_opens = w.gap_opens;
            p.last = w.last_move;
            p.status = w.ok ? 0 : 2;
        }
        if (d.overflow) p.status = 1;
        if (lane == 0) {
            a.part[t] = p;
            __threadfence();  // the side before the count
            if (atomicAdd(a.done + ti, 1u) == 1u) {  // the item's other side is done too
                __threadfence();
                const volatile int32_t *other = reinterpret_cast<const volatile int32_t *>(a.part + (t ^ 1ull));
                TbPart o2;
                for (int i = 0; i < static_cast<int>(sizeof(TbPart) / 4); ++i) reinterpret_cast<int32_t *>(&o2)[i] = other[i];
                const TbPart &l = is_left ? p : o2, &r = is_left ? o2 : p;
                TbOut o{};
                o.score = l.score + r.score;
                o.q_start = q_off + 1 - l.a;
                o.q_end = q_off + r.a + 1;
                o.s_start = s_off + 1 - l.b;
                o.s_end = s_off + r.b + 1;
                o.identities = l.identities + r.identities;
                o.positives = l.positives + r.positives;
                o.gaps = l.gaps + r.gaps;
                o.length = l.pairs + r.pairs + o.gaps;
                o.mismatches = l.pairs + r.pairs - o.identities;
                // a gap across the start point is one
                o.gap_opens = l.gap_opens + r.gap_opens - ((l.last > 0 && l.last == r.last) ? 1 : 0);
                o.status = l.status == 1 || r.status == 1 ? 1 : max(l.status, r.status);
                o.cells = l.cells + r.cells;
                a.out[ti] = o;
            }
        }
        __syncwarp();
    }
}

}  // namespace

cudaError_t launch_traceback(const TracebackArgs &a, bool window, int n_blocks, cudaStream_t st) {
    auto kernel = window ? traceback_kernel<true> : traceback_kernel<false>;
    kernel<<<n_blocks, kTracebackWarpsPerBlock * 32, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace blaze
