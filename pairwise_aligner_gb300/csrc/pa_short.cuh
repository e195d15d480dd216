// pa_short.cuh -- the short-pair DP kernel, and the strip of rows that it and the long-pair kernel
// (pa_long.cuh) share.
//
// The same recurrence, borders, trackers and wavefront as dp_kernel (pa_dp.cuh): a group of
// G lanes holds two pairs in the halves of s16x2 registers or one pair in s32 lanes, thread t
// holds R rows of sequence2, and the group sweeps sequence1 as an anti-diagonal wavefront.
// Scores (Scoring): the 4-byte tables of streamed DNA bases, raw byte comparison, or an int8
// profile of the held rows under a substitution matrix.
// The reference's hot loop it replaces is compute_block / compute_cell
// (dp_algorithm_template/dp_algorithm_template_base.hpp:82-129,
// affine/affine_dp_algorithm.hpp:133-156).  What differs is how little each column step
// costs besides the recurrence:
//  * every streamed column has one 16-byte slot {symbol of lane A, of lane B, top H, top
//    vertical gap} (a DNA symbol is its score table).  The group writes the slots of its unit once (symbols from the
//    sequence1 bytes, the top border of the first pass); the last thread writes the
//    pass's bottom row back into the .h/.e halves for the next pass;
//  * thread 0 reads one slot per column with a single vector load, one column ahead, and
//    the symbols travel down the group with the H and gap values by shuffle, so no
//    other thread loads anything per column (thread 0 selects the slot's values);
//  * the rows are written so that the diagonal term of row k + 1 is formed before row k's
//    new H replaces the old one (no register copies between column steps);
//  * the unit's description, the per-thread candidates and the column of the last local
//    improvement live in shared memory, so the registers hold the R rows (R = 32 halves
//    the column steps of R = 16).
#pragma once
#include "pa_dp.cuh"

namespace pa {

// How a cell is scored.
enum Scoring : int {
    SC_TABLE = 0,      // unitary scores of A/C/G/T rows: a byte of the streamed base's table
    SC_BYTES = 1,      // unitary scores of any bytes: equality (s32 lanes)
    SC_PROFILE = 2     // substitution matrix: a byte of the row's profile (s32 lanes)
};

// The unit a group works on: one pair, two in s16x2 lanes (lane B may be absent).
struct ShortUnit {
    uint32_t id[2];
    uint64_t toff[2];
    int32_t m[2], n[2];
    int32_t ms, nh, passes, has_b;
    Slot *slot;                    // slots 1..ms of the unit (slot 0 unused)
};

// Stored values of a lane type: true value + Kt (global modes: of H - shift * column), clamped
// at clampt; a global s16 result at or below floor_true may have met the clamp.
template <class V, int MODE>
struct StripConst {
    static constexpr bool S16 = V::LANES == 2;
    static constexpr int32_t Kt = !S16 ? 0 : MODE == M_LOCAL ? 2048 : 32767 - 512;
    static constexpr int32_t clampt = S16 ? 2048 : MODE == M_LOCAL ? 0 : INT32_MIN;
    static constexpr int32_t below = (S16 ? clampt : kNeg32) - 1;     // less than any stored value
    static constexpr int32_t floor_true = !S16 ? INT32_MIN : MODE == M_LOCAL ? 0 : 2048 - Kt;
};

// Per-thread shared-memory state of a block of NT threads: result candidates (score, end1, end2)
// of every lane and, in local mode, the column of each lane's last improvement in the pass.
template <class V, int NT = kBlock>
struct StripShared {
    int32_t (*c)[3][NT];           // [lane][field][thread]
    int32_t (*bi)[NT];             // [lane][thread]; free last rows: the column, then the value
    __device__ __forceinline__ int32_t &s(int l) { return c[l][0][threadIdx.x]; }
    __device__ __forceinline__ int32_t &i(int l) { return c[l][1][threadIdx.x]; }
    __device__ __forceinline__ int32_t &j(int l) { return c[l][2][threadIdx.x]; }
    __device__ __forceinline__ void offer(int l, int32_t xs, int32_t xi, int32_t xj)
    {
        if (better(xs, xi, xj, s(l), i(l), j(l))) { s(l) = xs; i(l) = xi; j(l) = xj; }
    }
};

// A held row's score selector: s16x2 lanes permute the tables of both streamed bases to it
// (V::selector); s32 lanes hold a one-hot byte, so that one dot product adds the row's score.
// A padded row (code < 0) scores 0 or -1.
template <class V>
__device__ __forceinline__ uint32_t strip_selector(int ca, int cb)
{
    if (V::LANES == 2) return V::selector(ca, cb);
    return ca < 0 ? 0u : 1u << (8 * ca);
}

// One column step of a strip of RA rows: H and the gap to the next column (Fr) of the rows, the
// vertical gap Ed running down the strip; prevH is H(i - 1, row above the strip).  diagonal(d, k)
// is d + the score of row k, in s16x2 lanes already the maximum with Fr[k].  Per row and lane
// register (whole-chip microbenchmark of the loop alone, 24 rows): s16x2 PRMT, VIADDMNMX
// (diagonal + score against Fr), VIMNMX3, two VIADDMNMX (both gaps) and a subtraction or two,
// 8.1 T cells/s with the column shift (7.4 with the gaps as a subtraction and a maximum); s32
// IDP4A, VIMNMX3, two VIADDMNMX, 4.8 (4.1 with PRMT, VIADDMNMX and subtract-and-maximum), as
// IDP4A leaves the ALU pipe free.
template <class V, int MODE, int RA, class D>
__device__ __forceinline__ void strip_column(uint32_t *H, uint32_t *Fr, uint32_t prevH, uint32_t &Ed,
                                             const StripGaps &g, D diagonal)
{
    constexpr bool SHIFTED = MODE != M_LOCAL;      // local mode has no column shift (P.shift == 0)
    const uint32_t CLAMP = V::splat(StripConst<V, MODE>::clampt);
    auto gap = [](uint32_t x, uint32_t ext_neg, uint32_t open) -> uint32_t {
        if (V::LANES == 2) return __viaddmax_s16x2(x, ext_neg, open);
        return (uint32_t)__viaddmax_s32((int)x, (int)ext_neg, (int)open);
    };
    uint32_t tt = diagonal(prevH, 0);
#pragma unroll
    for (int k = 0; k < RA; ++k) {
        // the next row's diagonal term uses this row's H before it is replaced
        const uint32_t tn = k + 1 < RA ? diagonal(H[k], k + 1) : 0u;
        uint32_t h;
        if (V::LANES == 2) h = V::hmax(tt, Ed, CLAMP);
        else if (MODE == M_LOCAL) h = (uint32_t)__vimax3_s32_relu((int)tt, (int)Fr[k], (int)Ed);
        else h = (uint32_t)__vimax3_s32((int)tt, (int)Fr[k], (int)Ed);
        H[k] = h;
        const uint32_t hoe = h - g.goe;
        Fr[k] = SHIFTED ? gap(Fr[k], g.ext_h_neg, h - g.goe_h) : gap(Fr[k], g.ext_neg, hoe);
        Ed = gap(Ed, g.ext_neg, hoe);
        tt = tn;
    }
}

// The diagonal term of a row under SC_TABLE.
template <class V>
__device__ __forceinline__ uint32_t table_diagonal(uint32_t d, uint32_t ta, uint32_t tb, uint32_t sel, uint32_t fr)
{
    if (V::LANES == 2) return __viaddmax_s16x2(d, prmt(ta, tb, sel), fr);
    return (uint32_t)__dp4a((int)ta, (int)sel, (int)d);
}

// Local mode, after a column: the best H so far of the thread's rows; on a strict improvement of
// a lane the column's number and its H values go to shared memory.
template <class V, int R, int RA, int NT>
__device__ __forceinline__ void strip_track(const uint32_t *H, uint32_t &best, int32_t i, uint4 *snap,
                                            StripShared<V, NT> &sh)
{
    const uint32_t cm = tree_max<V, RA>(H);
    const uint32_t nb = V::max2(best, cm);
    const uint32_t x = nb ^ best;
    best = nb;
    if (x != 0u) {
#pragma unroll
        for (int l = 0; l < V::LANES; ++l) {
            if (V::improved(x, l)) {
                sh.bi[l][threadIdx.x] = i;
#pragma unroll
                for (int v = 0; v < RA / 4; ++v)
                    snap[(l * (R / 4) + v) * NT] = make_uint4(H[4 * v], H[4 * v + 1], H[4 * v + 2], H[4 * v + 3]);
            }
        }
    }
}

// ... and after the pass: the first row of that column that holds the best value.
template <class V, int R, int RA, int NT>
__device__ __forceinline__ void strip_track_end(uint32_t best, int32_t j0, const uint4 *snap, StripShared<V, NT> &sh)
{
    constexpr int32_t Kt = StripConst<V, M_LOCAL>::Kt;
#pragma unroll
    for (int l = 0; l < V::LANES; ++l) {
        const int32_t b = V::get(best, l);
        if (b > Kt) {                             // improved in this pass: snapshot and column are set
            int32_t kk = 0;
            for (int v = RA / 4 - 1; v >= 0; --v) {
                const uint4 q = snap[(l * (R / 4) + v) * NT];
                if (V::get(q.w, l) == b) kk = 4 * v + 3;
                if (V::get(q.z, l) == b) kk = 4 * v + 2;
                if (V::get(q.y, l) == b) kk = 4 * v + 1;
                if (V::get(q.x, l) == b) kk = 4 * v;
            }
            sh.offer(l, b - Kt, sh.bi[l][threadIdx.x], j0 + kk + 1);
        }
    }
}

// Global modes, after column i: the end cell of every lane whose last row this thread holds and whose
// last column this is.  own_row(l) is the strip index of lane l's last row, or -1; the row's H is read
// back from shared memory, where the thread puts its column first (a chain of selects over the rows
// cost 60 ALU operations a column; the stores go to the idle LSU pipe).
template <class V, int MODE, int RA, int NT, class U, class O>
__device__ __forceinline__ void strip_ends(const DpParams &P, const U &u, const uint32_t *H, int32_t i, bool any_own,
                                           uint4 *snap, StripShared<V, NT> &sh, O own_row)
{
    if (any_own) {
#pragma unroll
        for (int v = 0; v < RA / 4; ++v)
            snap[v * NT] = make_uint4(H[4 * v], H[4 * v + 1], H[4 * v + 2], H[4 * v + 3]);
    }
#pragma unroll
    for (int l = 0; l < V::LANES; ++l) {
        if (l == 1 && !u.has_b) continue;
        const int32_t base = P.shift * i - StripConst<V, MODE>::Kt, ml = u.m[l], r = own_row(l);
        if (r >= 0 && i == ml) {
            const uint32_t *q = reinterpret_cast<const uint32_t *>(snap + (r >> 2) * NT);
            sh.offer(l, V::get(q[r & 3], l) + base, i, u.n[l]);
        }
    }
}

// ... the column at which the shorter lane ends, if its end rule needs it and it is not the last (else 0:
// no column), and its store.
template <class V, int MODE, class U>
__device__ __forceinline__ int32_t strip_cut_at(const DpParams &P, const U &u)
{
    if (V::LANES == 1 || MODE != M_GLOBAL_FREE || !P.last_row_free || !u.has_b || u.m[0] == u.m[1]) return 0;
    return min(u.m[0], u.m[1]);
}

template <int RA, int NT>
__device__ __forceinline__ void strip_cut(const uint32_t *H, uint4 *cut)
{
#pragma unroll
    for (int v = 0; v < RA / 4; ++v) cut[v * NT] = make_uint4(H[4 * v], H[4 * v + 1], H[4 * v + 2], H[4 * v + 3]);
}

// Free end of sequence1's last column: its first best row, offered once after the pass.  The longer
// lane's column is the last that the thread computed, so H still holds it; the shorter lane's was put
// into `cut` (16-byte words NT apart) when it was computed.  An offer per row in the column's step took
// 3,176 us for 60,000 pairs of 64-512 rows with all ends free, the scan in that step 1,710 (and 3-12 %
// of calls without this end rule, whose loop carried it), 1,323 here.
template <class V, int MODE, int RA, int NT, class U>
__device__ __forceinline__ void strip_column_offer(const DpParams &P, const U &u, const uint32_t *H, int32_t j0,
                                                   const uint4 *cut, StripShared<V, NT> &sh)
{
#pragma unroll
    for (int l = 0; l < V::LANES; ++l) {
        if (l == 1 && !u.has_b) continue;
        const int32_t ml = u.m[l], rows = u.n[l] - j0;
        const bool held = V::LANES == 1 || ml == u.ms;
        int32_t top = INT32_MIN, at = -1;
#pragma unroll
        for (int k = 0; k < RA; ++k) {
            const uint32_t h = held ? H[k] : reinterpret_cast<const uint32_t *>(cut + (k >> 2) * NT)[k & 3];
            const int32_t x = V::get(h, l);
            if (k < rows && (x > top || at < 0)) { top = x; at = k; }
        }
        if (at >= 0) sh.offer(l, top + P.shift * ml - StripConst<V, MODE>::Kt, ml, j0 + at + 1);
    }
}

// Free end of sequence2's last row, after every column of a thread that holds such a row (strip
// indices r0, r1 of the lanes): on a strict improvement the column and the stored value go to
// shared memory.  `seen` is the best so far as a stored value of the current column (H - shift *
// column, so one add-max moves it on), kept one below the clamp: a clamped value then counts
// exactly as its comparison in true scores would.  Comparing the candidates in shared memory on
// every column took 30 % of the kernel's instructions: 65,537 reads of 100-250 bp in windows 1,334
// -> 1,098 us (comparing only on an improvement: 1,514, as a read's first columns all improve).
template <class V, int MODE, int RA, int NT, class U>
__device__ __forceinline__ void strip_end_track(const U &u, const uint32_t *H, uint32_t &seen, uint32_t shift_neg,
                                                int32_t i, int32_t r0, int32_t r1, uint4 *snap, StripShared<V, NT> &sh)
{
    constexpr int NL = V::LANES;
#pragma unroll
    for (int v = 0; v < RA / 4; ++v) snap[v * NT] = make_uint4(H[4 * v], H[4 * v + 1], H[4 * v + 2], H[4 * v + 3]);
    const uint32_t *row = reinterpret_cast<const uint32_t *>(snap);
    uint32_t x = row[(r0 >> 2) * (4 * NT) + (r0 & 3)], moved;
    if (NL == 2) {
        x = prmt(x, row[(r1 >> 2) * (4 * NT) + (r1 & 3)], 0x7610);
        moved = __viaddmax_s16x2(seen, shift_neg, V::splat(StripConst<V, MODE>::below));
    } else {
        moved = (uint32_t)__viaddmax_s32((int)seen, (int)shift_neg, StripConst<V, MODE>::below);
    }
    seen = V::max2(moved, x);
#pragma unroll
    for (int l = 0; l < NL; ++l) {
        if (V::improved(seen ^ moved, l) && i <= u.m[l]) {
            sh.bi[l][threadIdx.x] = i;
            sh.bi[NL + l][threadIdx.x] = (int32_t)x;
        }
    }
}

// ... and after the pass: its candidates.
template <class V, int MODE, int NT, class U>
__device__ __forceinline__ void strip_end_offer(const DpParams &P, const U &u, const int32_t *own,
                                                StripShared<V, NT> &sh)
{
#pragma unroll
    for (int l = 0; l < V::LANES; ++l) {
        const int32_t i = sh.bi[l][threadIdx.x];
        if (own[l] >= 0 && i > 0)
            sh.offer(l, V::get((uint32_t)sh.bi[V::LANES + l][threadIdx.x], l) + P.shift * i - StripConst<V, MODE>::Kt,
                     i, u.n[l]);
    }
}

// Results of a finished unit from its candidates (one thread): the free-end borders, the s16
// exactness check (a result at the floor goes to the s32 redo list), the failed waits.
template <class V, int MODE>
__device__ __forceinline__ void strip_emit(const DpLaunch &L, const DpParams &P, const uint32_t *id, const int32_t *m,
                                           const int32_t *n, bool has_b, int32_t *cs, int32_t *ci, int32_t *cj,
                                           bool failed)
{
    using KC = StripConst<V, MODE>;
#pragma unroll
    for (int l = 0; l < V::LANES; ++l) {
        if (l == 1 && !has_b) continue;
        pa_result r;
        if (failed) {
            // a boundary cell was used before it was there: the score is not valid
            r.score = INT32_MIN;
            r.end1 = r.end2 = 0;
            r.width = V::WIDTH;
            r.flags = PA_RESULT_ERROR;
            r.band_rounds = 0;
            L.out[id[l]] = r;
            continue;
        }
        if (MODE == M_GLOBAL_FREE) {
            if (P.last_column_free) {            // H(0, n)
                const int32_t x = border(P, P.first_row_free, n[l]);
                if (better(x, 0, n[l], cs[l], ci[l], cj[l])) { cs[l] = x; ci[l] = 0; cj[l] = n[l]; }
            }
            if (P.last_row_free) {               // H(m, 0)
                const int32_t x = border(P, P.first_column_free, m[l]);
                if (better(x, m[l], 0, cs[l], ci[l], cj[l])) { cs[l] = x; ci[l] = m[l]; cj[l] = 0; }
            }
        }
        if (V::LANES == 2 && MODE != M_LOCAL &&
            (int64_t)cs[l] - (int64_t)P.shift * ci[l] <= (int64_t)KC::floor_true) {
            // a clamp may have reached this result: recompute it in s32
            const uint32_t slot = atomicAdd(L.rerun_count, 1u);
            L.rerun_list[slot] = id[l];
            continue;
        }
        r.score = cs[l];
        r.end1 = ci[l];
        r.end2 = cj[l];
        r.width = V::WIDTH;
        r.flags = V::LANES == 1 && L.rerun ? PA_RESULT_RERUN : 0;
        r.band_rounds = 0;
        if (MODE == M_LOCAL && cs[l] <= 0) { r.end1 = 0; r.end2 = 0; }
        L.out[id[l]] = r;
    }
}

// The int8 profile of a thread's rows (SC_PROFILE): for each symbol rank r one uint4 at
// prof[r * NT], its byte k the score of r against row k (minus the column shift).  A column then
// costs one 16-byte shared-memory load for all rows, without bank conflicts whatever the lanes'
// symbols, and IDP4A adds a row's byte to the diagonal; a matrix lookup per cell in global memory
// ran at 0.58 T cells/s.  `mat` holds the scores as bytes, 32 ranks per held symbol, symbol 32
// the padding rows.
template <int RA, int NT>
__device__ __forceinline__ void build_profile(uint4 *prof, const uint32_t (*mat)[8], const uint32_t *sym, int dim)
{
    for (int q = 0; 4 * q < dim; ++q) {
        uint32_t x[4][4];                         // [rank 4q + r][rows 4v .. 4v + 3]
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) w[k] = 4 * v + k < RA ? mat[sym[4 * v + k < RA ? 4 * v + k : 0]][q] : 0u;
            const uint32_t a = prmt(w[0], w[1], 0x5140), b = prmt(w[0], w[1], 0x7362);
            const uint32_t c = prmt(w[2], w[3], 0x5140), d = prmt(w[2], w[3], 0x7362);
            x[0][v] = prmt(a, c, 0x5410);
            x[1][v] = prmt(a, c, 0x7632);
            x[2][v] = prmt(b, d, 0x5410);
            x[3][v] = prmt(b, d, 0x7632);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) prof[(4 * q + r) * NT] = make_uint4(x[r][0], x[r][1], x[r][2], x[r][3]);
    }
}

// One pass p of the unit: rows p*G*R + t*RA + 1 .. + RA (1-based) on thread t.
template <class V, int SC, int MODE, int G, int R, int RA, int NT>
__device__ __forceinline__ void short_pass(const DpLaunch &L, const DpParams &P, const ShortUnit &u, int p, int t,
                                           int32_t ms_min, int32_t ms_max, uint4 *snap, uint4 *cut,
                                           StripShared<V, NT> sh, uint4 *prof, const uint32_t (*mat)[8])
{
    using KC = StripConst<V, MODE>;
    constexpr int NL = V::LANES;
    const int32_t rows_full = G * R;
    const int32_t j0 = p * rows_full + t * RA;
    const StripGaps gaps = NL == 2 ? L.gaps16 : L.gaps32;
    auto stored = [&](int32_t true_value) { return V::splat(max(true_value + KC::Kt, KC::clampt)); };

    uint32_t H[RA], Fr[RA], Sel[RA];
#pragma unroll
    for (int k = 0; k < RA; ++k) {
        const int32_t j = j0 + k;                 // 0-based row of sequence2
        if (SC == SC_TABLE) {
            const int ca = j < u.n[0] ? (int)dna_code(L.seq2[u.toff[0] + j]) : -1;
            const int cb = NL == 2 ? (j < u.n[1] ? (int)dna_code(L.seq2[u.toff[1] + j]) : -1) : ca;
            Sel[k] = strip_selector<V>(ca, cb);
        } else {
            const uint32_t b = j < u.n[0] ? (uint32_t)L.seq2[u.toff[0] + j] : 0x100u;
            Sel[k] = SC == SC_BYTES ? b : b < 0x100u ? (uint32_t)__ldg(L.rank_map + b) : 32u;
        }
        H[k] = stored(border(P, P.first_row_free, (int64_t)j + 1));
        Fr[k] = H[k] - gaps.goe_h;
    }
    if (SC == SC_PROFILE) build_profile<RA, NT>(prof, mat, Sel, L.mdim);
    uint32_t prevH = stored(border(P, P.first_row_free, j0));
    const bool writer = t == G - 1 && p + 1 < u.passes;
    const bool t0 = t == 0;
    const int32_t ms = p < u.passes ? u.ms : 0;   // a group past its last pass only goes along
    Slot *const slot = u.slot;
    const uint32_t hit = (uint32_t)(P.match - P.shift), miss = (uint32_t)(P.mismatch - P.shift);

    // the registers a thread hands on: bottom H and gap of its strip and the column's symbols
    uint32_t sH = 0, sE = 0, sA = 0, sB = 0;
    uint4 nx = make_uint4(0u, 0u, 0u, 0u);        // thread 0: the slot of its next column
    if (t0 && ms > 0) nx = *reinterpret_cast<const uint4 *>(slot + 1);
    uint32_t best = V::splat(KC::Kt);
    // global modes: whether a lane's last row is this thread's, and the first column a lane ends at
    int32_t own[NL];
    bool any_own = false;
    int32_t mmin = ms;
#pragma unroll
    for (int l = 0; l < NL; ++l) {
        const int32_t r = (u.n[l] - 1) - j0;
        own[l] = MODE != M_LOCAL && r >= 0 && r < RA && (u.n[l] - 1) / rows_full == p ? r : -1;
        any_own |= own[l] >= 0;
        mmin = min(mmin, u.m[l]);
    }

    // the end rule of the last row (strip_end_track)
    const bool row_end = MODE == M_GLOBAL_FREE && P.last_column_free && any_own;
    uint32_t seen = V::splat(KC::below);
    const uint32_t shift_neg = V::splat(-P.shift);
    const int32_t r0 = max(own[0], 0), r1 = max(own[NL - 1], 0);
    if (row_end) {
#pragma unroll
        for (int l = 0; l < NL; ++l) sh.bi[l][threadIdx.x] = 0;
    }

    const int32_t cut_at = strip_cut_at<V, MODE>(P, u);
    // step s of the pass: thread t computes column i = s - t + 1 when 1 <= i <= ms
    auto step = [&](int32_t s, bool active) {
        const int32_t i = s - t + 1;
        const uint32_t xH = __shfl_up_sync(0xffffffffu, sH, 1, G);
        const uint32_t xE = __shfl_up_sync(0xffffffffu, sE, 1, G);
        const uint32_t xA = __shfl_up_sync(0xffffffffu, sA, 1, G);
        const uint32_t xB = NL == 2 ? __shfl_up_sync(0xffffffffu, sB, 1, G) : 0u;
        if (active) {
            const uint32_t upH = t0 ? nx.z : xH;
            uint32_t Ed = t0 ? nx.w : xE;
            const uint32_t ta = t0 ? nx.x : xA;
            const uint32_t tb = NL == 2 ? (t0 ? nx.y : xB) : ta;
            if (t0 && i < ms) nx = *reinterpret_cast<const uint4 *>(slot + i + 1);
            if (SC == SC_TABLE) {
                strip_column<V, MODE, RA>(H, Fr, prevH, Ed, gaps, [&](uint32_t d, int k) {
                    return table_diagonal<V>(d, ta, tb, Sel[k], Fr[k]);
                });
            } else if (SC == SC_BYTES) {
                strip_column<V, MODE, RA>(H, Fr, prevH, Ed, gaps,
                                          [&](uint32_t d, int k) { return d + (Sel[k] == ta ? hit : miss); });
            } else {
                const uint4 q = prof[ta];
                const uint32_t w[4] = {q.x, q.y, q.z, q.w};
                strip_column<V, MODE, RA>(H, Fr, prevH, Ed, gaps, [&](uint32_t d, int k) {
                    return (uint32_t)__dp4a((int)w[k >> 2], 1 << (8 * (k & 3)), (int)d);
                });
            }
            prevH = upH;
            sH = H[RA - 1];
            sE = Ed;
            sA = ta;
            sB = tb;
            if (writer) *reinterpret_cast<uint2 *>(&slot[i].h) = make_uint2(sH, sE);
            if (MODE == M_LOCAL)
                strip_track<V, R, RA>(H, best, i, snap, sh);
            else {
                if (row_end) strip_end_track<V, MODE, RA, NT>(u, H, seen, shift_neg, i, r0, r1, snap, sh);
                if (i >= mmin) {
                    strip_ends<V, MODE, RA>(P, u, H, i, any_own, snap, sh, [&](int l) { return own[l]; });
                    if (MODE == M_GLOBAL_FREE && NL == 2 && i == cut_at) strip_cut<RA, NT>(H, cut);
                }
            }
        }
    };
    // The groups of a warp keep step with one another: loops of their own would let them drift apart
    // and run one after the other (4 lanes per group: 16.5 ms for 262,144 local pairs).  s16x2
    // lanes: one loop for fill, steady state and drain, so that the 32-row bodies take less of the
    // instruction cache (local 4,694 -> 4,648 us); s32 lanes: a loop of their own for the steps
    // with every thread active (proteins 1,598 -> 1,525 us).
    int32_t s = 0;
    if (NL == 1) {
        for (; s < min(G, ms_max + G - 1); ++s) step(s, (uint32_t)(s - t) < (uint32_t)ms);
        for (; s < ms_min; ++s) step(s, true);
    }
    for (; s < ms_max + G - 1; ++s) step(s, (uint32_t)(s - t) < (uint32_t)ms);
    if (MODE == M_LOCAL) strip_track_end<V, R, RA>(best, j0, snap, sh);
    if (row_end) strip_end_offer<V, MODE, NT>(P, u, own, sh);
    if (MODE == M_GLOBAL_FREE && P.last_row_free && ms > 0) strip_column_offer<V, MODE, RA, NT>(P, u, H, j0, cut, sh);
}

// With fewer work items than warps, only the first warps of every block take any: otherwise the
// warps of the blocks that start first would take them all and leave the other SMs empty.  1,024
// pairs of 150 bp (512 units on 2,432 warps): 136 -> 112 us a call.
__device__ __forceinline__ bool strip_warp_takes_part(uint32_t items)
{
    return (threadIdx.x >> 5) < (items + gridDim.x - 1) / gridDim.x;
}

// One warp unit of 32/G groups (x two pairs in s16x2 lanes): its pairs are order[first] .. below
// position `end`, a group's first pair at first + g * lanes.
template <class V, int SC, int MODE, int G, int R, int NT>
__device__ __forceinline__ void short_unit(const DpLaunch &L, const DpParams &P, const uint32_t *order, uint32_t first,
                                           uint32_t end, ShortUnit *s_unit, uint4 *snap, uint4 *cut,
                                           StripShared<V, NT> sh, uint4 *prof, const uint32_t (*mat)[8])
{
    constexpr int NL = V::LANES;
    const int lane = threadIdx.x & 31;
    const int t = lane & (G - 1);
    const int g = lane / G;
    ShortUnit &su = s_unit[threadIdx.x / G];
    first += (uint32_t)g * NL;
    const bool idle = first >= end;                  // a group without a pair, in a list's last unit
    const uint32_t match4 = (uint8_t)(P.match - P.shift) * 0x01010101u;
    const uint32_t mis4 = (uint8_t)(P.mismatch - P.shift) * 0x01010101u;
    auto symbol = [&](uint32_t b) -> uint32_t {
        return SC == SC_TABLE ? score_table(b, match4, mis4) : SC == SC_BYTES ? b : (uint32_t)__ldg(L.rank_map + b) * NT;
    };
    if (t == 0) {
        ShortUnit u{};
        if (!idle) {
            u.id[0] = order[first];
            u.has_b = NL == 2 && first + 1 < end;
            u.id[1] = u.has_b ? order[first + 1] : u.id[0];
            for (int l = 0; l < 2; ++l) {
                const uint64_t q0 = L.off1[u.id[l]];
                u.m[l] = (int32_t)(L.off1[u.id[l] + 1] - q0);
                u.toff[l] = L.off2[u.id[l]];
                u.n[l] = (int32_t)(L.off2[u.id[l] + 1] - u.toff[l]);
            }
            u.ms = max(u.m[0], u.m[1]);
            u.nh = max(u.n[0], u.n[1]);
            u.passes = (u.nh + G * R - 1) / (G * R);
            const uint32_t owner = u.m[1] > u.m[0] ? u.id[1] : u.id[0];
            u.slot = L.slots + (L.off1[owner] + owner);   // slots 0..m(owner) = 0..ms
        }
        su = u;
    }
    for (int l = 0; l < NL; ++l) {
        sh.s(l) = MODE == M_LOCAL ? 0 : INT32_MIN;
        sh.i(l) = 0;
        sh.j(l) = 0;
    }
    __syncwarp();
    // the unit's slots: the lanes' symbols (a padding table past a lane's end) and the top
    // border of the first pass, H(i, 0) - shift * i
    if (!idle) {
        using KC = StripConst<V, MODE>;
        const uint64_t qa = L.off1[su.id[0]], qb = L.off1[su.id[1]];
        const int32_t ma = su.m[0], mb = su.m[1];
        const uint32_t goe = NL == 2 ? L.gaps16.goe : L.gaps32.goe;
        for (int32_t i = 1 + t; i <= su.ms; i += G) {
            const uint32_t a = i <= ma ? symbol(L.seq1[qa + i - 1]) : 0x80808080u;
            const uint32_t b = NL == 2 ? (i <= mb ? symbol(L.seq1[qb + i - 1]) : 0x80808080u) : 0u;
            const int64_t top = (int64_t)border(P, P.first_column_free, i) - (int64_t)P.shift * i + KC::Kt;
            const uint32_t h = V::splat((int32_t)max(top, (int64_t)KC::clampt));
            *reinterpret_cast<uint4 *>(su.slot + i) = make_uint4(a, b, h, h - goe);
        }
    }
    __syncwarp();
    const int32_t passes = __reduce_max_sync(0xffffffffu, su.passes);
    for (int p = 0; p < passes; ++p) {
        const ShortUnit u = su;
        // rows per thread and columns of the pass, for all groups of the warp
        const int32_t rem = __reduce_max_sync(0xffffffffu, u.nh - p * G * R);
        const int32_t rpt = rem >= G * R ? R : ((rem + G * kChunk - 1) / (G * kChunk)) * kChunk;
        const int32_t ms = p < u.passes ? u.ms : 0;
        const int32_t ms_min = __reduce_min_sync(0xffffffffu, ms), ms_max = __reduce_max_sync(0xffffffffu, ms);
#define PA_SHORT_PASS(RA) \
    short_pass<V, SC, MODE, G, R, (R >= RA ? RA : R), NT>(L, P, u, p, t, ms_min, ms_max, snap, cut, sh, prof, mat)
        switch (rpt / kChunk) {
        case 1: PA_SHORT_PASS(4); break;
        case 2: PA_SHORT_PASS(8); break;
        case 3: PA_SHORT_PASS(12); break;
        case 4: PA_SHORT_PASS(16); break;
        case 5: PA_SHORT_PASS(20); break;
        case 6: PA_SHORT_PASS(24); break;
        case 7: PA_SHORT_PASS(28); break;
        default: PA_SHORT_PASS(R); break;
        }
#undef PA_SHORT_PASS
        __syncwarp();
    }
    // reduce over the group, then thread 0 writes the results
    int32_t cs[NL], ci[NL], cj[NL];
#pragma unroll
    for (int l = 0; l < NL; ++l) {
        cs[l] = sh.s(l);
        ci[l] = sh.i(l);
        cj[l] = sh.j(l);
        for (int off = G >> 1; off >= 1; off >>= 1) {
            const int32_t os = __shfl_xor_sync(0xffffffffu, cs[l], off, G);
            const int32_t oi = __shfl_xor_sync(0xffffffffu, ci[l], off, G);
            const int32_t oj = __shfl_xor_sync(0xffffffffu, cj[l], off, G);
            if (better(os, oi, oj, cs[l], ci[l], cj[l])) { cs[l] = os; ci[l] = oi; cj[l] = oj; }
        }
    }
    if (t == 0 && !idle) {
        const ShortUnit u = su;
        strip_emit<V, MODE>(L, P, u.id, u.m, u.n, u.has_b != 0, cs, ci, cj, false);
    }
    __syncwarp();
}

// The short-pair kernel: a persistent grid whose warps take units of 32/G groups (x two pairs in
// s16x2 lanes) from the class's list, largest shapes first; R rows of sequence2 per thread, NT
// threads per block.  SC_PROFILE keeps the profiles in dynamic shared memory: blocks of 128
// threads pack it into an SM best (16 warps with up to 20 symbols, 12 with 24 to 32).
template <class V, int SC, int MODE, int G, int R, int NT>
__global__ void __launch_bounds__(NT, 512 / NT) dp_short(DpLaunch L, DpParams P)
{
    static_assert(R % kChunk == 0 && R <= 32, "R must be a multiple of the chunk");
    constexpr int NL = V::LANES;
    __shared__ uint4 snap_store[(MODE == M_LOCAL ? NL : 1) * (R / 4) * NT];
    __shared__ uint4 cut_store[MODE == M_GLOBAL_FREE && NL == 2 ? (R / 4) * NT : 1];
    __shared__ ShortUnit s_unit[NT / G];
    __shared__ int32_t s_cand[NL][3][NT];
    __shared__ int32_t s_bi[MODE == M_LOCAL ? NL : MODE == M_GLOBAL_FREE ? 2 * NL : 1][NT];
    __shared__ uint32_t s_mat[SC == SC_PROFILE ? 33 : 1][8];
    extern __shared__ uint4 s_prof[];
    uint4 *snap = snap_store + threadIdx.x;
    uint4 *cut = cut_store + (MODE == M_GLOBAL_FREE && NL == 2 ? threadIdx.x : 0);
    uint4 *prof = s_prof + threadIdx.x;
    StripShared<V, NT> sh{s_cand, s_bi};
    const uint32_t count = *L.count_ptr;
    constexpr uint32_t ppw = (uint32_t)(32 / G) * NL;    // pairs per warp unit
    const uint32_t n_units = (count + ppw - 1) / ppw;
    if (n_units == 0) return;
    if (SC == SC_PROFILE) {
        // the matrix as bytes (the host checked that they fit), transposed
        for (int x = threadIdx.x; x < 33 * 32; x += NT) {
            const int held = x >> 5, r = x & 31;
            const int32_t v = held < L.mdim && r < L.mdim ? __ldg(L.matrix + r * L.mdim + held) : P.spad;
            reinterpret_cast<int8_t *>(s_mat)[x] = (int8_t)(v - P.shift);
        }
        __syncthreads();
    }
    if (!strip_warp_takes_part(n_units)) return;
    const uint32_t *order = L.order + *L.begin_ptr;
    for (;;) {
        uint32_t uu = 0;
        if ((threadIdx.x & 31) == 0) uu = atomicAdd(L.unit_counter, 1u);
        uu = __shfl_sync(0xffffffffu, uu, 0);
        if (uu >= n_units) break;
        short_unit<V, SC, MODE, G, R, NT>(L, P, order, (n_units - 1 - uu) * ppw, count, s_unit, snap, cut, sh, prof, s_mat);
        __syncwarp();
    }
}

}  // namespace pa
