// pa_long.cuh -- the DP of long pairs: one queue of row passes for the whole GPU.
//
// Same recurrence, borders and trackers as the short-pair kernel (pa_short.cuh; the
// reference's compute_block / compute_cell, dp_algorithm_template/
// dp_algorithm_template_base.hpp:82-129, affine/affine_dp_algorithm.hpp:133-156).  A unit is
// two pairs in s16x2 lanes or one in s32 lanes; its matrix is cut into passes of 32 * rpt
// rows of sequence2 (long_rows), and one warp sweeps a whole pass as an anti-diagonal wavefront with rpt
// rows per thread.  The task queue lists the passes of all units, largest unit first and a
// unit's passes in order (k_long_plan), so every warp of the GPU takes the next pass of
// whatever unit is open: a pair is not tied to a block, and nothing idles until the queue is
// empty.  A pass follows the one above it, column by column, wherever that one runs.
//
// The boundary row.  Pass p - 1 hands its bottom row to pass p through one 16-byte cell per
// column, {H, vertical gap, tag}, written and read with single 128-bit relaxed accesses at
// GPU scope.  The tag names the launch and the pass, so a reader that finds it has the whole
// cell: no flag, no fence, no order between cells is needed.  The cells are the pair's column slots
// of the short-pair kernel (a memory of their own would add 16 bytes per base of sequence1 to every
// call that may hold a long pair); no slot's contents look like a tag (kTagMark).  The row is reused in
// place:
// pass p overwrites column i only after its own first thread read column i.  The reader
// fetches blocks of kStage columns, one block ahead (lane t the block's column t), and hands
// them to thread 0 through shared memory with the score tables; a cell that is not there yet
// is polled, at most spin_limit times.
// A task waits only for a task handed out before it, which some running warp holds, so every
// wait ends.  At the end of a pass the unit's best candidate goes to the next pass through a
// record released by a per-unit pass counter; the last pass writes the results.
//
// Bound: the integer ALU pipe, as in the short-pair kernel, while the queue is full; the column
// steps of the longest passes at its end.  Measured per call (GB300) against blocks, 4-warp teams
// and clusters of 4 blocks per pair: 4,001 global long reads of 500-20,000 bp 75.7 -> 14.4 ms
// (5.1 T cells/s), 32,768 pairs of a mixed stream 678 -> 94-108 ms by draw (5.3 T), 500 local
// contig pairs, part s32, 72.8 -> 10.8 ms.  Reading the boundary one column ahead instead of in
// staged blocks of 16 took 1.2-1.3 times as long.  Blocks of one or two warps instead of eight:
// long reads 14.1 -> 15.8 / 15.5 ms.
#pragma once
#include "pa_launch.h"
#include "pa_short.cuh"

namespace pa {

struct LongUnit {
    uint32_t id[2];
    uint64_t toff[2];
    int32_t m[2], n[2];
    int32_t ms, nh, passes, has_b;
    int32_t rpt;                   // rows per thread of a full pass
    const uint32_t *qt[2];         // score tables of the streamed bases
    ulonglong2 *row;               // boundary cells 0..ms (cell 0 unused)
    uint64_t tag;                  // of the cells this pass writes: launch epoch, pass
    int2 win[3];                   // band mode: first and last column of the passes p - 1, p, p + 1
    int32_t fail;                  // a wait of this pass ran out
};

// A cell's tag: the mark, the launch (a counter of the context, below 2^38), the pass.  Where a slot
// keeps its vertical gap, a tag has its upper half, which the mark sets to a value that no gap has: bits
// 31 and 30 are 1 0, but s32 gaps lie within 2^30 of zero (the classifier's overflow bound), and both
// s16x2 halves are positive (clamped H is at least 2,048, opening a gap takes at most 1,000).
constexpr int kTagPassBits = 24;
constexpr uint64_t kTagMark = 1ull << 63;
__device__ __forceinline__ uint64_t pass_tag(uint64_t epoch, int32_t pass)
{
    return kTagMark | (epoch << kTagPassBits) | (uint32_t)pass;
}

__device__ __forceinline__ ulonglong2 load_cell128(const ulonglong2 *p)
{
    ulonglong2 v;
    asm volatile("{ .reg .b128 r; ld.relaxed.gpu.global.b128 r, [%2]; mov.b128 {%0, %1}, r; }"
                 : "=l"(v.x), "=l"(v.y) : "l"(p));
    return v;
}

__device__ __forceinline__ void store_cell128(ulonglong2 *p, uint64_t x, uint64_t y)
{
    asm volatile("{ .reg .b128 r; mov.b128 r, {%1, %2}; st.relaxed.gpu.global.b128 [%0], r; }" ::"l"(p), "l"(x), "l"(y)
                 : "memory");
}

__device__ __forceinline__ uint32_t load_acquire_gpu(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.acquire.gpu.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void store_release_gpu(uint32_t *p, uint32_t v)
{
    asm volatile("st.release.gpu.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// The cell of column `p` with the wanted tag; polled until it is there.
static __device__ __noinline__ ulonglong2 wait_cell(const ulonglong2 *p, uint64_t tag, uint32_t limit, uint32_t *err,
                                             int32_t *fail)
{
    ulonglong2 v = make_ulonglong2(0ull, 0ull);
    if (*fail == 0) {
        for (uint32_t it = 0; it <= limit; ++it) {
            v = load_cell128(p);
            if (v.y == tag) return v;
            if (it >= 64) __nanosleep(64);
        }
        *fail = 1;
        if (err) atomicOr(err, kErrWaitTimeout);
    }
    return v;
}

// Columns that a warp stages at a time: score tables and top inputs go through shared memory.
constexpr int kStage = 16;

// Pass p of the unit: rows p * rows_full + t * RA + 1 .. + RA (1-based) on thread t.
template <class V, int MODE, int R, int RA>
__device__ __forceinline__ void long_pass(const DpLaunch &L, const LongQueue &Q, const DpParams &P, LongUnit &u, int p,
                                          int32_t rows_full, int t, uint4 *snap, uint4 *cut, StripShared<V> sh, uint4 *stage,
                                          int32_t *ub)
{
    using KC = StripConst<V, MODE>;
    constexpr int NL = V::LANES;
    const int32_t j0 = p * rows_full + t * RA;
    const StripGaps gaps = NL == 2 ? L.gaps16 : L.gaps32;
    const uint32_t CLAMP = V::splat(KC::clampt);
    auto stored = [&](int32_t true_value) { return V::splat(max(true_value + KC::Kt, KC::clampt)); };

    // the columns of the pass: ibase + 1 .. iend (band mode: its window; outside it -infinity)
    constexpr bool BAND = MODE == M_BAND;
    const uint32_t NEGV = V::LANES == 2 ? CLAMP : (uint32_t)kNeg32;
    const int32_t ibase = BAND ? u.win[1].x - 1 : 0, iend = BAND ? u.win[1].y : u.ms, ms = iend - ibase;
    const bool left_out = BAND && ibase > 0;

    uint32_t H[RA], Fr[RA], Sel[RA];
#pragma unroll
    for (int k = 0; k < RA; ++k) {
        const int32_t j = j0 + k;                 // 0-based row of sequence2
        const int ca = j < u.n[0] ? (int)dna_code(L.seq2[u.toff[0] + j]) : -1;
        const int cb = NL == 2 ? (j < u.n[1] ? (int)dna_code(L.seq2[u.toff[1] + j]) : -1) : ca;
        Sel[k] = strip_selector<V>(ca, cb);
        H[k] = left_out ? NEGV : stored(border(P, P.first_row_free, (int64_t)j + 1));
        Fr[k] = H[k] - gaps.goe_h;
    }
    const bool t0 = t == 0;
    uint32_t prevH = left_out ? NEGV : stored(border(P, P.first_row_free, j0));
    if (left_out && t0 && p > 0 && ibase >= u.win[0].x && ibase <= u.win[0].y)   // the diagonal into the window
        prevH = (uint32_t)wait_cell(u.row + ibase, u.tag - 1, L.spin_limit, L.error, &u.fail).x;
    const bool writer = t == 31 && p + 1 < u.passes;
    // columns that the pass above computed
    const int32_t above_a = BAND ? u.win[0].x : 1, above_b = BAND ? (p > 0 ? u.win[0].y : 0) : p > 0 ? iend : 0;
    auto from_above = [&](int32_t col) { return (!BAND || col >= above_a) && col <= above_b; };
    uint32_t sH = 0, sE = 0, sA = 0, sB = 0;
    // lane t < kStage: the tables and the boundary cell of column c0 + t of the next block
    uint32_t nA = 0, nB = 0;
    ulonglong2 nc = make_ulonglong2(0ull, 0ull);
    auto fetch = [&](int32_t c0) {
        const int32_t col = ibase + c0 + t;
        if (t >= kStage || col > iend) return;
        nA = __ldg(u.qt[0] + (NL == 2 ? min(col - 1, u.m[0]) : col - 1));
        if (NL == 2) nB = __ldg(u.qt[1] + min(col - 1, u.m[1]));
        if (from_above(col)) nc = load_cell128(u.row + col);
    };
    auto commit = [&](int32_t c0) {
        const int32_t col = ibase + c0 + t;
        if (t < kStage && col <= iend) {
            uint32_t h, e;
            if (from_above(col)) {
                const uint64_t tag_in = u.tag - 1;
                if (nc.y != tag_in) nc = wait_cell(u.row + col, tag_in, L.spin_limit, L.error, &u.fail);
                h = (uint32_t)nc.x;
                e = (uint32_t)(nc.x >> 32);
            } else if (BAND && p > 0) {           // outside the window of the pass above
                h = e = NEGV;
            } else {                              // the top border
                h = stored(border(P, P.first_column_free, col) - P.shift * col);
                e = h - gaps.goe;
            }
            stage[(c0 + t) & (2 * kStage - 1)] = make_uint4(nA, nB, h, e);
        }
        __syncwarp();
    };
    fetch(1);
    uint32_t best = V::splat(KC::Kt);
    // global modes: a lane's last row as an index into the strip (-1: not this thread's), and the first
    // column a lane ends at
    int32_t own[NL];
    bool any_own = false;
    int32_t mmin = u.ms;
    auto find_row = [&](int l) -> int32_t {
        const int32_t r = (u.n[l] - 1) - j0;
        return MODE != M_LOCAL && r >= 0 && r < RA && (u.n[l] - 1) / rows_full == p ? r : -1;
    };
#pragma unroll
    for (int l = 0; l < NL; ++l) {
        own[l] = find_row(l);
        any_own |= own[l] >= 0;
        mmin = min(mmin, u.m[l]);
    }
    auto own_row = [&](int l) { return BAND ? find_row(l) : own[l]; };   // band mode has no registers to keep it
    // the end rule of the last row (strip_end_track; with a comparison in shared memory on every column
    // a free-end pair of 200,000 x 100 took 132.6 ms, now 86.6)
    const bool row_end = MODE == M_GLOBAL_FREE && P.last_column_free && any_own;
    uint32_t seen = V::splat(KC::below);
    const uint32_t shift_neg = V::splat(-P.shift);
    const int32_t r0 = max(own[0], 0), r1 = max(own[NL - 1], 0);
    if (row_end) {
#pragma unroll
        for (int l = 0; l < NL; ++l) sh.bi[l][threadIdx.x] = 0;
    }

    const int32_t cut_at = strip_cut_at<V, MODE>(P, u);
    auto step = [&](int32_t s, bool active) {
        const int32_t i = ibase + s - t + 1;
        if ((s & (kStage - 1)) == 0 && s < ms) {
            commit(s + 1);
            fetch(s + 1 + kStage);
        }
        const uint4 top = stage[(s + 1) & (2 * kStage - 1)];    // thread 0's column
        const uint32_t xH = __shfl_up_sync(0xffffffffu, sH, 1);
        const uint32_t xE = __shfl_up_sync(0xffffffffu, sE, 1);
        const uint32_t xA = __shfl_up_sync(0xffffffffu, sA, 1);
        const uint32_t xB = NL == 2 ? __shfl_up_sync(0xffffffffu, sB, 1) : 0u;
        if (active) {
            const uint32_t upH = t0 ? top.z : xH;
            uint32_t Ed = t0 ? top.w : xE;
            const uint32_t ta = t0 ? top.x : xA;
            const uint32_t tb = NL == 2 ? (t0 ? top.y : xB) : ta;
            strip_column<V, MODE, RA>(H, Fr, prevH, Ed, gaps, [&](uint32_t d, int k) {
                return table_diagonal<V>(d, ta, tb, Sel[k], Fr[k]);
            });
            prevH = upH;
            sH = H[RA - 1];
            sE = Ed;
            sA = ta;
            sB = tb;
            if (writer) store_cell128(u.row + i, (uint64_t)sH | ((uint64_t)sE << 32), u.tag);
            if (MODE == M_LOCAL)
                strip_track<V, R, RA>(H, best, i, snap, sh);
            else {
                if (row_end) strip_end_track<V, MODE, RA, kBlock>(u, H, seen, shift_neg, i, r0, r1, snap, sh);
                else if (i >= mmin)
                    strip_ends<V, MODE, RA>(P, u, H, i, any_own, snap, sh, own_row);
                if (MODE == M_GLOBAL_FREE && NL == 2 && i == cut_at) strip_cut<RA, kBlock>(H, cut);
            }
        }
    };
    // fill: thread t starts at step t; steady: every thread active; drain
    const int32_t fill_end = min(32, ms + 31);
    int32_t s = 0;
    for (; s < fill_end; ++s) {
        const int32_t i = s - t + 1;
        step(s, i >= 1 && i <= ms);
    }
    for (; s < ms; ++s) step(s, true);
    for (; s < ms + 31; ++s) {
        const int32_t i = s - t + 1;
        step(s, i >= 1 && i <= ms);
    }
    if (MODE == M_LOCAL) strip_track_end<V, R, RA>(best, j0, snap, sh);
    if (row_end) strip_end_offer<V, MODE, kBlock>(P, u, own, sh);
    if (MODE == M_GLOBAL_FREE && P.last_row_free) strip_column_offer<V, MODE, RA, kBlock>(P, u, H, j0, cut, sh);
    if (BAND) {
        // upper bounds on the paths that leave the window (exit_bound): first through its right
        // edge, cells (iend + 1, j), by a horizontal gap from (iend, j) or diagonally from
        // (iend, j - 1), the value that prevH holds for the strip's first row
        const int32_t jlo = p * rows_full + 1, jhi = p * rows_full + 32 * RA;
        const int32_t goe = P.gap_open + P.gap_ext;
        __syncwarp();
#pragma unroll
        for (int l = 0; l < NL; ++l) {
            if (l == 1 && !u.has_b) continue;
            const int32_t ml = u.m[l], nl = u.n[l];
            auto exits = [&](int32_t gv, int32_t dv, int32_t i, int32_t j) {
                ub[l] = max(ub[l], exit_bound(P, gv, dv, i, j, ml, nl));
            };
            if (iend < ml) {
#pragma unroll
                for (int k = 0; k < RA; ++k) {
                    const int32_t j = j0 + k + 1;
                    if (j <= nl)
                        exits(V::get(Fr[k], l) - KC::Kt + P.shift * (iend + 1),
                              V::get(k == 0 ? prevH : H[k - 1], l) - KC::Kt + P.shift * iend + P.smax, iend + 1, j);
                }
            }
            if (jlo > nl) continue;
            if (t0 && L.dp_cells)
                atomicAdd(L.dp_cells, (unsigned long long)(iend - ibase) * (unsigned)(min(jhi, nl) - jlo + 1));
            if (p == 0)       // along the top border past the window, then down into row 1
                for (int32_t i = iend + 1 + t; i <= ml; i += 32)
                    exits(border(P, 0, i) + goe, border(P, 0, i - 1) + P.smax, i, 1);
            if (ibase > 0)    // down the left border, then into column 1 of this pass
                for (int32_t j = jlo + t; j <= min(jhi, nl); j += 32)
                    exits(border(P, 0, j) + goe, border(P, 0, j - 1) + P.smax, 1, j);
            if (p + 1 < u.passes && jhi < nl) {   // through the bottom edge left of the next window
                const int32_t nx = u.win[2].x, last = min(min(iend, nx - 1), ml);
                for (int32_t i = ibase + 1 + t; i <= last; i += 32) {
                    const uint64_t c = load_cell128(u.row + i).x;     // this pass's own cells: no later pass writes them
                    const int32_t cv = P.shift * i - KC::Kt;
                    exits(V::get((uint32_t)(c >> 32), l) + cv, kNeg32, i, jhi + 1);
                    if (i + 1 < nx) exits(kNeg32, V::get((uint32_t)c, l) + cv + P.smax, i + 1, jhi + 1);
                }
            }
        }
    }
}

// Band mode: the column window of pass p, the union of the lanes' windows of the table (monotone
// and overlapping per lane; a lane past its last pass keeps its last window, which ends at its
// column m, so the union is too).
template <int NL>
__device__ __forceinline__ int2 long_window(const DpLaunch &L, const LongUnit &u, int32_t p)
{
    int32_t a = INT32_MAX, b = 0;
#pragma unroll
    for (int l = 0; l < NL; ++l) {
        if (l == 1 && !u.has_b) continue;
        const int32_t pl = (u.n[l] + L.band_rows - 1) / L.band_rows;
        const uint64_t slot = (L.off2[u.id[l]] - L.off2[0]) / (uint64_t)L.band_rows + u.id[l];
        const int2 x = L.band_win[slot + min(p, pl - 1)];
        a = min(a, x.x);
        b = max(b, x.y);
    }
    a = p == 0 ? 1 : max(a, 1);
    return make_int2(a, min(max(b, a), u.ms));
}

// Pair order[first] (and order[first + 1] in s16x2 lanes) as a unit; one thread.
template <int NL>
__device__ __forceinline__ LongUnit long_unit(const DpLaunch &L, const uint32_t *order, uint32_t first, uint32_t count)
{
    LongUnit u;
    u.id[0] = order[first];
    u.has_b = NL == 2 && first + 1 < count;
    u.id[1] = u.has_b ? order[first + 1] : u.id[0];
    for (int l = 0; l < 2; ++l) {
        const uint64_t q0 = L.off1[u.id[l]];
        u.m[l] = (int32_t)(L.off1[u.id[l] + 1] - q0);
        u.toff[l] = L.off2[u.id[l]];
        u.n[l] = (int32_t)(L.off2[u.id[l] + 1] - u.toff[l]);
        u.qt[l] = L.qtab + q0 + u.id[l];
    }
    u.ms = max(u.m[0], u.m[1]);
    u.nh = max(u.n[0], u.n[1]);
    u.fail = 0;
    return u;
}

// The unit that holds ticket `k`: the last u with start[u] <= k (start[0] = 0, start[units] =
// the task count), by a 32-way search of the warp.
__device__ __forceinline__ uint32_t find_unit(const uint32_t *start, uint32_t units, uint32_t k, int lane)
{
    uint32_t lo = 0, hi = units;                  // start[lo] <= k < start[hi]
    while (hi - lo > 1) {
        const uint32_t span = (hi - lo + 31) / 32;
        const uint32_t at = lo + span * (uint32_t)lane;
        const bool le = at < hi && __ldg(start + at) <= k;
        const uint32_t last = 31 - __clz(__ballot_sync(0xffffffffu, le));   // lane 0 always holds
        lo += span * last;
        hi = min(hi, lo + span);
    }
    return lo;
}

// Band mode: the outcome of a unit at list position `first` (band_code: 0 certified, 1 widen, 3
// redo in s32), and the results of certified pairs.
template <class V>
__device__ __forceinline__ void long_band_emit(const DpLaunch &L, const DpParams &P, const LongUnit &u, uint32_t first,
                                               const int32_t *cs, const int32_t *ci, const int32_t *cj,
                                               const int32_t *ub, bool failed)
{
    using KC = StripConst<V, M_BAND>;
#pragma unroll
    for (int l = 0; l < V::LANES; ++l) {
        if (l == 1 && !u.has_b) continue;
        pa_result r;
        r.score = failed ? INT32_MIN : cs[l];
        r.end1 = failed ? 0 : ci[l];
        r.end2 = failed ? 0 : cj[l];
        r.width = V::WIDTH;
        r.flags = failed ? PA_RESULT_ERROR : (uint8_t)(PA_RESULT_BANDED | (L.rerun ? PA_RESULT_RERUN : 0));
        r.band_rounds = failed ? 0 : (uint16_t)L.band_round;
        uint8_t code = 1;
        if (failed) code = 0;
        else if (V::LANES == 2 && (int64_t)cs[l] - (int64_t)P.shift * ci[l] <= (int64_t)KC::floor_true)
            code = 3;                             // a clamp may have reached it
        else if (cs[l] != INT32_MIN && ub[l] <= cs[l])
            code = 0;                             // no path that leaves the band scores more
        if (code == 0) L.out[u.id[l]] = r;
        L.band_code[first + l] = code;
        if (L.band_ub) L.band_ub[u.id[l]] = failed ? INT32_MAX : ub[l];
    }
}

// The queue of a band round's units (one block): their passes in the order of the windows' first
// columns (512 at a time), so that a pass is handed out about when the pass above it reaches its
// window -- a unit's passes one after another would leave most of them waiting in their warps,
// as a window keeps only a part of its unit's passes busy.  One thread lists a unit's passes, so
// a pass never stands before the one above it.  Learned band on the mixed stream of 32,768 pairs
// (1 % of 20-50 kb): 79.6 ms per call, 572 with teams, blocks and clusters per pair.
template <int NL>
__global__ void __launch_bounds__(1024) k_band_plan(DpLaunch L, LongQueue Q, unsigned long long *epoch)
{
    __shared__ uint32_t bucket[2048];
    __shared__ uint32_t part[32];
    const uint32_t count = *L.count_ptr, units = (count + NL - 1) / NL;
    const uint32_t *order = L.order + *L.begin_ptr;
    for (int k = threadIdx.x; k < 2048; k += 1024) bucket[k] = 0;
    __syncthreads();
    auto each_pass = [&](auto take) {
        for (uint32_t uu = threadIdx.x; uu < units; uu += 1024) {
            const LongUnit u = long_unit<NL>(L, order, (units - 1 - uu) * NL, count);
            const int32_t passes = (u.nh + L.band_rows - 1) / L.band_rows;
            uint32_t b = 0;
            for (int32_t p = 0; p < passes; ++p) {
                b = max(b, min((uint32_t)long_window<NL>(L, u, p).x >> 9, 2047u));
                take(uu, (uint32_t)p, b);
            }
        }
    };
    each_pass([&](uint32_t, uint32_t, uint32_t b) { atomicAdd(&bucket[b], 1u); });
    __syncthreads();
    // exclusive scan of the 2,048 buckets, two per thread
    const uint32_t x0 = bucket[2 * threadIdx.x], x1 = bucket[2 * threadIdx.x + 1];
    const int lane = threadIdx.x & 31;
    uint32_t v = x0 + x1;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
    }
    if (lane == 31) part[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t before = 0;
    for (int w = 0; w < (int)(threadIdx.x >> 5); ++w) before += part[w];
    const uint32_t ex = before + v - x0 - x1;
    bucket[2 * threadIdx.x] = ex;
    bucket[2 * threadIdx.x + 1] = ex + x0;
    if (threadIdx.x == 1023) {
        Q.words->tasks = before + v;
        Q.words->epoch = (uint64_t)atomicAdd(epoch, 1ull) + 1ull;
    }
    for (uint32_t uu = threadIdx.x; uu < units; uu += 1024) { Q.done[uu] = 0u; Q.fail[uu] = 0u; }
    __syncthreads();
    each_pass([&](uint32_t uu, uint32_t p, uint32_t b) { Q.tasks[atomicAdd(&bucket[b], 1u)] = make_uint2(uu, p); });
}

template <class V, int MODE, int R>
__global__ void __launch_bounds__(kBlock, 2) dp_long(DpLaunch L, LongQueue Q, DpParams P)
{
    using KC = StripConst<V, MODE>;
    constexpr int NL = V::LANES;
    constexpr int NW = kBlock / 32;
    constexpr bool BAND = MODE == M_BAND;
    __shared__ uint4 snap_store[(MODE == M_LOCAL ? NL : 1) * (R / 4) * kBlock];
    __shared__ uint4 cut_store[MODE == M_GLOBAL_FREE && NL == 2 ? (R / 4) * kBlock : 1];
    __shared__ LongUnit s_unit[NW];
    __shared__ uint4 s_stage[NW][2 * kStage];
    __shared__ int32_t s_cand[NL][3][kBlock];
    __shared__ int32_t s_bi[MODE == M_LOCAL ? NL : MODE == M_GLOBAL_FREE ? 2 * NL : 1][kBlock];
    uint4 *snap = snap_store + threadIdx.x;
    uint4 *cut = cut_store + (MODE == M_GLOBAL_FREE && NL == 2 ? threadIdx.x : 0);
    StripShared<V> sh{s_cand, s_bi};
    const int t = threadIdx.x & 31;
    LongUnit &su = s_unit[threadIdx.x >> 5];
    const uint32_t count = *L.count_ptr;
    const uint32_t units = (count + NL - 1) / NL;
    const uint32_t total = Q.words->tasks;
    if (!strip_warp_takes_part(total)) return;
    const uint64_t epoch = Q.words->epoch;
    const uint32_t *order = L.order + *L.begin_ptr;

    for (;;) {
        uint32_t ticket = 0;
        if (t == 0) ticket = atomicAdd(L.unit_counter, 1u);
        ticket = __shfl_sync(0xffffffffu, ticket, 0);
        if (ticket >= total) break;
        uint32_t uu;
        int p;
        if (BAND) {
            const uint2 task = __ldg(Q.tasks + ticket);
            uu = task.x;
            p = (int)task.y;
        } else {
            uu = find_unit(Q.start, units, ticket, t);
            p = (int)(ticket - __ldg(Q.start + uu));
        }
        if (t == 0) {
            LongUnit u = long_unit<NL>(L, order, (units - 1 - uu) * NL, count);   // largest units first
            u.rpt = BAND ? L.band_rows / 32 : __ldcg(&Q.rec[uu].rpt);
            u.passes = (u.nh + 32 * u.rpt - 1) / (32 * u.rpt);
            const uint32_t owner = u.m[1] > u.m[0] ? u.id[1] : u.id[0];
            u.row = Q.cells + (L.off1[owner] + owner);        // cells 0..m(owner) = 0..ms
            u.tag = pass_tag(epoch, p);
            if (BAND)
                for (int k = 0; k < 3; ++k) u.win[k] = long_window<NL>(L, u, min(max(p + k - 1, 0), u.passes - 1));
            su = u;
        }
#pragma unroll
        for (int l = 0; l < NL; ++l) {
            sh.s(l) = MODE == M_LOCAL ? 0 : INT32_MIN;
            sh.i(l) = 0;
            sh.j(l) = 0;
        }
        __syncwarp();
        int32_t ub[NL];
#pragma unroll
        for (int l = 0; l < NL; ++l) ub[l] = INT32_MIN;
        {
            const int32_t rows_full = 32 * su.rpt, rem = su.nh - p * rows_full;
            const int32_t rpt = rem >= rows_full ? su.rpt : ((rem + 32 * kChunk - 1) / (32 * kChunk)) * kChunk;
            switch (rpt / kChunk) {
            case 1: long_pass<V, MODE, R, 4>(L, Q, P, su, p, rows_full, t, snap, cut, sh, s_stage[threadIdx.x >> 5], ub); break;
            case 2: long_pass<V, MODE, R, 8>(L, Q, P, su, p, rows_full, t, snap, cut, sh, s_stage[threadIdx.x >> 5], ub); break;
            case 3: long_pass<V, MODE, R, 12>(L, Q, P, su, p, rows_full, t, snap, cut, sh, s_stage[threadIdx.x >> 5], ub); break;
            case 4: long_pass<V, MODE, R, 16>(L, Q, P, su, p, rows_full, t, snap, cut, sh, s_stage[threadIdx.x >> 5], ub); break;
            case 5: long_pass<V, MODE, R, R >= 20 ? 20 : R>(L, Q, P, su, p, rows_full, t, snap, cut, sh, s_stage[threadIdx.x >> 5], ub); break;
            default: long_pass<V, MODE, R, R>(L, Q, P, su, p, rows_full, t, snap, cut, sh, s_stage[threadIdx.x >> 5], ub); break;
            }
        }
        __syncwarp();
        int32_t cs[NL], ci[NL], cj[NL];
#pragma unroll
        for (int l = 0; l < NL; ++l) {
            cs[l] = sh.s(l);
            ci[l] = sh.i(l);
            cj[l] = sh.j(l);
            for (int off = 16; off >= 1; off >>= 1) {
                const int32_t os = __shfl_xor_sync(0xffffffffu, cs[l], off);
                const int32_t oi = __shfl_xor_sync(0xffffffffu, ci[l], off);
                const int32_t oj = __shfl_xor_sync(0xffffffffu, cj[l], off);
                if (better(os, oi, oj, cs[l], ci[l], cj[l])) { cs[l] = os; ci[l] = oi; cj[l] = oj; }
            }
            if (BAND) ub[l] = __reduce_max_sync(0xffffffffu, ub[l]);
        }
        if (t == 0) {
            const LongUnit u = su;
            // the exits assume monotone, overlapping windows: refuse to certify otherwise
            if (BAND && p > 0 && (u.win[1].x < u.win[0].x || u.win[1].y < u.win[0].y || u.win[1].x > u.win[0].y))
                for (int l = 0; l < NL; ++l) ub[l] = INT32_MAX;
            int32_t fail = u.fail;
            LongRecord *rec = Q.rec + uu;
            if (p > 0) {                          // the candidates of the passes above
                bool ready = false;
                for (uint32_t it = 0; it <= L.spin_limit; ++it) {
                    if (load_acquire_gpu(Q.done + uu) >= (uint32_t)p) { ready = true; break; }
                    if (it >= 64) __nanosleep(64);
                }
                if (!ready) {
                    fail = 1;
                    if (L.error) atomicOr(L.error, kErrWaitTimeout);
                } else {
                    fail |= (int32_t)__ldcg(Q.fail + uu);
#pragma unroll
                    for (int l = 0; l < NL; ++l) {
                        const int32_t os = __ldcg(&rec->s[l]), oi = __ldcg(&rec->i[l]), oj = __ldcg(&rec->j[l]);
                        if (better(os, oi, oj, cs[l], ci[l], cj[l])) { cs[l] = os; ci[l] = oi; cj[l] = oj; }
                        if (BAND) ub[l] = max(ub[l], __ldcg(&rec->ub[l]));
                    }
                }
            }
            if (p + 1 < u.passes) {
                // the fail word is set once and stays: a unit with a wait that ran out is an error
                // whatever its record holds
                if (fail) Q.fail[uu] = 1u;
#pragma unroll
                for (int l = 0; l < NL; ++l) { rec->s[l] = cs[l]; rec->i[l] = ci[l]; rec->j[l] = cj[l]; rec->ub[l] = ub[l]; }
                store_release_gpu(Q.done + uu, (uint32_t)p + 1);
            } else if (BAND) {
                long_band_emit<V>(L, P, u, (units - 1 - uu) * NL, cs, ci, cj, ub, fail != 0);
            } else {
                strip_emit<V, MODE>(L, P, u.id, u.m, u.n, u.has_b != 0, cs, ci, cj, fail != 0);
            }
        }
        __syncwarp();
    }
}

}  // namespace pa
