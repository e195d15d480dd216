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
// cell: no flag, no fence, no order between cells is needed.  The row is reused in place:
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
// and clusters of 4 blocks per pair: 4,001 global long reads of 500-20,000 bp 75.7 -> 15.0 ms
// (4.9 T cells/s of DP), 32,768 pairs of a mixed stream 678 -> 105 ms (5.2 T), 500 local contig
// pairs, part s32, 72.8 -> 12.4 ms.  Reading the boundary one column ahead instead of in staged
// blocks of 16: 19.1, 131 and 14.8 ms.
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
    int32_t fail;                  // a wait of this pass ran out
};

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
        for (uint32_t it = 0; it < limit; ++it) {
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
                                          int32_t rows_full, int t, uint4 *snap, StripShared<V> sh, uint4 *stage)
{
    using KC = StripConst<V, MODE>;
    constexpr int NL = V::LANES;
    constexpr bool SHIFTED = MODE != M_LOCAL;
    const int32_t j0 = p * rows_full + t * RA;
    // the gap constants in lane form, operands from the kernel's parameters
    const uint32_t GOEA = Q.goea, EXTA = Q.exta, GOEH = SHIFTED ? Q.goeh : Q.goea, EXTH = SHIFTED ? Q.exth : Q.exta;
    const uint32_t CLAMP = V::splat(KC::clampt);
    auto stored = [&](int32_t true_value) { return V::splat(max(true_value + KC::Kt, KC::clampt)); };

    uint32_t H[RA], Fr[RA], Sel[RA];
#pragma unroll
    for (int k = 0; k < RA; ++k) {
        const int32_t j = j0 + k;                 // 0-based row of sequence2
        const int ca = j < u.n[0] ? (int)dna_code(L.seq2[u.toff[0] + j]) : -1;
        const int cb = NL == 2 ? (j < u.n[1] ? (int)dna_code(L.seq2[u.toff[1] + j]) : -1) : ca;
        Sel[k] = V::selector(ca, cb);
        H[k] = stored(border(P, P.first_row_free, (int64_t)j + 1));
        Fr[k] = V::subc(H[k], GOEH);
    }
    uint32_t prevH = stored(border(P, P.first_row_free, j0));
    const bool t0 = t == 0;
    const bool writer = t == 31 && p + 1 < u.passes;
    const int32_t ms = u.ms;
    uint32_t sH = 0, sE = 0, sA = 0, sB = 0;
    // lane t < kStage: the tables and the boundary cell of column c0 + t of the next block
    uint32_t nA = 0, nB = 0;
    ulonglong2 nc = make_ulonglong2(0ull, 0ull);
    auto fetch = [&](int32_t c0) {
        const int32_t col = c0 + t;
        if (t >= kStage || col > ms) return;
        nA = __ldg(u.qt[0] + (NL == 2 ? min(col - 1, u.m[0]) : col - 1));
        if (NL == 2) nB = __ldg(u.qt[1] + min(col - 1, u.m[1]));
        if (p > 0) nc = load_cell128(u.row + col);
    };
    auto commit = [&](int32_t c0) {
        const int32_t col = c0 + t;
        if (t < kStage && col <= ms) {
            uint32_t h, e;
            if (p > 0) {
                const uint64_t tag_in = u.tag - 1;
                if (nc.y != tag_in) nc = wait_cell(u.row + col, tag_in, L.spin_limit, L.error, &u.fail);
                h = (uint32_t)nc.x;
                e = (uint32_t)(nc.x >> 32);
            } else {                              // the top border
                h = stored(border(P, P.first_column_free, col) - P.shift * col);
                e = V::subc(h, GOEA);
            }
            stage[col & (2 * kStage - 1)] = make_uint4(nA, nB, h, e);
        }
        __syncwarp();
    };
    fetch(1);
    uint32_t best = V::splat(KC::Kt);
    // global modes: whether a lane's last row is this thread's, and the first column a lane ends at
    auto own_row = [&](int l) -> int32_t {        // its index in the strip, or -1
        const int32_t r = (u.n[l] - 1) - j0;
        return r >= 0 && r < RA && (u.n[l] - 1) / rows_full == p ? r : -1;
    };
    bool any_own = false;
    int32_t mmin = ms;
    if (MODE != M_LOCAL) {
#pragma unroll
        for (int l = 0; l < NL; ++l) {
            any_own |= own_row(l) >= 0;
            mmin = min(mmin, u.m[l]);
        }
    }

    auto step = [&](int32_t s, bool active) {
        const int32_t i = s - t + 1;
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
            uint32_t tt = V::addmax(prevH, prmt(ta, tb, Sel[0]), Fr[0]);
#pragma unroll
            for (int k = 0; k < RA; ++k) {
                // the next row's diagonal term uses this row's H before it is replaced
                const uint32_t tn = k + 1 < RA ? V::addmax(H[k], prmt(ta, tb, Sel[k + 1]), Fr[k + 1]) : 0u;
                const uint32_t h = V::hmax(tt, Ed, CLAMP);
                H[k] = h;
                const uint32_t hoe = V::subc(h, GOEA);
                Fr[k] = V::max2(V::subc(Fr[k], EXTH), SHIFTED ? V::subc(h, GOEH) : hoe);
                Ed = V::max2(V::subc(Ed, EXTA), hoe);
                tt = tn;
            }
            prevH = upH;
            sH = H[RA - 1];
            sE = Ed;
            sA = ta;
            sB = tb;
            if (writer) store_cell128(u.row + i, (uint64_t)sH | ((uint64_t)sE << 32), u.tag);
            if (MODE == M_LOCAL) {
                const uint32_t cm = tree_max<V, RA>(H);
                const uint32_t nb = V::max2(best, cm);
                const uint32_t x = nb ^ best;
                best = nb;
                if (x != 0u) {
#pragma unroll
                    for (int l = 0; l < NL; ++l) {
                        if (V::improved(x, l)) {
                            sh.bi[l][threadIdx.x] = i;
#pragma unroll
                            for (int v = 0; v < RA / 4; ++v)
                                snap[(l * (R / 4) + v) * kBlock] =
                                    make_uint4(H[4 * v], H[4 * v + 1], H[4 * v + 2], H[4 * v + 3]);
                        }
                    }
                }
            } else if ((MODE == M_GLOBAL_FREE && P.last_column_free && any_own) || i >= mmin) {
                if (any_own) {
#pragma unroll
                    for (int v = 0; v < RA / 4; ++v)
                        snap[v * kBlock] = make_uint4(H[4 * v], H[4 * v + 1], H[4 * v + 2], H[4 * v + 3]);
                }
#pragma unroll
                for (int l = 0; l < NL; ++l) {
                    if (l == 1 && !u.has_b) continue;
                    const int32_t base = P.shift * i - KC::Kt, ml = u.m[l], r = own_row(l);
                    if (r >= 0 && (i == ml || (MODE == M_GLOBAL_FREE && P.last_column_free && i < ml))) {
                        // the row's H, read back from the snapshot
                        const uint32_t *q = reinterpret_cast<const uint32_t *>(snap + (r >> 2) * kBlock);
                        sh.offer(l, V::get(q[r & 3], l) + base, i, u.n[l]);
                    }
                    if (MODE == M_GLOBAL_FREE && P.last_row_free && i == ml) {
#pragma unroll
                        for (int k = 0; k < RA; ++k)
                            if (j0 + k + 1 <= u.n[l]) sh.offer(l, V::get(H[k], l) + base, i, j0 + k + 1);
                    }
                }
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
    if (MODE == M_LOCAL) {
#pragma unroll
        for (int l = 0; l < NL; ++l) {
            const int32_t b = V::get(best, l);
            if (b > KC::Kt) {                     // improved in this pass: snapshot and column are set
                int32_t kk = 0;
                for (int v = RA / 4 - 1; v >= 0; --v) {
                    const uint4 q = snap[(l * (R / 4) + v) * kBlock];
                    if (V::get(q.w, l) == b) kk = 4 * v + 3;
                    if (V::get(q.z, l) == b) kk = 4 * v + 2;
                    if (V::get(q.y, l) == b) kk = 4 * v + 1;
                    if (V::get(q.x, l) == b) kk = 4 * v;
                }
                sh.offer(l, b - KC::Kt, sh.bi[l][threadIdx.x], j0 + kk + 1);
            }
        }
    }
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

template <class V, int MODE, int R>
__global__ void __launch_bounds__(kBlock, 2) dp_long(DpLaunch L, LongQueue Q, DpParams P)
{
    using KC = StripConst<V, MODE>;
    constexpr int NL = V::LANES;
    constexpr int NW = kBlock / 32;
    __shared__ uint4 snap_store[(MODE == M_LOCAL ? NL : 1) * (R / 4) * kBlock];
    __shared__ LongUnit s_unit[NW];
    __shared__ uint4 s_stage[NW][2 * kStage];
    __shared__ int32_t s_cand[NL][3][kBlock];
    __shared__ int32_t s_bi[MODE == M_LOCAL ? NL : 1][kBlock];
    uint4 *snap = snap_store + threadIdx.x;
    StripShared<V> sh{s_cand, s_bi};
    const int t = threadIdx.x & 31;
    LongUnit &su = s_unit[threadIdx.x >> 5];
    const uint32_t count = *L.count_ptr;
    const uint32_t units = (count + NL - 1) / NL;
    const uint32_t total = Q.words->tasks;
    const uint32_t budget = Q.words->budget;
    const int32_t floor_rows = Q.words->floor_rows;
    const uint64_t epoch = Q.words->epoch;
    const uint32_t *order = L.order + *L.begin_ptr;

    for (;;) {
        uint32_t ticket = 0;
        if (t == 0) ticket = atomicAdd(L.unit_counter, 1u);
        ticket = __shfl_sync(0xffffffffu, ticket, 0);
        if (ticket >= total) break;
        const uint32_t uu = find_unit(Q.start, units, ticket, t);
        const int p = (int)(ticket - __ldg(Q.start + uu));
        if (t == 0) {
            const uint32_t first = (units - 1 - uu) * NL;     // largest units first
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
            u.rpt = long_rows(budget, floor_rows, u.ms);
            u.passes = (u.nh + 32 * u.rpt - 1) / (32 * u.rpt);
            const uint32_t owner = u.m[1] > u.m[0] ? u.id[1] : u.id[0];
            u.row = Q.cells + (L.off1[owner] + owner);        // cells 0..m(owner) = 0..ms
            u.tag = (epoch << 13) | (uint32_t)p;              // at most 2^20 / 128 = 8,192 passes
            u.fail = 0;
            su = u;
        }
#pragma unroll
        for (int l = 0; l < NL; ++l) {
            sh.s(l) = MODE == M_LOCAL ? 0 : INT32_MIN;
            sh.i(l) = 0;
            sh.j(l) = 0;
        }
        __syncwarp();
        {
            const int32_t rows_full = 32 * su.rpt, rem = su.nh - p * rows_full;
            const int32_t rpt = rem >= rows_full ? su.rpt : ((rem + 32 * kChunk - 1) / (32 * kChunk)) * kChunk;
            switch (rpt / kChunk) {
            case 1: long_pass<V, MODE, R, 4>(L, Q, P, su, p, rows_full, t, snap, sh, s_stage[threadIdx.x >> 5]); break;
            case 2: long_pass<V, MODE, R, 8>(L, Q, P, su, p, rows_full, t, snap, sh, s_stage[threadIdx.x >> 5]); break;
            case 3: long_pass<V, MODE, R, 12>(L, Q, P, su, p, rows_full, t, snap, sh, s_stage[threadIdx.x >> 5]); break;
            case 4: long_pass<V, MODE, R, 16>(L, Q, P, su, p, rows_full, t, snap, sh, s_stage[threadIdx.x >> 5]); break;
            case 5: long_pass<V, MODE, R, 20>(L, Q, P, su, p, rows_full, t, snap, sh, s_stage[threadIdx.x >> 5]); break;
            default: long_pass<V, MODE, R, 24>(L, Q, P, su, p, rows_full, t, snap, sh, s_stage[threadIdx.x >> 5]); break;
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
        }
        if (t == 0) {
            const LongUnit u = su;
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
                    }
                }
            }
            if (p + 1 < u.passes) {
                // the fail word is set once and stays: a unit with a wait that ran out is an error
                // whatever its record holds
                if (fail) Q.fail[uu] = 1u;
#pragma unroll
                for (int l = 0; l < NL; ++l) { rec->s[l] = cs[l]; rec->i[l] = ci[l]; rec->j[l] = cj[l]; }
                store_release_gpu(Q.done + uu, (uint32_t)p + 1);
            } else {
                strip_emit<V, MODE>(L, P, u.id, u.m, u.n, u.has_b != 0, cs, ci, cj, fail != 0);
            }
        }
        __syncwarp();
    }
}

}  // namespace pa
