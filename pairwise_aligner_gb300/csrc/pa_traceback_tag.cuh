// pa_traceback_tag.cuh -- traceback with tagged values.
//
// The recurrence, borders and ties are those of pa_traceback.cu; what differs is where a cell's
// direction comes from.  Values are held times 16, and bits 2-3 name the candidate: H candidates
// carry 12 (local start), 8 (diagonal), 4 (P) or 0 (Q), so the maximum that decides H also
// decides, with the right ties, where it came from.  An opening P carries 1 more and an opening Q
// 2, an extending one nothing, so the gap maxima leave the bits "opened" in place.  The nibble of
// a cell is the low bits of the three results XORed: 8 ALU operations for the whole cell (9 in
// local mode) instead of about 27 with compares and selects.  Under SC_TABLE the 8 of the diagonal
// comes with the score: the table holds 2 * score + 1, the row's one-hot byte is 8.
//
// Nibble: bits 2-3 the candidate of H(i,j), XOR 4 (P always carries its 4); bit 0 P(i+1,j) opens from
// H(i,j); bit 1 Q(i,j+1) opens.
//
// The passes (512 rows, 16 per lane; the last one ra = ceil(rows left / 128) * 4 per lane) of all
// pairs of a chunk stand in one queue, largest pair first, and hand their bottom rows on through
// tagged cells as in pa_long.cuh; a pass leaves its end-cell candidate, and k_tb_walk walks the
// paths when all passes are done.  If a wait ran out it walks none, and the caller runs k_traceback.  Words of pass p of a pair start at p * (m + 31) * 64; a step
// holds a word per lane (ra <= 8) or two; row k of a lane's first word is its nibble k (of a
// shorter strip: k + 8 - ra), rows 8.. are in the second (nibble k - 8 + 16 - ra).
//
// Bound: the integer ALU pipe, 76 % busy over the 4.74 ms of k_tb_dp (the last passes are padded to
// 128 rows), and the host copies around it: 4,096 global pairs of 500-2,000 rows 6.4 ms per call, 17.0
// with one pair per warp and compares.  Strip heights in steps of 2 instead of 4: 7.6, as eight bodies
// do not stay in the instruction cache (neighbouring warps run last passes of different heights).
#pragma once
#include "pa_long.cuh"

namespace pa {

constexpr int kTagThreads = 128;
constexpr int kTagRows = 16;
constexpr int kTagPassRows = 32 * kTagRows;
static_assert(kTagPassRows == 2 * kTracebackPassRows, "the host sizes the direction words in half passes");

__device__ __forceinline__ bool tag_better(int32_t v, int32_t i, int32_t j, int32_t bv, int32_t bi, int32_t bj)
{
    return v > bv || (v == bv && (i < bi || (i == bi && j < bj)));
}

// The launch's number, and cleared queue heads.
__global__ void k_tb_start(TbLaunch L)
{
    *L.my_epoch = ++*L.epoch;
    L.queue[0] = L.queue[1] = 0u;
}

struct TagPass {
    int32_t m, n, passes, ra;
    const uint8_t *a_seq, *b_seq;
    uint32_t *D;
    ulonglong2 *row;
    uint64_t tag;
    int32_t fail;
};

// Rows per lane of pass p.
__device__ __forceinline__ int32_t tag_rows(int32_t n, int32_t p, int32_t passes)
{
    return p + 1 < passes ? kTagRows : 4 * ((n - p * kTagPassRows + 127) / 128);
}

template <bool LOCAL, int SC, int RA>
__device__ __forceinline__ void tag_pass(const TbLaunch &L, const DpParams &P, TagPass &w, int p, int t, uint4 *stage,
                                         uint32_t *snap, int32_t &bv, int32_t &bi, int32_t &bj)
{
    const int32_t goe16 = 16 * (P.gap_open + P.gap_ext), ext16 = 16 * P.gap_ext;
    const int32_t hit16 = 16 * P.match + 8, miss16 = 16 * P.mismatch + 8;
    const int32_t m = w.m, n = w.n, j0 = p * kTagPassRows + t * RA;
    const uint32_t match4 = (uint8_t)(2 * P.match + 1) * 0x01010101u, mis4 = (uint8_t)(2 * P.mismatch + 1) * 0x01010101u;
    const bool t0 = t == 0, writer = t == 31 && p + 1 < w.passes;
    int32_t H[RA], Pg[RA];
    uint32_t Sel[RA];
#pragma unroll
    for (int k = 0; k < RA; ++k) {
        const int32_t j = j0 + k;
        const uint32_t b = j < n ? (uint32_t)w.b_seq[j] : 0x100u;
        if (SC == SC_TABLE) Sel[k] = b < 0x100u ? 8u << (8 * dna_code(b)) : 0u;       // a padding row scores 0
        else if (SC == SC_BYTES) Sel[k] = b;
        else Sel[k] = b < 0x100u ? (uint32_t)__ldg(L.rank + b) : 0x400u;
        H[k] = 16 * border(P, P.first_row_free, (int64_t)j + 1);
        Pg[k] = H[k] + goe16 + 4;
    }
    int32_t prevH = 16 * border(P, P.first_row_free, j0);
    int32_t sH = 0, sQ = 0;
    uint32_t sA = 0, nA = 0;
    ulonglong2 nc = make_ulonglong2(0ull, 0ull);
    auto fetch = [&](int32_t c0) {
        const int32_t col = c0 + t;
        if (t >= kStage || col > m) return;
        const uint32_t a = w.a_seq[col - 1];
        nA = SC == SC_TABLE ? score_table(a, match4, mis4) : SC == SC_BYTES ? a : (uint32_t)(__ldg(L.rank + a) * L.dim);
        if (p > 0) nc = load_cell128(w.row + col);
    };
    auto commit = [&](int32_t c0) {
        const int32_t col = c0 + t;
        if (t < kStage && col <= m) {
            int32_t h, q;
            if (p > 0) {
                if (nc.y != w.tag - 1) nc = wait_cell(w.row + col, w.tag - 1, L.spin_limit, L.error, &w.fail);
                h = (int32_t)(uint32_t)nc.x;
                q = (int32_t)(uint32_t)(nc.x >> 32);
            } else {
                h = 16 * border(P, P.first_column_free, col);
                q = h + goe16;
            }
            stage[col & (2 * kStage - 1)] = make_uint4(nA, 0u, (uint32_t)h, (uint32_t)q);
        }
        __syncwarp();
    };
    fetch(1);
    // the strip index of row n, or -1 (global modes); the best H so far (local mode)
    const int32_t own = !LOCAL && n > j0 && n <= j0 + RA ? n - 1 - j0 : -1;
    const bool lcf = P.last_column_free, lrf = P.last_row_free;
    int32_t best = 0, best_i = 0;
    uint32_t *D = w.D;
    constexpr int WORDS = RA > 8 ? 2 : 1;

    auto step = [&](int32_t s, bool active) {
        const int32_t i = s - t + 1;
        if ((s & (kStage - 1)) == 0 && s < m) {
            commit(s + 1);
            fetch(s + 1 + kStage);
        }
        const uint4 top = stage[(s + 1) & (2 * kStage - 1)];
        const int32_t xH = __shfl_up_sync(0xffffffffu, sH, 1);
        const int32_t xQ = __shfl_up_sync(0xffffffffu, sQ, 1);
        const uint32_t xA = __shfl_up_sync(0xffffffffu, sA, 1);
        if (active) {
            const int32_t upH = t0 ? (int32_t)top.z : xH;
            int32_t Q = t0 ? (int32_t)top.w : xQ;
            const uint32_t a = t0 ? top.x : xA;
            int32_t d = prevH;
            uint32_t word[2] = {0u, 0u};
#pragma unroll
            for (int k = 0; k < RA; ++k) {
                int32_t x;
                if (SC == SC_TABLE) x = __dp4a((int)a, (int)Sel[k], d);
                else if (SC == SC_BYTES) x = d + (Sel[k] == a ? hit16 : miss16);
                else x = d + (Sel[k] < 0x400u ? 16 * __ldg(L.matrix + a + Sel[k]) + 8 : 16 * P.spad);
                int32_t h = __vimax3_s32(x, Pg[k], Q);
                if (LOCAL) h = max(h, 12);
                d = H[k];
                const int32_t hn = h & ~15;
                H[k] = hn;
                const int32_t pn = __viaddmax_s32(Pg[k], ext16, hn + (goe16 + 5));
                const int32_t qn = __viaddmax_s32(Q, ext16, hn + (goe16 + 2));
                word[k >> 3] = __funnelshift_r(word[k >> 3], (uint32_t)(h ^ pn ^ qn), 4);
                Pg[k] = pn & ~1;
                Q = qn & ~2;
            }
            prevH = upH;
            sH = H[RA - 1];
            sQ = Q;
            sA = a;
            const int64_t at = (int64_t)s * 32 + t;
            if (WORDS == 2) reinterpret_cast<uint2 *>(D)[at] = make_uint2(word[0], word[1]);
            else D[at] = word[0];
            if (writer) store_cell128(w.row + i, (uint64_t)(uint32_t)sH | ((uint64_t)(uint32_t)sQ << 32), w.tag);
            if (LOCAL) {
                int32_t cm = H[0];
#pragma unroll
                for (int k = 1; k < RA; k += 2) cm = __vimax3_s32(cm, H[k], H[k + 1 < RA ? k + 1 : k]);
                if (cm > best) {
                    best = cm;
                    best_i = i;
#pragma unroll
                    for (int k = 0; k < RA; ++k) snap[k * kTagThreads] = (uint32_t)H[k];
                }
            } else if (lcf || i == m) {
                if (own >= 0) {
#pragma unroll
                    for (int k = 0; k < RA; ++k) snap[k * kTagThreads] = (uint32_t)H[k];
                    const int32_t v = (int32_t)snap[own * kTagThreads] >> 4;
                    if (tag_better(v, i, n, bv, bi, bj)) { bv = v; bi = i; bj = n; }
                }
                if (lrf && i == m) {
#pragma unroll
                    for (int k = 0; k < RA; ++k) {
                        const int32_t j = j0 + k + 1;
                        if (j <= n && tag_better(H[k] >> 4, m, j, bv, bi, bj)) { bv = H[k] >> 4; bi = m; bj = j; }
                    }
                }
            }
        }
    };
    // one loop for fill, steady state and drain: with a body for each, the strips' code did not stay
    // in the instruction cache
    for (int32_t s = 0; s < m + 31; ++s) step(s, (uint32_t)(s - t) < (uint32_t)m);
    if (LOCAL && best > 0) {
        // the first row of column best_i with the best value; a row past n never wins: the value
        // that reaches it stands in an earlier column or an earlier row
        int32_t k = 0;
        while ((int32_t)snap[k * kTagThreads] != best) ++k;
        bv = best >> 4;
        bi = best_i;
        bj = j0 + k + 1;
    }
}

template <bool LOCAL, int SC>
__global__ void __launch_bounds__(kTagThreads, 4) k_tb_dp(TbLaunch L, DpParams P)
{
    constexpr int NW = kTagThreads / 32;
    __shared__ uint4 s_stage[NW][2 * kStage];
    __shared__ uint32_t s_snap[kTagRows * kTagThreads];
    __shared__ TagPass s_pass[NW];
    const int t = threadIdx.x & 31;
    TagPass &w = s_pass[threadIdx.x >> 5];
    uint4 *stage = s_stage[threadIdx.x >> 5];
    uint32_t *snap = s_snap + threadIdx.x;
    const uint32_t total = L.start[L.count];
    if (!strip_warp_takes_part(total)) return;
    const uint64_t epoch = *L.my_epoch;
    for (;;) {
        uint32_t ticket = 0;
        if (t == 0) ticket = atomicAdd(L.queue, 1u);
        ticket = __shfl_sync(0xffffffffu, ticket, 0);
        if (ticket >= total) break;
        const uint32_t u = find_unit(L.start, L.count, ticket, t);
        const int32_t p = (int32_t)(ticket - __ldg(L.start + u));
        if (t == 0) {
            const uint32_t q = L.order[u], k = L.first + q;
            TagPass x;
            const uint64_t q0 = L.off1[k], r0 = L.off2[k];
            x.m = (int32_t)(L.off1[k + 1] - q0);
            x.n = (int32_t)(L.off2[k + 1] - r0);
            x.passes = (x.n + kTagPassRows - 1) / kTagPassRows;
            x.ra = tag_rows(x.n, p, x.passes);
            x.a_seq = L.seq1 + q0;
            x.b_seq = L.seq2 + r0;
            x.D = L.dir + L.dir_off[q] + (uint64_t)p * (uint32_t)(x.m + 31) * 64u;
            x.row = L.cells + (q0 - L.off1[0]) + k;
            x.tag = pass_tag(epoch, p);
            x.fail = 0;
            w = x;
        }
        __syncwarp();
        int32_t bv = INT32_MIN, bi = INT32_MAX, bj = INT32_MAX;
        // tables serve rows of A/C/G/T; a pass with another byte compares bytes
        bool dna = SC == SC_TABLE;
        if (SC == SC_TABLE) {
            for (int32_t j = p * kTagPassRows + t; j < min(w.n, (p + 1) * kTagPassRows); j += 32) dna &= dna_valid(w.b_seq[j]);
            dna = __all_sync(0xffffffffu, dna);
        }
#define PA_TAG_PASS(RA)                                                                                  \
    case RA / 2:                                                                                         \
        if (SC != SC_TABLE || dna) tag_pass<LOCAL, SC, RA>(L, P, w, p, t, stage, snap, bv, bi, bj);       \
        else tag_pass<LOCAL, SC == SC_TABLE ? (int)SC_BYTES : SC, RA>(L, P, w, p, t, stage, snap, bv, bi, bj); \
        break
        switch (w.ra / 2) {
            PA_TAG_PASS(4);
            PA_TAG_PASS(8);
            PA_TAG_PASS(12);
            PA_TAG_PASS(16);
        }
#undef PA_TAG_PASS
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const int32_t ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
            const int32_t oj = __shfl_xor_sync(0xffffffffu, bj, o);
            if (tag_better(ov, oi, oj, bv, bi, bj)) { bv = ov; bi = oi; bj = oj; }
        }
        if (t == 0) L.cand[ticket] = make_int4(bv, bi, bj, 0);
        __syncwarp();
    }
}

// One warp per pair: the end cell from the passes' candidates, then the path, up to 32 cells a
// round: the lanes look at the next 32 cells of the diagonal (or of the gap) at once, since a
// chain of one dependent load per cell costs a memory latency each.
template <bool LOCAL>
__global__ void __launch_bounds__(kTagThreads) k_tb_walk(TbLaunch L, DpParams P)
{
    const int lane = threadIdx.x & 31;
    const int fcf = P.first_column_free, frf = P.first_row_free;
    const bool lcf = P.last_column_free, lrf = P.last_row_free;
    if (__ldcg(L.error)) return;                  // directions are missing: the call computes them again
    for (;;) {
        uint32_t u = 0;
        if (lane == 0) u = atomicAdd(L.queue + 1, 1u);
        u = __shfl_sync(0xffffffffu, u, 0);
        if (u >= L.count) break;
        const uint32_t q = L.order[u], k = L.first + q;
        const uint64_t q0 = L.off1[k], r0 = L.off2[k];
        const int32_t m = (int32_t)(L.off1[k + 1] - q0), n = (int32_t)(L.off2[k + 1] - r0);
        const uint8_t *a_seq = L.seq1 + q0, *b_seq = L.seq2 + r0;
        const uint32_t *D = L.dir + L.dir_off[q];
        const int32_t passes = (n + kTagPassRows - 1) / kTagPassRows;
        int32_t bv = INT32_MIN, bi = INT32_MAX, bj = INT32_MAX;
        auto cand = [&](int32_t v, int32_t i, int32_t j) {
            if (tag_better(v, i, j, bv, bi, bj)) { bv = v; bi = i; bj = j; }
        };
        for (uint32_t x = L.start[u] + lane; x < L.start[u + 1]; x += 32) cand(L.cand[x].x, L.cand[x].y, L.cand[x].z);
        if (!LOCAL && lane == 0) {
            if (m == 0 || n == 0) cand(m == 0 ? border(P, frf, n) : border(P, fcf, m), m, n);
            if (lcf) {
                cand(border(P, frf, n), 0, n);
                if (n == 0)
                    for (int32_t i = 1; i <= m; ++i) cand(border(P, fcf, i), i, 0);
            }
            if (lrf) {
                cand(border(P, fcf, m), m, 0);
                if (m == 0)
                    for (int32_t j = 1; j <= n; ++j) cand(border(P, frf, j), 0, j);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const int32_t ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
            const int32_t oj = __shfl_xor_sync(0xffffffffu, bj, o);
            if (tag_better(ov, oi, oj, bv, bi, bj)) { bv = ov; bi = oi; bj = oj; }
        }
        uint8_t *ops = L.ops + (q0 - L.off1[0]) + (r0 - L.off2[0]);
        int32_t score = bv, e1 = bi, e2 = bj;
        if (LOCAL) {
            if (m == 0 || n == 0) { score = INT32_MIN; e1 = e2 = 0; }
            else if (bv <= 0) { score = max(bv, 0); e1 = e2 = 0; }
        }
        int32_t nops = 0, i = 0, j = 0;
        if (!(LOCAL && (m == 0 || n == 0 || score <= 0))) {
            // the nibble of cell (ci, cj)
            auto nib = [&](int32_t ci, int32_t cj) -> uint32_t {
                const int32_t p = (cj - 1) / kTagPassRows, r = (cj - 1) % kTagPassRows;
                const int32_t ra = tag_rows(n, p, passes), t = r / ra, kk = r % ra, wide = ra > 8;
                const uint32_t *W = D + (uint64_t)p * (uint32_t)(m + 31) * 64u;
                const uint32_t word = __ldg(W + ((((int64_t)ci + t - 1) * 32 + t) << wide) + (kk >> 3));
                return word >> (4 * (kk < 8 ? (wide ? kk : kk + 8 - ra) : kk + 8 - ra));
            };
            i = e1;
            j = e2;
            int32_t state = 0;                        // uniform over the warp
            for (;;) {
                if (state == 0) {
                    if (i == 0 || j == 0) {
                        const int32_t left = i == 0 && !frf ? j : j == 0 && !fcf ? i : 0;
                        for (int32_t x = lane; x < left; x += 32) ops[nops + x] = i == 0 ? 'I' : 'D';
                        nops += left;
                        if (left) i = j = 0;
                        break;
                    }
                    const int32_t ci = i - lane, cj = j - lane;
                    const bool in = ci >= 1 && cj >= 1;
                    // 0 Q, 1 P, 2 the diagonal, 3 local start, 4 the border
                    const uint32_t src = in ? (nib(ci, cj) >> 2 & 3u) ^ 1u : 4u;
                    const uint32_t diag = __ballot_sync(0xffffffffu, src == 2u);
                    const int32_t run = diag == 0xffffffffu ? 32 : __ffs(~diag) - 1;
                    if (lane < run) ops[nops + lane] = a_seq[ci - 1] == b_seq[cj - 1] ? '=' : 'X';
                    i -= run;
                    j -= run;
                    nops += run;
                    if (run == 32) continue;
                    const uint32_t next = __shfl_sync(0xffffffffu, src, run);
                    if (next == 3u) break;
                    if (next < 2u) state = next == 1u ? 1 : 2;       // 4: the border, handled above
                } else {
                    // 'D' steps down sequence1 (state 1), 'I' down sequence2: one, and one more
                    // for every following cell whose gap extends
                    const int32_t ci = state == 1 ? i - 1 - lane : i, cj = state == 1 ? j : j - 1 - lane;
                    const bool ext = ci >= 1 && cj >= 1 && !(nib(ci, cj) & (state == 1 ? 1u : 2u));
                    const uint32_t e = __ballot_sync(0xffffffffu, ext);
                    const int32_t more = e == 0xffffffffu ? 32 : __ffs(~e) - 1, steps = min(more + 1, 32);
                    if (lane < steps) ops[nops + lane] = state == 1 ? 'D' : 'I';
                    if (state == 1) i -= steps;
                    else j -= steps;
                    nops += steps;
                    if (more < 32) state = 0;
                }
            }
        }
        __syncwarp();
        for (int32_t x = lane; x < nops / 2; x += 32) {             // path order
            const uint8_t y = ops[x];
            ops[x] = ops[nops - 1 - x];
            ops[nops - 1 - x] = y;
        }
        if (lane == 0) {
            pa_result res;
            res.score = score;
            res.end1 = e1;
            res.end2 = e2;
            res.width = 32;
            res.flags = (m == 0 || n == 0) ? PA_RESULT_TRIVIAL : 0;
            res.band_rounds = 0;
            L.out[k] = res;
            pa_alignment al;
            al.begin1 = i;
            al.begin2 = j;
            al.n_ops = (uint32_t)nops;
            al.reserved = 0;
            L.aln[k] = al;
        }
        __syncwarp();
    }
}

}  // namespace pa
