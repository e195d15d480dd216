// pa_launch.h -- host-side entry points of the DP kernel instantiations.
// Each kernel variant lives in its own translation unit (pa_kern_v*.cu) so that
// the library builds in parallel.
#pragma once
#include "pa_common.cuh"

namespace pa {

// lanes16: s16x2 lanes (else s32); gen: byte-compare scoring; mode: Mode.
// Returns the resident blocks per SM of the selected kernel.
int dp_occupancy(int variant, bool lanes16, bool gen, int mode);
void dp_launch(int variant, bool lanes16, bool gen, int mode, int grid, cudaStream_t stream, const DpLaunch &L,
               const DpParams &P);

// Short-pair kernel (pa_short.cuh) on groups of L.G = 4, 8, 16 or 32 lanes; L.slots must hold seq1_bytes + n_pairs column slots.  s16x2 lanes with unitary DNA scores: form
// 0 (16 rows of sequence2 per thread) or 1 (32 rows).  s32 lanes: scoring is a Scoring (tables,
// raw bytes, or the int8 profile of a substitution matrix of dim symbols), 16 rows.
constexpr int kShortFormCount = 2;
int dp_short_occupancy(int form, int mode);
void dp_short_launch(int form, int mode, int grid, cudaStream_t stream, const DpLaunch &L, const DpParams &P);
int dp_short32_occupancy(int scoring, int mode, int dim);
void dp_short32_launch(int scoring, int mode, int grid, cudaStream_t stream, const DpLaunch &L, const DpParams &P);
inline bool dp_short_supports(int G) { return G == 4 || G == 8 || G == 16 || G == 32; }

// Rows per thread of a unit's full passes.  24 rows spread a column's fixed cost best without
// spilling registers (mixed stream of 32,768 pairs: 113.3 ms; 32 rows, which spill, 116.8; 16
// rows 121.5; 8 rows 159).  A pass is one warp's serial work, so the passes of the longest units
// must not outlast the rest of the queue: rows x columns of a pass stay within the budget that
// k_long_plan sets from the launch's work.  The floor is 4 rows, and 8 in local mode, whose
// columns cost more (90 contig pairs: 5.1 ms with 8 rows, 6.3 with 4; 60 global long reads the
// other way round, 3.2 and 2.7).
constexpr int kLongRows = 24;
// A pair of many more rows than columns is a chain of passes of which few overlap: a pass waits for
// the first 47 columns of the one above, so fewer and higher passes end it sooner.  The floor of such a
// pair grows with the root of rows / columns, where the chain's steps and a pass's own balance: one
// global pair of 100 x 200,000 32.6 ms on passes of 128 rows, 9.3 on 768; 100 of 300 x 8,000 1,106 us
// and 383.
__device__ inline int32_t long_rows(uint32_t budget, int32_t floor_rows, int32_t columns, int32_t rows)
{
    const int32_t c = columns > 0 ? columns : 1;
    const int32_t r = (int32_t)min(budget / (uint32_t)c, (uint32_t)kLongRows) & ~3;
    int32_t f = floor_rows;
    while (f < kLongRows && (int64_t)(f + 4) * (f + 4) * c <= (int64_t)floor_rows * floor_rows * rows) f += 4;
    return r < f ? f : r;
}

// The queue of a launch: unit u's passes are tickets start[u] .. start[u + 1] - 1.
struct LongWords {
    uint32_t tasks;                // tickets
    uint32_t pad;
    uint64_t epoch;                // names the launch in the cell tags
};
struct LongRecord {                // a unit's best candidates between its passes
    int32_t s[2], i[2], j[2];
    int32_t ub[2];                 // band mode: the largest exit bound
    int32_t rpt;                   // rows per thread of a full pass, from k_long_plan (not in band mode)
    int32_t pad;
};
struct LongQueue {
    LongWords *words;
    uint32_t *start;
    uint2 *tasks;                  // band mode: {unit, pass} per ticket
    uint32_t *done;                // passes finished per unit
    uint32_t *fail;                // per unit: a wait ran out
    LongRecord *rec;
    ulonglong2 *cells;             // (seq1_bytes + n_pairs) boundary cells, pair k's at off1[k] + k (DpLaunch::slots)
};

// Long pairs with unitary DNA scores (pa_long.cuh): the row passes of all units in one queue.
int dp_long_occupancy(bool lanes16, int mode);
void dp_long_launch(bool lanes16, int mode, int grid, cudaStream_t stream, const DpLaunch &L, const LongQueue &Q,
                    const DpParams &P);
// The banded DP of long pairs on the same queue: plan and run the list of L.
int dp_long_band_occupancy(bool lanes16);
void dp_long_band_launch(bool lanes16, int grid, cudaStream_t stream, const DpLaunch &L, const LongQueue &Q,
                         const DpParams &P, unsigned long long *epoch);

// CTA mode (long pairs of the byte-compare class): whole blocks per pair; L.ring must hold grid * 8 rows of
// L.ring_stride cells.
int dp_cta_occupancy(int mode);
void dp_cta_launch(int mode, int grid, cudaStream_t stream, const DpLaunch &L, const DpParams &P);
// The same pairs on teams of 4 warps (two units per block, same ring rows as CTA mode).
int dp_team_occupancy(int mode);
void dp_team_launch(int mode, int grid, cudaStream_t stream, const DpLaunch &L, const DpParams &P);

// Cluster mode (the largest of them): clusters of kClusterBlocks blocks per pair; the grid is a
// multiple of the cluster size and L.ring holds grid * 8 rows.
int dp_cluster_grid(int mode, int max_blocks);
cudaError_t dp_cluster_launch(int mode, int grid, cudaStream_t stream, const DpLaunch &L, const DpParams &P);

// Traceback (pa_traceback.cu): one warp per pair, direction words of pair q at dir + dir_off[q],
// passes * (m + 31) * 32 words with passes = ceil(n / kTracebackPassRows).
constexpr int kTracebackPassRows = 256;
struct TbLaunch {
    const uint8_t *seq1, *seq2;
    const uint64_t *off1, *off2;
    uint32_t first, count;          // the chunk: pairs first .. first + count - 1
    const uint64_t *dir_off;        // per chunk pair: first direction word
    uint32_t *dir;
    Cell *bnd;                      // pass boundary: (H(i, last row of the pass), Q(i, next row))
    pa_result *out;
    pa_alignment *aln;
    uint8_t *ops;                   // pair k at (off1[k] - off1[0]) + (off2[k] - off2[0]), m + n bytes
    const int8_t *rank;             // substitution matrix (or null: match / mismatch)
    const int32_t *matrix;
    int32_t dim;
    // tagged kernels: the chunk's pairs largest first, their first tickets (count + 1 words), a
    // candidate per ticket, the queue heads (2 words), boundary cells (cell 0 of pair k at
    // (off1[k] - off1[0]) + k), the launch counter and this launch's number
    const uint32_t *order, *start;
    int4 *cand;
    uint32_t *queue;
    ulonglong2 *cells;
    unsigned long long *epoch, *my_epoch;
    uint32_t *error;
    uint32_t spin_limit;
    int32_t tables;                 // 2 * match + 1 and 2 * mismatch + 1 fit a signed byte
};
int traceback_grid(int sm_count);
void traceback_launch(int grid, cudaStream_t stream, const TbLaunch &L, const DpParams &P);
// The tagged kernels (scores below 2^26): all passes of the chunk in one queue, then the walks.
void traceback_tag_launch(int sm_count, cudaStream_t stream, const TbLaunch &L, const DpParams &P);

}  // namespace pa
