// Interface of the backward on sorted points (msda_sorted.cu) towards the C ABI.
#pragma once

#include <algorithm>
#include <type_traits>

#include "msda_common.cuh"

namespace msda_b200 {

constexpr int kCols = 7;   // pixel columns (of the top left corner) of a cell

constexpr int kRunKinds = 4;

// Runs of one length: `each` in every plane from plane0 on, of 2^log2_size units, the first at unit0.
struct WalkRuns {
    unsigned run0, plane0, each, unit0;
    int log2_size;
};

// Layout of the workspace and shape of the launches for the samples of one pass.
struct SortPlan {
    unsigned *header;        // magnitude cells (as in the scaled float16 scratch)
    unsigned *tickets;       // per plane: CTAs of the counting kernel that have finished
    unsigned *counts;        // per plane and cell: points, later the next free place
    unsigned *offsets;       // per plane and cell: first place
    int *item_cell;          // per plane and unit of item_points places: the cell it begins in
    uint4 *records;          // per plane: the points in order of their cells
    float *grad_prob;        // gradient of every weight (softmax: of the probability), float32
    float2 *stats;           // softmax only: (max, 1 / sum) of every pair's logits
    int64_t plane_points;    // Q * L * K
    int64_t cell_stride;     // elements between planes in counts / offsets
    size_t cleared_bytes;    // header, tickets and counts, to be zero at the start
    int cell_bound;          // cells a plane has room for
    int shared_cells;        // cells a scatter CTA has room for in shared memory
    int count_cells;         // the same of the counting kernel
    int chunk_queries, chunks;             // queries of a scatter CTA, such stretches of a sample
    bool scatter_by_level;                 // a turn of the scatter takes one level:
    int level_queries, level_stretches;    // its queries, such stretches of a sample,
    unsigned level_turns;                  // its turns,
    int level_cells;                       // cells it has room for
    bool count_by_level;                   // CTAs of the counting kernel take one level
    int count_queries, count_stretches;    // the same of the counting kernel
    int count_ctas;                        // its CTAs per plane
    int prepare_ctas;        // CTAs of the counting kernel that prepare instead
    int item_points, items;  // places of a unit, units of a plane
    WalkRuns runs[kRunKinds];   // by the order they are handed out in
    unsigned all_runs;
};

// Whether a call is dense enough for the sort to pay (and within the record's field widths).
// `offsets`: the call takes reference points and offsets.
bool sorting_pays(const Params &p, int dtype, bool offsets);
// Fills the plan for `samples` samples over `workspace`; returns the bytes it takes.
int64_t plan_sorted(SortPlan &sp, const Params &p, bool softmax, int64_t samples, void *workspace);
// The call restricted to samples b .. b + n - 1.
Params samples_of(const Params &p, int64_t b, int64_t n);
int64_t sorted_workspace_bytes(const Params &p, bool softmax, int64_t samples);
// Samples that sort together in a workspace of `bytes`; 0 if it is too small to be worth it.
int64_t sorted_samples_per_turn(const Params &p, bool softmax, int64_t bytes);
cudaError_t launch_backward_sorted(const Params &p, const SortPlan &sp, int dtype, bool softmax,
                                   cudaStream_t stream);

}  // namespace msda_b200
