// Host-visible interface of the fused single-query passes (wk_pipe.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "wk_explore.h"

namespace wk {

// One step of a pass that gives each row at most one output row: a filter, or a
// known_to_unknown step on a functional predicate (every list of its segment has one entry),
// which appends its neighbour as a column.
struct PipeOp {
    uint64_t start_key;      // const_to_known / index_to_known: the key of the one list
    SegDesc seg;
    uint32_t pid;
    uint32_t end_const;      // kXK2C
    uint32_t mt;             // kXI2K
    uint8_t op, dir, cs, ce; // ExploreOp; columns of the row as it is at this step
    uint8_t type_index;      // the last step: get_index lists (TYPE_ID, IN)
    uint8_t pad[3];
};

constexpr int kMaxPipeOps = 6;
constexpr int kMaxPipeCols = 3;   // columns a pass appends before its last step

// A pass: its rows (a table's, or the entries of one list), the steps above, and optionally one
// known_to_unknown step on any predicate, whose neighbours multiply the rows.
struct PipeArgs {
    DevStore store;
    uint32_t seg_index[2];
    int32_t from_list;           // rows are the list of src_key (its mt slice), one column
    int32_t src_known;           // the list is edges[src_off, src_off + src_len); else it is looked up
    uint64_t src_off, src_len;
    uint64_t src_key;
    SegDesc src_seg;
    int32_t mt_tid, mt_factor;
    const uint64_t* in_rows;     // else: a table
    const uint32_t* in;
    int32_t w_in;                // its columns (1 for a list)
    uint64_t in_cap_rows;
    int32_t n_ops;
    int32_t has_last;
    PipeOp ops[kMaxPipeOps];
    PipeOp last;
    uint32_t* out;
    int32_t w_out;
    uint64_t out_cap_rows;
    uint64_t* out_rows;
    HeavyItem* heavy;
    uint64_t heavy_cap;
    StepCtl* ctl;
    unsigned long long* status;
    int32_t sorted_lists;
    int32_t account;             // add the steps' bytes and list entries to ctl (a profile)
    uint32_t slice_rows;         // as ExploreArgs
    uint64_t spin_limit;
};

constexpr int kPipeMaxTileRows = 16384;   // rows of the largest chunk (one status word each)
int pipe_grid(int sm_count);
// The grid of a serving lane's passes, beside other_ctas CTAs of shape `other` on every SM.
int pipe_grid_beside(int sm_count, const CtaUse& other, int other_ctas);
cudaError_t launch_pipe(const PipeArgs& a, int grid, cudaStream_t s);
cudaError_t pipe_kernel_attrs();

}  // namespace wk
