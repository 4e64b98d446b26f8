// Host-visible interface of the fused levels of a batch (wk_level.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "wk_explore.h"

namespace wk {

// What one query does at one level: n_ops steps that give a row at most one output row each (a
// filter, or known_to_unknown on a functional predicate), then optionally one step that multiplies
// rows (or, at level 0, starts them).
struct LevelRun {
    uint32_t first;    // its first step in LevelArgs::steps
    uint8_t n_ops;
    uint8_t flags;     // kRunLast, kRunFinal
    uint8_t cin;       // columns of its rows on entry
    uint8_t pad;
};
enum : uint8_t {
    kRunLast = 1,      // step first + n_ops multiplies the rows
    kRunFinal = 2,     // the query's result is this level's output
};
static_assert(sizeof(LevelRun) == 8, "a run is one 8-byte word");

constexpr int kMaxLevelCols = 3;   // columns a level appends before its last step

struct LevelArgs {
    DevStore store;
    uint32_t n_segs;
    uint32_t seg_index[2];
    const StepDesc* steps;
    const LevelRun* runs;        // [n_queries]
    uint32_t n_queries;
    int32_t virtual_rows;        // row r is query r's start (no input table)
    const uint64_t* in_rows;
    const uint32_t* owner_in;
    const uint32_t* in;
    int32_t w_in;
    uint64_t in_cap_rows;
    uint32_t* out;
    int32_t w_out;
    uint64_t out_cap_rows;
    uint64_t* out_rows;
    uint32_t* owner_out;
    unsigned long long* qfirst;  // [n_queries] of the queries whose result this level holds
    unsigned long long* qcount;
    HeavyItem* heavy;
    uint64_t heavy_cap;
    StepCtl* ctl;
    unsigned long long* status;
    int32_t sorted_lists;
    int32_t account;             // add the steps' bytes and list entries to ctl (a profile)
    uint32_t slice_rows;
    uint64_t spin_limit;
};

int level_grid(int sm_count);
cudaError_t launch_level(const LevelArgs& a, int grid, cudaStream_t s);
cudaError_t level_kernel_attrs();

}  // namespace wk
