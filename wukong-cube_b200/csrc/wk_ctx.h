// Device context, tables and plan resolution shared by the C-ABI translation units.
#pragma once
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "wk_internal.h"
#include "wk_explore.h"
#include "wk_flat.h"
#include "wk_pipe.h"
#include "wk_kernels.h"
#include "wk_versatile.h"

// A device result table (the reference's rbuf + GPUResult, query.hpp:311-362).
struct wk_table {
    uint32_t* d = nullptr;     // row-major elements
    uint64_t cap = 0;          // elements held
    uint64_t* d_rows = nullptr;// row count, written by the kernels
    int32_t cols = 0;
    // The row count where the host has read it since the last launch that writes the table (every
    // such launch goes through written()), so that it is not read again.
    mutable bool rows_known = false;
    mutable uint64_t rows = 0;
    // A caller's own captured graph writes the table, whenever it is replayed: nothing is kept then.
    bool replayed = false;
    void written() { rows_known = false; }
};

namespace wk {

// Host mirror of SPARQLQuery::Result's column bookkeeping (query.hpp:409-459).
struct ColMap {
    int nvars = 0;
    int col_num = 0;
    std::vector<int32_t> v2c;   // NO_RESULT (0xFFFF) when unbound
    explicit ColMap(int n) : nvars(n), v2c(n > 0 ? n : 0, WK_NO_RESULT) {}
    // 0 = KNOWN, 1 = UNKNOWN, 2 = CONST; -1 = invalid variable id (VERTEX_INVALID)
    int var_stat(int32_t id) const {
        if (id >= 0) return 2;
        int idx = -(id + 1);
        if (idx >= nvars) return -1;
        return v2c[idx] == WK_NO_RESULT ? 1 : 0;
    }
    int col(int32_t id) const { return v2c[-(id + 1)]; }
    void bind(int32_t id, int c) { v2c[-(id + 1)] = c; }
    // bind an unbound variable; false if it is bound already (add_var2col's assertion)
    bool bind_new(int32_t id, int c) {
        if (v2c[-(id + 1)] != WK_NO_RESULT) return false;
        v2c[-(id + 1)] = c;
        return true;
    }
};

// One resolved exploration step of a plan.
//   kIndex index_to_unknown, kConst const_to_unknown, kK2U / kK2K / kK2C known_to_*,
//   kC2K const_to_known, kI2K index_to_known (single steps only: a query starts unbound),
//   kCUU / kCUC / kKUU / kKUC the unknown-predicate (versatile) operators.
struct PlanStep {
    enum Kind { kIndex, kConst, kK2U, kK2K, kK2C, kC2K, kI2K, kCUU, kCUC, kKUU, kKUC } kind;
    uint32_t pid = 0;
    int32_t dir = 0;
    uint32_t start_const = 0;   // kIndex: tpid; kConst: start vertex
    int32_t cs = 0, ce = 0;     // input columns
    uint32_t end_const = 0;     // kK2C, kKUC, kCUC
    int32_t in_cols = 0, out_cols = 0;
    int32_t mt_tid = 0, mt_factor = 1;   // kI2K: the slice of the index list
};

// Resolve a planned pattern list into steps, as SPARQLEngine::execute_one_pattern dispatches
// (sparql.hpp:932-1055; the GPU engine's gpu_engine.hpp:265-338 is its subset).  With
// `versatile` (the store holds the vertex-predicate lists) an unknown predicate goes to the
// versatile operators, else it is WK_UNKNOWN_PATTERN.  Returns a WK_* status; fills v2c_map /
// col_num of the result.
int resolve_plan(const wk_query& q, int max_cols, std::vector<PlanStep>& steps, ColMap& cm,
                 bool versatile = false);
inline bool is_versatile_step(int kind) {
    return kind == PlanStep::kCUU || kind == PlanStep::kCUC || kind == PlanStep::kKUU || kind == PlanStep::kKUC;
}

}  // namespace wk

struct wk_ctx {
    std::mutex mu;
    wk_config cfg{};
    int device = 0;
    int sm_count = 148;
    cudaStream_t stream = nullptr;

    // resident store
    wk::Slot* d_slots = nullptr;
    uint64_t n_slots = 0;
    uint32_t* d_edges = nullptr;
    uint64_t n_edges = 0;
    std::vector<wk_seg_meta> segs;
    wk::SegIndex index;
    std::vector<wk::SegDesc> seg_desc;   // of each segment, with its directory
    std::vector<uint32_t> seg_longest;   // entries of each segment's longest list
    bool zero_ids = false;               // a list of the store holds id 0 (see step_gives_one)
    wk::SegDesc* d_segs = nullptr;       // DevStore::segs: an absent segment, then seg_desc
    wk::DirBlock* d_dir_blocks = nullptr;   // vertex directories (wk_dir.cu)
    void* d_dir_words = nullptr;
    size_t dir_bytes = 0;
    bool has_dir = false;                // some segment has a directory
    bool serving = false;                // a serving run is on: its lanes read the store as it is
    uint64_t store_gen = 0;              // stores this context has held (captured launches hold
                                         // the addresses of theirs)
    bool has_store = false;
    bool versatile = false;           // the store holds the vertex-predicate lists
    wk::PredSeg* d_pseg = nullptr;    // predicate segments by pid * 2 + dir (versatile steps)
    uint32_t n_pseg = 0;
    struct IndexList {
        uint64_t ptr;    // pointer word
        bool probed;     // a probe of the key ends at it (else the word is only good for an estimate)
    };
    std::map<uint32_t, IndexList> index_ptr;   // tpid * 2 + dir -> its index list
    uint64_t* d_inline_orig = nullptr;   // (slot index, original pointer word) of every slot
    uint64_t n_inline = 0;               // whose one-entry list is kept in the slot itself
    bool borrowed_store = false;   // a serving lane: the store belongs to its parent context
    wk::CtaUse beside_use{0, 0, 0};   // a serving lane leaves room on every SM for this many
    int beside_ctas = 0;              // resident CTAs of this size (the iteration launches)
    int sorted_lists = 0;
    int default_lanes = 2;
    int batch_lanes = 4;
    std::map<int, int> tuned_lanes;
    uint64_t spin_limit = 0;         // polls of a bounded wait on another CTA (0: the default)
    uint32_t slice_rows = 0;         // list length above which rows go to the slice queue
    uint32_t batch_slice_rows = 0;   // (0: the kernel's default, kHeavyRows)
    int32_t batch_flat = 0;          // bit k: batch level k runs as the flat passes, not tiles
    // single steps with at least this many input rows, and whole plans, run as fused passes (0: never)
    uint64_t flat_min_rows = 65536;
    void* d_flat = nullptr;          // its scratch (wk_flat.h)
    uint64_t flat_cap_rows = 0;
    void* d_final_scratch = nullptr;   // scratch of the post-pattern stage and the BOUND filter
    size_t final_scratch_bytes = 0;

    // scan control of the context stream
    wk::StepCtl* d_ctl = nullptr;
    wk::HeavyItem* d_heavy = nullptr;    // long-list slices of the context stream
    uint64_t heavy_cap = 0;
    unsigned long long* d_status = nullptr;
    uint64_t status_cap = 0;
    wk::StepCtl* h_ctl = nullptr;     // pinned; as d_ctl it is followed by the row counts of rbuf
    uint32_t* h_small = nullptr;      // pinned: the first elements of a query's table, which come
    uint64_t small_elems = 0;         // with its control block (how many the last query brought)
    uint64_t* h_rows = nullptr;       // pinned
    uint32_t inject_err = 0;          // error bits the next control-block read reports (tests)

    // ping-pong result buffers for whole queries (GPUMem rbuf pair, gpu_mem.hpp:53-60)
    wk_table rbuf[2];

    // CUDA graphs of resident query plans
    struct GraphEntry {
        cudaGraphExec_t exec = nullptr;
    };
    std::map<std::string, GraphEntry> graphs;

    std::map<long long, int> bps_cache;   // (op, cols) -> blocks per SM
    std::string last_error;

    // batch / serving state (wk_batch.cu); batch2 is the second state of the pipelined path
    void* batch = nullptr;
    void* batch2 = nullptr;
    void* batch_host = nullptr;   // plans, streams and events reused by every batch call
    void* serve = nullptr;        // buffers kept between serving runs (wk_serve.cu)
    // serving lanes, kept between serving runs so their tables stay grown (wk_serve.cu)
    std::vector<wk_ctx*> lanes;
    wk::CtaUse lanes_use{0, 0, 0};
    int lanes_ctas = 0;

    wk::DevStore dev_store() const {
        wk::DevStore s;
        s.slots = d_slots;
        s.n_buckets = n_slots / wk::kAssoc;
        s.edges = d_edges;
        s.n_edges = n_edges;
        s.segs = d_segs;
        return s;
    }
    wk::SegDesc seg_of(uint64_t vid, uint32_t pid, int dir) const {
        const uint32_t i = seg_id(vid, pid, dir);
        return i ? seg_desc[i - 1] : wk::SegDesc{};
    }
    // its entry in DevStore::segs (0: absent)
    uint32_t seg_id(uint64_t vid, uint32_t pid, int dir) const {
        const int32_t i = index.find(vid, pid, dir);
        return i >= 0 && pid < (1u << wk::kNbitsIdx) ? (uint32_t)i + 1 : 0;
    }
    int fail(int code, const std::string& msg) {
        last_error = msg;
        return code;
    }
    int cuda_fail(cudaError_t e, const char* what) {
        last_error = std::string(what) + ": " + cudaGetErrorString(e);
        return WK_E_CUDA;
    }
    int blocks_per_sm(int op, int cols, int lanes);
    // Lanes per probe group of a launch that asks for `lanes`: a store with vertex directories is
    // looked up by one thread per row (a directory lookup is one block and one word, so a group
    // has nothing to share); the group widths serve stores without.
    int probe_lanes(int lanes) const { return has_dir ? 1 : lanes; }
    // lanes per probe group for (op, cols): the tuned choice, else 2 (one 32-byte sector)
    int lanes_for(int op, int cols) const {
        auto it = tuned_lanes.find(op * 1000 + cols);
        return probe_lanes(it != tuned_lanes.end() ? it->second : default_lanes);
    }
    void drop_graphs();
    int ensure_status(uint64_t tiles);
    int ensure_heavy(uint64_t out_rows_cap);
    int ensure_flat(uint64_t in_rows_cap);
    // Free the store (`spare`: its slots and edges kept aside for the build that follows, when the
    // device has plenty of room).
    void drop_store(bool spare = false);
    void drop_spare();
    // Give the vertex directories back to an allocation of `bytes` (lookups go by hash from then on);
    // false where it would not fit all the same, or something running or captured may still read them.
    bool drop_directories(size_t bytes);
    struct Spare {
        void* p = nullptr;
        size_t bytes = 0;
    };
    Spare spare_slots, spare_edges;
    size_t slots_bytes = 0, edges_bytes = 0;   // what d_slots and d_edges were allocated with
    // A store array: the spare one where it is large enough (and at most twice as large).
    template <class T>
    cudaError_t store_malloc(Spare& sp, T** p, size_t bytes);
    int final_scratch_reserve(size_t bytes);
    int table_reserve(wk_table* t, uint64_t elems);
    int read_ctl(uint32_t* err, uint64_t* need, const wk_table* t = nullptr);
    void release_serve();
    int clear_ctl_err();
};

namespace wk {
// Device block of a context's control words: StepCtl, then the row counts of rbuf[0] and rbuf[1], so
// that one copy brings all of them.
constexpr size_t kCtlBlockBytes = sizeof(StepCtl) + 2 * sizeof(uint64_t);
constexpr uint64_t kSmallElems = 4096;
// dev_malloc that gives back what the context only keeps to be faster, and tries again, when the
// device is full: the kept serving buffers, then the vertex directories.
template <class T>
cudaError_t ctx_malloc(wk_ctx* ctx, T** p, size_t bytes) {
    cudaError_t e = dev_malloc(p, bytes);
    if (e != cudaSuccess && ctx->serve) {
        cudaGetLastError();
        ctx->release_serve();
        e = dev_malloc(p, bytes);
    }
    if (e != cudaSuccess && ctx->has_dir) {
        cudaGetLastError();
        if (ctx->drop_directories(bytes)) e = dev_malloc(p, bytes);
    }
    return e;
}
}  // namespace wk

template <class T>
cudaError_t wk_ctx::store_malloc(Spare& sp, T** p, size_t bytes) {
    const size_t have = sp.bytes;
    if (sp.p && have >= bytes && have / 2 <= bytes) {
        *p = static_cast<T*>(sp.p);
        sp = Spare{};
        (&sp == &spare_slots ? slots_bytes : edges_bytes) = have;
        return cudaSuccess;
    }
    drop_spare();
    (&sp == &spare_slots ? slots_bytes : edges_bytes) = bytes;
    return wk::ctx_malloc(this, p, bytes);
}

namespace wk {
// Enqueue one resolved step reading `in` (may be null for index/const starts) into `out`: a
// start or versatile step by its own launch, a known_to_* step by the tile launch.
int enqueue_step(wk_ctx* ctx, const PlanStep& st, const wk_table* in, wk_table* out,
                 int32_t mt_tid, int32_t mt_factor, cudaStream_t s);
// Consecutive steps [first, first + n) of a plan that run as one launch: a fused pass
// (wk_pipe.cu), or (pipe false) one step by enqueue_step.
struct PlanPass {
    int first, n;
    bool pipe;
};
// Whether a step of a plan gives each row at most one output row: a filter, or known_to_unknown on a
// predicate whose lists all have at most one entry.  A row's vertex comes from the store's lists; where
// one of those holds id 0, which names the predicate's index list, that list counts among them.
bool step_gives_one(const wk_ctx* ctx, const PlanStep& s);
// The passes of a plan.
std::vector<PlanPass> plan_passes(const wk_ctx* ctx, const std::vector<PlanStep>& steps);
// Enqueue one pass reading `in` (null when it starts the plan) into `out`.  `fuse` false: every
// known_to_unknown step multiplies rows (a single step over a caller's table with vertex 0 in it);
// `account`: the steps' bytes and list entries are added to the control block (a profile).
int enqueue_pass(wk_ctx* ctx, const std::vector<PlanStep>& steps, const PlanPass& p, const wk_table* in, wk_table* out,
                 int32_t mt_tid, int32_t mt_factor, bool fuse, cudaStream_t s, bool account = false);
// The device descriptor of a resolved step.
StepDesc make_step_desc(const wk_ctx* ctx, const PlanStep& s);

// A context on its own (lowest-priority) stream with its own control block, status array,
// slice queue and tables, reading the parent's resident store; its exploration launches
// leave room on every SM for `beside_ctas` CTAs of size `beside_use`.  Released with
// wk_ctx_destroy, before the parent.
int ctx_make_child(wk_ctx* parent, const CtaUse& beside_use, int beside_ctas, wk_ctx** out);
// Run a whole query (mode: WK_MODE_RESIDENT or WK_MODE_GRAPH) and report its final table and row
// count (host sync).
int query_run_rows(wk_ctx* ctx, const wk_query* q, int32_t mode, const wk_table** t, uint64_t* rows);
// A table's row count (host sync, unless the host knows it already).
int table_rows(wk_ctx* ctx, const wk_table* t, uint64_t* rows);
// Copy `elems` elements of a device table to host memory (host sync).
int table_copy_out(wk_ctx* ctx, const wk_table* t, uint64_t elems, uint32_t* host);
// Size a serving lane's tables and scan scratch for `elems`-element tables up front.
int lane_prepare(wk_ctx* lane, uint64_t elems);
// Make device arrays (dev_malloc'd) the context's store; the context owns them from here on.
int store_adopt(wk_ctx* ctx, Slot* d_slots, uint64_t n_slots, uint32_t* d_edges, uint64_t n_edges,
                const std::vector<wk_seg_meta>& segs);
cudaError_t gbuild_kernel_attrs();   // wk_gbuild.cu
// Lanes for one (explore op, input columns) step of single queries (the autotuner's choice).
int tune_step_lanes(wk_ctx* ctx, int op, int cols, int lanes);
}  // namespace wk
