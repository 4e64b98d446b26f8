// Fused levels of a batch: every query's next run of steps in one launch.
//
// All queries of a batch advance together, their rows tagged with their owner query, contiguous
// and in query order.  A launch per pattern moved every row through memory once per pattern and
// paid a look-back per 64 to 256 rows; here a row runs as many of its query's steps as give it at
// most one output row (filters, known_to_unknown on functional predicates) and then one step that
// multiplies rows, and only the outcome is written.  A batch of 2- to 6-pattern queries takes three
// or four levels instead of six.
//
// A launch is shaped like the fused pass of a single query (wk_pipe.cu): CTAs claim chunks of
// consecutive rows (1,024 on a large level, fewer as long as there is a CTA for more), count, take a
// decoupled look-back, and write what they counted, short lists through shared memory.  One row per
// thread: rows of different queries run different steps, and a warp's 32 rows mostly belong to one or
// two queries.  Rows whose lists are longer than the slice threshold go to the slice queue that CTAs
// without work drain (128 entries unless knob 3 says otherwise; 64 took the same time).
//
// What bounds it: a chunk waits for the counts of the chunks before it (11 us of a chunk's 40 on the
// last level of 16,384 light queries over 2,000 organisations), and the chain of a row's dependent
// reads; issue is a quarter used, DRAM less than a tenth.  Levels of that batch, us: 37 + 125 + 173 + 147, against 46
// + 123 + 105 + 114 + 82 + 66 for a launch per pattern; 64 queries 88 against 145.  Measured without
// gain: two or four rows per thread where a warp's rows are one query's, chunks of 256 or 512 rows
// (191 and 152 against 147 on the last level), three or five CTAs per SM, descriptors a step ahead.
#include <cuda_runtime.h>

#include <algorithm>

#include "wk_device.cuh"
#include "wk_level.h"

namespace wk {
namespace {
using namespace dev;

constexpr int kLevThreads = 256;
constexpr int kLevWarps = kLevThreads / 32;
constexpr int kLevCtas = 4;           // CTAs per SM: 64 registers a thread
constexpr int kGroups = 4;            // 32-row groups of a warp's chunk at most
constexpr int kStageWords = 512;      // output words staged per warp
constexpr int kStageRows = 128;       // and their rows' owners
constexpr uint32_t kLaneList = 16;    // a warp with no longer list writes a row's outputs by its lane

// The directory half of a SegDesc; segments past kSmemSegs are read where they are.
struct SegDir {
    const uint2* dir;
    const void* words;
    uint32_t vid_lo, vid_span, values, pad;
};
static_assert(sizeof(SegDir) == 32, "the first half of a SegDesc");
constexpr uint32_t kSmemSegs = 64;


// Shared memory of a CTA.
struct LevelSmem {
    uint64_t off[kGroups][kLevThreads];                  // the rows' lists
    uint32_t cnt[kGroups][kLevThreads];                  // and output rows
    uint32_t app[kGroups][kMaxLevelCols][kLevThreads];   // columns the level appended
    uint32_t stage[kLevWarps][kStageWords];
    uint32_t owner[kLevWarps][kStageRows];
    SegDir segs[kSmemSegs];   // an L2 round trip per step less (L1 is what shared memory leaves)
};

// A step's descriptor in registers.
struct Step {
    uint64_t start_key;
    uint32_t seg, pid, end_const, mt;
    uint32_t op, dir, cs, ce, type_index;
};
__device__ __forceinline__ Step load_step(const StepDesc* p) {
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(p)), b = __ldg(reinterpret_cast<const uint4*>(p) + 1);
    Step s;
    s.start_key = (uint64_t)a.y << 32 | a.x;
    s.seg = a.z;
    s.pid = a.w;
    s.end_const = b.x;
    s.op = b.y & 0xFF;
    s.dir = b.y >> 8 & 0xFF;
    s.cs = b.z & 0xFF;
    s.ce = b.z >> 8 & 0xFF;
    s.type_index = b.z >> 16 & 0xFF;
    s.mt = b.w;
    return s;
}

// Pointer word of a key by hash, out of line.
__device__ __noinline__ uint64_t level_slow(const Slot* slots, uint64_t n_buckets, const SegDesc* sg, uint64_t key,
                                            unsigned* err) {
    if (sg->num_buckets == 0 || key == 0) return 0;
    return hash_lookup(slots, n_buckets, sg->bucket_start, sg->num_buckets, sg->magic, key, err);
}

// List of a step for start vertex `cur` (ignored where the step names its key itself); an entry kept
// in the directory or the slot comes as a tagged offset.
__device__ __forceinline__ void step_list(const LevelArgs& a, const SegDir* segs, const Step& s, uint32_t cur,
                                          uint64_t* off, uint64_t* deg) {
    const bool own_key = s.op == kXStart || s.op == kXC2K || s.op == kXI2K;
    if (own_key) cur = (uint32_t)key_vid(s.start_key);
    const SegDir sd = s.seg < kSmemSegs ? segs[s.seg] : *reinterpret_cast<const SegDir*>(a.store.segs + s.seg);
    uint64_t p = 0;
    if (sd.vid_span && cur != 0 && !s.type_index) {
        const uint32_t i = cur - sd.vid_lo;
        if (i < sd.vid_span) {
            const uint2 b = __ldg(sd.dir + (i >> 5));
            if (dir_has(b, i)) {
                const uint32_t at = dir_place(b, i);
                if (sd.values) {   // every list has one entry and the directory holds it
                    *off = kInlineTag | __ldg(static_cast<const uint32_t*>(sd.words) + at);
                    *deg = 1;
                    return;
                }
                p = __ldg(static_cast<const unsigned long long*>(sd.words) + at);
            }
        }
    } else {
        const SegDesc* sg = a.store.segs + s.seg;
        uint64_t key = s.start_key;
        if (!own_key) {
            // get_index(cur, IN) (sparql.hpp:342-345), only 17-bit ids can be keys; vid 0 names the
            // index of the predicate
            key = s.type_index ? make_key(0, cur, kIn) : make_key(cur, s.pid, s.dir);
            if (s.type_index) sg = a.store.segs + a.seg_index[kIn];
            else if (cur == 0) sg = a.store.segs + (s.dir & 1 ? a.seg_index[1] : a.seg_index[0]);
            if (s.type_index && cur >= (1u << kNbitsIdx)) key = 0;
        }
        p = level_slow(a.store.slots, a.store.n_buckets, sg, key, &a.ctl->err);
    }
    list_of_ptr(p, a.store.n_edges, &a.ctl->err, off, deg);
}

struct LevelAcc {
    unsigned long long alg, sd;
};

// One row through its query's run: its output rows, the list of its last step and the columns it
// appended (app[j * kLevThreads]).
__device__ __forceinline__ uint32_t level_row(const LevelArgs& a, const SegDir* segs, const LevelRun& run,
                                              const uint32_t* row, uint32_t* app, uint64_t* off, LevelAcc* acc) {
    const StepDesc* steps = a.steps + run.first;
    int w = run.cin;
    const int n = run.n_ops + (run.flags & kRunLast ? 1 : 0);
    *off = 0;
    uint32_t cnt = n ? 1 : 0;   // (a finished query's rows go no further)
#pragma unroll 1
    for (int i = 0; i < n && cnt; ++i) {
        const Step s = load_step(steps + i);
        const bool last = i == run.n_ops;
        auto col = [&](int c) { return c < run.cin ? __ldg(row + c) : app[(c - run.cin) * kLevThreads]; };
        uint32_t cur = 0, target = s.end_const;
        if (s.op == kXC2K || s.op == kXI2K) {
            target = col(s.ce);
        } else if (s.op != kXStart) {
            cur = col(s.cs);
            if (s.op == kXK2K) target = col(s.ce);
            if (cur == kBlankId) {
                cnt = 0;
                break;
            }
        }
        uint64_t deg;
        step_list(a, segs, s, cur, off, &deg);
        if (s.op == kXI2K) {   // index_to_known reads its mt slice of the list
            uint64_t lo, hi;
            mt_slice(s.mt, deg, &lo, &hi);
            *off += lo;
            deg = hi - lo;
        }
        if (acc) {
            acc->sd += deg;
            acc->alg += (s.op == kXStart ? 0 : w * 4) + 16 + deg * 4;
        }
        if (last) {
            cnt = (uint32_t)deg;
            ++w;
        } else if (s.op == kXK2U) {
            cnt = deg ? 1 : 0;
            if (deg) app[(w - run.cin) * kLevThreads] = list_at(a.store.edges, *off, 0);
            ++w;
        } else {
            cnt = deg && thread_member(a.store.edges, *off, deg, target, a.sorted_lists != 0) ? 1 : 0;
        }
        if (acc) acc->alg += (unsigned long long)cnt * w * 4;
    }
    return cnt;
}

__device__ __forceinline__ LevelRun load_run(const LevelArgs& a, uint32_t q) {
    const uint2 x = __ldg(reinterpret_cast<const uint2*>(a.runs) + q);
    LevelRun r;
    r.first = x.x;
    r.n_ops = x.y & 0xFF;
    r.flags = x.y >> 8 & 0xFF;
    r.cin = x.y >> 16 & 0xFF;
    return r;
}

__global__ void __launch_bounds__(kLevThreads, kLevCtas) level_kernel(const __grid_constant__ LevelArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    LevelSmem& S = *reinterpret_cast<LevelSmem*>(smem_raw);
    __shared__ uint64_t s_warp[kLevWarps];
    __shared__ unsigned long long s_claim, s_excl;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned epoch = *(volatile unsigned*)&a.ctl->epoch;
    uint64_t R = a.virtual_rows ? a.n_queries : *(volatile const uint64_t*)a.in_rows;
    if (!a.virtual_rows && R > a.in_cap_rows) R = 0;   // past capacity: the level before overflowed
    // rows of a warp: 32, up to kGroups times that as long as every CTA has a chunk; the starts, which
    // multiply at once, are spread thinner (64 starts: 25 -> 19 us; a level of 15,000 rows spread the
    // same way went from 21 to 32, more CTAs waiting on one another for less work each)
    const uint64_t share = (R + (uint64_t)gridDim.x * kLevWarps - 1) / ((uint64_t)gridDim.x * kLevWarps);
    const uint32_t per = a.virtual_rows ? (uint32_t)min((unsigned long long)32, (unsigned long long)share) : 32;
    const int groups = share <= 32 ? 1 : (int)min((unsigned long long)kGroups, (unsigned long long)((share + 31) / 32));
    const uint32_t warp_rows = per * groups, tile_rows = warp_rows * kLevWarps;
    uint64_t ntiles = R ? (R + tile_rows - 1) / tile_rows : 0;
    if (ntiles > a.ctl->status_cap) {
        if (threadIdx.x == 0) atomicOr(&a.ctl->err, kErrStatus);
        ntiles = 0;
    }
    if (ntiles == 0 && blockIdx.x == 0 && threadIdx.x == 0) *a.out_rows = 0;
    // no chunk for this CTA: it leaves, and the others count without it
    const unsigned active = (unsigned)min((unsigned long long)gridDim.x, (unsigned long long)ntiles);
    if (blockIdx.x >= active) return;
    const uint32_t thr = a.slice_rows ? min(max(a.slice_rows, (uint32_t)kMinSliceRows), 1u << 23) : (uint32_t)kHeavyRows;
    const unsigned long long spin = a.spin_limit ? a.spin_limit : kDefaultSpinLimit;
    const int wo = a.w_out;
    uint32_t* const stage = S.stage[warp];
    uint32_t* const owners = S.owner[warp];
    LevelAcc sums{0, 0};
    uint32_t done = 0;   // chunks this CTA has written
    for (uint32_t i = threadIdx.x; i < 2 * min(kSmemSegs, a.n_segs + 1); i += kLevThreads)
        reinterpret_cast<uint4*>(S.segs)[i] = __ldg(reinterpret_cast<const uint4*>(a.store.segs + i / 2) + i % 2);
    if (threadIdx.x == 0) s_claim = atomicAdd(&a.ctl->tile_counter, 1ull);
    __syncthreads();
    for (uint64_t tile = s_claim; tile < ntiles; ++done) {
        const uint64_t w0 = tile * tile_rows + (uint64_t)warp * warp_rows + lane;   // the warp's rows
        uint64_t total = 0, o0 = 0;   // output rows of the warp, and its next one
        // t < 0 counts group t + groups, t >= 0 writes group t (one body for both); the look-back
        // lies between
#pragma unroll 1
        for (int t = -groups; t < groups; ++t) {
            if (t == 0) {
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) total += __shfl_xor_sync(kFull, total, d);
                if (lane == 0) s_warp[warp] = total;
                __syncthreads();
                uint64_t before = 0, all = 0;
#pragma unroll
                for (int w = 0; w < kLevWarps; ++w) {
                    if (w < warp) before += s_warp[w];
                    all += s_warp[w];
                }
                if (warp == 0) {
                    if (lane == 0) publish_aggregate(a.status, tile, all, epoch);
                    __syncwarp();
                    const uint64_t ex = resolve_prefix(a.status, a.ctl, tile, all, epoch, spin);
                    if (lane == 0) s_excl = ex;
                }
                __syncthreads();
                const uint64_t excl = s_excl;
                o0 = excl + before;
                if (tile == ntiles - 1 && threadIdx.x == 0) *a.out_rows = excl + all;
                if (excl + all > a.out_cap_rows) {
                    if (threadIdx.x == 0) {
                        atomicOr(&a.ctl->err, kErrOverflow);
                        atomicMax(&a.ctl->need, (unsigned long long)(excl + all));
                    }
                    break;
                }
                if (!total) break;
            }
            const bool count = t < 0;
            const int g = count ? t + groups : t;
            const uint64_t r = w0 + 32 * g;
            const bool live = r < R && lane < per;
            const uint32_t* row = a.in + r * (uint64_t)a.w_in;
            uint32_t q = 0xFFFFFFFFu;
            LevelRun run{0, 0, 0, 0, 0};
            if (live) {
                q = a.virtual_rows ? (uint32_t)r : __ldg(a.owner_in + r);
                run = load_run(a, q);
            }
            uint32_t* app = &S.app[g][0][threadIdx.x];
            if (count) {
                uint64_t off = 0;
                const uint32_t cnt = live ? level_row(a, S.segs, run, row, app, &off, a.account ? &sums : nullptr) : 0;
                S.off[g][threadIdx.x] = off;
                S.cnt[g][threadIdx.x] = cnt;
                total += cnt;
                continue;
            }
            const uint32_t cnt = S.cnt[g][threadIdx.x];
            const uint64_t off = S.off[g][threadIdx.x];
            uint64_t st = cnt;   // output rows before the lane's
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint64_t y = __shfl_up_sync(kFull, st, d);
                if (lane >= d) st += y;
            }
            const uint64_t n_all = __shfl_sync(kFull, st, 31);
            if (!n_all) continue;
            // the ranges of the queries whose result this is: (end - start) of every run of rows
            {
                const uint32_t qp = __shfl_up_sync(kFull, q, 1), qn = __shfl_down_sync(kFull, q, 1);
                if (live && (run.flags & kRunFinal)) {
                    if (lane == 0 || qp != q) {
                        atomicMin(a.qfirst + q, (unsigned long long)(o0 + st - cnt));
                        atomicAdd(a.qcount + q, (unsigned long long)(0 - (o0 + st - cnt)));
                    }
                    if (lane == 31 || qn != q) atomicAdd(a.qcount + q, (unsigned long long)(o0 + st));
                }
            }
            st -= cnt;
            // columns of the lane's output rows but the last step's
            const bool last = run.flags & kRunLast;
            int w_row = run.cin;
            if (cnt) {
                for (int i = 0; i < run.n_ops; ++i)
                    w_row += (__ldg(reinterpret_cast<const uint32_t*>(a.steps + run.first + i) + 5) & 0xFF) == kXK2U;
            }
            const uint32_t mx = __reduce_max_sync(kFull, cnt);
            if (mx <= min(kLaneList, thr)) {
                // short lists: each lane lays its row's outputs out in the stage, as many rows as fit
                // at a time
                const uint32_t n = (uint32_t)n_all, s0 = (uint32_t)st, fit = min(kStageWords / wo, kStageRows);
                for (uint32_t c0 = 0; c0 < n; c0 += fit) {
                    const uint32_t lo = max(s0, c0), hi = min(s0 + cnt, c0 + fit);
                    if (lo < hi) {
                        const int m = (int)(hi - lo);
                        uint32_t* d = stage + (lo - c0) * wo;
                        for (int j = 0; j < m; ++j) owners[lo - c0 + j] = q;
                        if (last) {
                            if (off & kInlineTag) {
                                d[w_row] = (uint32_t)off;
                            } else {
                                const uint32_t* p = a.store.edges + off + (lo - s0);
#pragma unroll 1
                                for (int j = 0; j < m; j += 4) {
                                    uint32_t e[4];
#pragma unroll
                                    for (int u = 0; u < 4; ++u)
                                        if (j + u < m) e[u] = __ldg(p + j + u);
#pragma unroll
                                    for (int u = 0; u < 4; ++u)
                                        if (j + u < m) d[(j + u) * wo + w_row] = e[u];
                                }
                            }
                        }
                        for (int c = 0; c < w_row; c += 4) {
                            uint32_t x[4];
#pragma unroll
                            for (int u = 0; u < 4; ++u)
                                if (c + u < w_row)
                                    x[u] = c + u < run.cin ? __ldg(row + c + u) : app[(c + u - run.cin) * kLevThreads];
                            uint32_t* y = d + c;
                            for (int j = 0; j < m; ++j, y += wo) {
#pragma unroll
                                for (int u = 0; u < 4; ++u)
                                    if (c + u < w_row) y[u] = x[u];
                            }
                        }
                    }
                    __syncwarp();
                    // (columns past a query's own are never read; whatever the stage held goes out)
                    const uint32_t rows = min(n - c0, fit);
                    uint32_t* dst = a.out + (o0 + c0) * wo;
#pragma unroll 4
                    for (uint32_t i = lane; i < rows * wo; i += 32) dst[i] = stage[i];
                    for (uint32_t i = lane; i < rows; i += 32) a.owner_out[o0 + c0 + i] = owners[i];
                    __syncwarp();
                }
                o0 += n;
                continue;
            }
            // Longer lists: those past the threshold go to the queue as slices; the other rows'
            // outputs are spread over the lanes, eight in flight each, an output row finding its
            // input row by a binary search of the rows' positions.
            const bool slices = cnt > thr;
            if (slices)
                push_slices(a.ctl, a.heavy, a.heavy_cap, epoch, r, off, o0 + st, cnt, q);
            uint32_t ls = slices ? 0 : cnt;   // the outputs written here before the lane's
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, ls, d);
                if (lane >= d) ls += y;
            }
            const uint32_t n = __shfl_sync(kFull, ls, 31);
            if (!slices) ls -= cnt;
            owners[lane] = ls;
            owners[32 + lane] = q;
            owners[64 + lane] = (uint32_t)w_row | (uint32_t)run.cin << 8 | (uint32_t)last << 16;
            uint64_t* const at_of = reinterpret_cast<uint64_t*>(stage);   // where each row's outputs go
            at_of[lane] = o0 + st;
            __syncwarp();
            for (uint32_t c0 = lane; c0 < n; c0 += 32 * 8) {
                uint32_t e[8];
                int of[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const uint32_t o = c0 + 32 * u;
                    of[u] = -1;
                    if (o >= n) continue;
                    int lo = 0;   // the last row whose position is <= o (a row without outputs has
                                  // the next one's)
#pragma unroll
                    for (int step = 16; step > 0; step >>= 1)
                        if (owners[lo + step] <= o) lo += step;
                    of[u] = lo;
                    e[u] = 0;
                    if (owners[64 + lo] >> 16)
                        e[u] = list_at(a.store.edges, S.off[g][threadIdx.x - lane + lo], o - owners[lo]);
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    if (of[u] < 0) continue;
                    const uint64_t at = at_of[of[u]] + (c0 + 32 * u - owners[of[u]]);
                    const uint32_t info = owners[64 + of[u]];
                    const int rw = info & 0xFF, rc = info >> 8 & 0xFF, d = of[u] - lane;
                    uint32_t* dst = a.out + at * wo;
                    for (int c = 0; c < rw; ++c)
                        dst[c] = c < rc ? __ldg(row + d * a.w_in + c) : (app + d)[(c - rc) * kLevThreads];
                    if (info >> 16) dst[rw] = e[u];
                    a.owner_out[at] = owners[32 + of[u]];
                }
            }
            __syncwarp();
            o0 += n_all;
        }
        // The next chunk: claimed only now, since the CTAs behind it wait for its count (claimed a
        // look-back ahead it held them up by this one's writing), and whatever the grid, so that a
        // launch never needs its last CTAs to be resident.
        if (threadIdx.x == 0) s_claim = atomicAdd(&a.ctl->tile_counter, 1ull);
        __syncthreads();
        tile = s_claim;
    }

    // Out of chunks: every warp says how many it has written (its slices are reserved by then);
    // then write queued slices until every chunk is done and the queue is drained.
    if (lane == 0 && done) {
        __threadfence();   // (after any slices its lanes pushed)
        atomicAdd(&a.ctl->tiles_done, (unsigned long long)done);
    }
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_claim = claim_slice(a.ctl, a.heavy, a.heavy_cap, ntiles * kLevWarps, epoch, spin);
        __syncthreads();
        const unsigned long long idx = s_claim;
        if (idx == ~0ull) break;
        const HeavyItem* it = a.heavy + idx;
        const uint64_t in_row = __ldcg((const unsigned long long*)&it->in_row);
        const uint64_t l_off = __ldcg((const unsigned long long*)&it->off);
        const uint64_t out_pos = __ldcg((const unsigned long long*)&it->out_pos);
        const uint32_t count = __ldcg((const unsigned int*)&it->count);
        const uint32_t q = __ldcg((const unsigned int*)&it->q);
        // the row's appended columns again: its steps are the same for every thread
        LevelRun run = load_run(a, q);
        const uint32_t* row = a.in + in_row * (uint64_t)a.w_in;
        uint32_t* app = &S.app[0][0][threadIdx.x];
        uint64_t off;
        run.flags &= ~kRunLast;
        level_row(a, S.segs, run, row, app, &off, nullptr);
        int w_row = run.cin;
        for (int i = 0; i < run.n_ops; ++i)
            w_row += (__ldg(reinterpret_cast<const uint32_t*>(a.steps + run.first + i) + 5) & 0xFF) == kXK2U;
        uint32_t* dst = a.out + out_pos * wo;
        for (int c = 0; c < w_row; ++c) {
            const uint32_t x = c < run.cin ? __ldg(row + c) : app[(c - run.cin) * kLevThreads];
            for (uint32_t j = threadIdx.x; j < count; j += kLevThreads) dst[j * (uint64_t)wo + c] = x;
        }
        for (uint32_t j = threadIdx.x; j < count; j += kLevThreads) {
            dst[j * (uint64_t)wo + w_row] = __ldg(a.store.edges + l_off + j);
            a.owner_out[out_pos + j] = q;
        }
    }
    if (a.account) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sums.alg += __shfl_xor_sync(kFull, sums.alg, o);
            sums.sd += __shfl_xor_sync(kFull, sums.sd, o);
        }
        if (lane == 0) {
            atomicAdd(&a.ctl->alg_bytes, sums.alg);
            atomicAdd(&a.ctl->sum_deg, sums.sd);
        }
    }
    exit_protocol(a.ctl, a.status, epoch, a.heavy ? &a.heavy[0].tag : nullptr, sizeof(HeavyItem) / sizeof(uint32_t),
                  a.heavy ? a.heavy_cap : 0, active, a.out_rows);
}

}  // namespace

int level_grid(int sm_count) { return sm_count * kLevCtas; }

cudaError_t launch_level(const LevelArgs& a, int grid, cudaStream_t s) {
    level_kernel<<<std::max(grid, 1), kLevThreads, sizeof(LevelSmem), s>>>(a);
    return cudaGetLastError();
}

cudaError_t level_kernel_attrs() {
    cudaError_t e = cudaFuncSetAttribute(level_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(LevelSmem));
    return e != cudaSuccess ? e : use_max_shared_carveout(level_kernel);
}

}  // namespace wk
