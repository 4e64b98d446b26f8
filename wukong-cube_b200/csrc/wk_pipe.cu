// Fused passes of a single query: several steps in one launch.
//
// A planned query is a start list and a chain of steps.  Most steps give each row at most one
// output row: the filters, and known_to_unknown on a functional predicate (one whose lists all
// have one entry, found when the store is loaded).  A pass runs a whole run of those on a row held
// in registers, from the start list or the previous pass's table, and may end with one step whose
// lists multiply the rows; only what survives is written.  The triangle (predicate index,
// memberOf, subOrganizationOf, degreeFrom membership) is one launch that reads the index list and
// two columns of directory words and writes the closing rows; the star is one launch too.
//
// One launch per pass: CTAs claim chunks of consecutive rows (two per CTA on a large input) from a
// device counter.  A chunk's warps first count: each runs free over its own rows, 32 at a time, one
// per lane and two or four per thread with their lookups in flight together.  Then one decoupled
// look-back gives the chunk its output position, and the warps write, through shared memory so that
// stores are coalesced whatever the row width.  A chunk of up to four rounds (1.2 M rows on 148 SMs)
// keeps what it counted, as far as the columns it appends fit; a larger one runs its surviving rows
// again from L2, which is cheaper than the alternatives measured: a look-back per round put every
// warp behind the slowest of a wave (triangle at 10,000 organisations: 288 us against 190), and
// positions kept in memory (count, place and expand launches per step, the form before) cost 32
// bytes a row and step (390 us).  What bounds it: issue and the latency of the lookups; DRAM runs at
// a fifth of its rate.  Every lane of a round loads, a lost row's from the first place of the array
// it reads: a branch per lookup was 43 branches and 368 instructions per 32 rows of the triangle's
// three steps, 204 us; without them 152, and 119 with four rows per thread.
// Rows come out row-major, then in list order, as the CPU engine appends them (sparql.hpp:328-370).
// A row whose list is longer than the slice threshold goes to the slice queue that idle CTAs drain,
// so a hub vertex is spread over the device.
//
// Sizes are read on the device, so passes chain without a host round trip and can be captured.
// An output that does not fit sets kErrOverflow and the rows needed.  A row whose vertex is 0 names
// an index list.  A plan's rows hold it only where the store's own lists do, which is found when the
// store is loaded, and its steps are then taken for what they are; a single step over a caller's table,
// whose rows may hold anything, sets kErrUnfuse where the list has more than one entry, and the host
// runs it again as a step that multiplies rows.
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/wukong_b200.h"
#include "wk_device.cuh"
#include "wk_pipe.h"

namespace wk {
namespace {
using namespace dev;

constexpr int kPipeThreads = 256;
constexpr int kPipeWarps = kPipeThreads / 32;
// Rows per thread in flight x CTAs per SM (registers), kernel us of the star at 1,000 organisations /
// the star over a Zipf graph of 3,001 / 1 M rows expanded, which end with a last step, and the
// triangle at 10,000 / 2.5 M rows filtered, which do not: 2 x 4 (64) 32/64/84, 152/120; 3 x 4 33/61/95,
// 133/122; 4 x 4 43/90/118, 118/122; 4 x 3 (80) 29/60/93, 208/114; 2 x 5 (48) 36/106/116, 158/131;
// 2 x 3 32/72/92, 285/119; 1 x 6 (40) 39/104/163, 354/148.  A last step's lists take the registers,
// and so do a table's columns, whose loads hold a filter either way.
template <bool kLast, bool kList>
constexpr int kPipeRows = !kLast && kList ? 4 : 2;   // rows per thread: a round is 32 times that per warp
constexpr int kMaxGroups = kPipeMaxTileRows / kPipeThreads;   // 32-row groups of a warp's chunk
constexpr int kPipeCtas = 4;           // CTAs per SM: 64 registers a thread
constexpr int kStageWords = 512;       // output words staged per warp
constexpr int kMaxTableCols = 32;      // columns of the widest table (wk_config::max_cols)
// Output rows of `cols` words staged at once where they are spread over the lanes: one to four for
// each lane, or, for rows so wide that the stage holds fewer than 32 (from 17 columns on), as many as
// it holds.  Never none: the loop over a warp's output rows advances by it.
__host__ __device__ constexpr uint32_t spread_rows(int cols) {
    const uint32_t fit = (uint32_t)(kStageWords / cols);
    return fit >= 128 ? 128 : fit >= 32 ? fit & ~31u : fit;
}
constexpr bool spread_ends() {
    for (int c = 1; c <= kMaxTableCols; ++c)
        if (spread_rows(c) < 1 || spread_rows(c) * c > (uint32_t)kStageWords) return false;
    return true;
}
static_assert(spread_ends(), "the stage holds a row of any table");
constexpr int kKeepRounds = 4;         // rounds of a chunk whose counted lists are kept for writing
template <bool kLast>
constexpr int kHeldSlots = kLast ? 12 : 16;   // words a thread holds: columns x rows x rounds
static_assert(kHeldSlots<true> >= (kMaxPipeCols + 1) * kPipeRows<true, true> &&
                  kHeldSlots<false> >= (kMaxPipeCols + 1) * kPipeRows<false, true>,
              "one round's columns are always held");
constexpr uint32_t kLaneList = 16;     // a warp with no longer list writes a row's outputs by its lane
constexpr uint32_t kWarpList = 256;    // a warp with a longer list than this writes row by row

// How a step finds its list.
enum StepHow : uint32_t {
    kHowValue,   // a directory of values: every list has one entry
    kHowWord,    // a directory of pointer words
    kHowHash,    // no directory
    kHowOne,     // one list for every row (const_to_known, index_to_known)
};

// A step as the rounds read it, from shared memory.
struct alignas(16) StepRow {
    const uint2* dir;
    const void* words;
    uint32_t vid_lo, vid_span;
    uint32_t end_const;
    uint8_t op, how, col, tcol;   // start column (kHowOne: the target's); known_to_known's target column
    uint64_t one_off;             // kHowOne: the list
    uint32_t one_deg;
    uint32_t pad;
};
static_assert(sizeof(StepRow) == 48, "StepRow is three 16-byte words");

// The rows of a thread: row k of the round is lane `lane` of the warp's group k.  Columns of the
// input are read where they are; a list's entries and the columns the pass appends are kept in
// shared memory, where the steps index them by column.
template <bool kList>
struct Rows {
    const uint32_t* src;    // a table: row 0 (row k is 32 * k rows on)
    const uint32_t* safe;   // its first row, read in the place of a row that is not there
    int w_in;               // columns read from src (0 for a list)
    uint32_t* held;         // held column j of row k: held[j * stride + k * kPipeThreads]
    int stride;
    __device__ __forceinline__ uint32_t& at(int k, int c) const {
        return held[(c - w_in) * stride + k * kPipeThreads];
    }
    __device__ __forceinline__ uint32_t col(int k, int c) const {
        return kList || c >= w_in ? at(k, c) : __ldg(src + 32 * k * w_in + c);
    }
    // the same, of a row that is there only if `live` (else any word)
    __device__ __forceinline__ uint32_t col_if(bool live, int k, int c) const {
        if (kList || c >= w_in) return at(k, c);
        return __ldg((live ? src + 32 * k * w_in : safe) + c);
    }
    // the same of lane `of`
    __device__ __forceinline__ uint32_t col_of(int k, int c, int of) const {
        const int d = of - (int)(threadIdx.x & 31);
        return kList || c >= w_in ? (&at(k, c))[d] : __ldg(src + (32 * k + d) * w_in + c);
    }
};

// Pointer word of a key by hash, and of the index list that a vertex id of 0, or a type step's id,
// names (get_index, sparql.hpp:342-345); for the live rows of a round, out of line.
__device__ __forceinline__ uint64_t slow_word(const PipeArgs& a, const PipeOp& o, uint32_t cur) {
    const bool index = o.type_index || cur == 0;
    if (o.type_index && cur >= (1u << kNbitsIdx)) return 0;   // only 17-bit ids can be keys
    const SegDesc& sg = !index ? o.seg : a.store.segs[a.seg_index[o.type_index ? kIn : o.dir & 1]];
    const uint64_t key = o.type_index ? make_key(0, cur, kIn) : make_key(cur, o.pid, o.dir);
    return sg.num_buckets && key ? thread_probe(a.store, key, bucket_of(key, sg), &a.ctl->err) : 0;
}
template <int K>
struct SlowWords {
    uint64_t p[K];
};
template <int K>
struct SlowIds {
    uint32_t id[K];
};
template <int K>
__device__ __noinline__ SlowWords<K> slow_words(const PipeArgs& a, const PipeOp& o, SlowIds<K> cur, unsigned live) {
    SlowWords<K> w;
#pragma unroll
    for (int k = 0; k < K; ++k) w.p[k] = live >> k & 1 ? slow_word(a, o, cur.id[k]) : 0;
    return w;
}

// Pointer word of a start's key, found as the start list's own launch (list_kernel) finds it: anywhere
// in a bucket, and past it only where none of its slots is empty.
__device__ __noinline__ uint64_t start_word(const DevStore& st, uint64_t key, uint64_t bucket, unsigned* err) {
    for (int hop = 0; hop < kMaxProbeIters; ++hop) {
        if (bucket >= st.n_buckets) break;
        const Slot* b = st.slots + bucket * kAssoc;
        bool empty = false;
        uint64_t link = 0;
        for (int i = 0; i < kAssoc; i += 2) {
            ulonglong2 s0, s1;
            load_sector(b + i, &s0, &s1);
            if (s0.x == key) return s0.y;
            link = s1.x;
            empty |= s0.x == 0 || link == 0;   // (slot 7 empty: no chain)
            if (i + 1 < kAssoc - 1 && s1.x == key) return s1.y;
        }
        if (empty) return 0;
        bucket = key_vid(link);
    }
    atomicOr(err, kErrCorrupt);
    return 0;
}

// The one list of a step (or of the start), worked out once per CTA.
struct OneList {
    uint64_t off, deg;
};
__device__ __forceinline__ OneList one_list(const PipeArgs& a, const SegDesc& sg, uint64_t key, uint32_t mt,
                                            bool start) {
    OneList l{0, 0};
    if (sg.num_buckets == 0 || key == 0) return l;
    const uint64_t p = start ? start_word(a.store, key, bucket_of(key, sg), &a.ctl->err)
                             : hash_lookup(a.store, sg, key, &a.ctl->err);
    list_of_ptr(p, a.store.n_edges, &a.ctl->err, &l.off, &l.deg);
    if (mt) {
        uint64_t lo, hi;
        mt_slice(mt, l.deg, &lo, &hi);
        l.off += lo;
        l.deg = hi - lo;
    }
    return l;
}

// found[k]: target[k] in the list edges[off, off + deg) of the rows in `look`, short lists by quads
// as thread_member does, every row's quad in flight together.
template <int K>
__device__ __forceinline__ void pipe_member(const PipeArgs& a, const uint64_t (&off)[K],
                                            const uint32_t (&deg)[K], const uint32_t (&target)[K],
                                            const bool (&look)[K], bool (&found)[K]) {
    bool more = false, slow = false, quads[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        quads[k] = look[k] && deg[k] <= kQuadList && !(off[k] & kInlineTag);
        found[k] = look[k] && (off[k] & kInlineTag) && (uint32_t)off[k] == target[k];
        slow |= look[k] && !quads[k] && !(off[k] & kInlineTag);
        more |= quads[k];
    }
    if (slow) {
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (look[k] && !quads[k] && !(off[k] & kInlineTag))
                found[k] = thread_member(a.store.edges, off[k], deg[k], target[k], a.sorted_lists != 0);
    }
    for (int q = 0; more; q += 4) {
        uint4 x[K];
        more = false;
        const uint4* e4 = reinterpret_cast<const uint4*>(a.store.edges) + (q >> 2);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            // (a row without a quad here reads the first one: the array is padded)
            const uint4* p = reinterpret_cast<const uint4*>(a.store.edges);
            if (quads[k]) p = e4 + (off[k] >> 2);
            x[k] = __ldg(p);
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int lo = (int)(off[k] & 3), hi = lo + (int)deg[k];
            const uint32_t t = target[k];
            const bool here = quads[k] & (((x[k].x == t) & (q >= lo)) | ((x[k].y == t) & (q + 1 >= lo) & (q + 1 < hi)) |
                                          ((x[k].z == t) & (q + 2 >= lo) & (q + 2 < hi)) |
                                          ((x[k].w == t) & (q + 3 >= lo) & (q + 3 < hi)));
            found[k] |= here;
            quads[k] = quads[k] & !here & (q + 4 < hi);
            more |= quads[k];
        }
    }
}

// Directory lookup of a round: has[k] stays where cur[k] has a key, and at[k] is then the place of its
// word (0 elsewhere, so that every lane may load).  Every lane loads: a load per lane that needs one
// was a branch each, 43 a row group in the triangle and a third of its instructions.
template <int K>
__device__ __forceinline__ void dir_places(const StepRow& s, const uint32_t (&cur)[K],
                                           bool (&has)[K], uint32_t (&at)[K]) {
    const uint2* dir = s.dir;
    const uint32_t lo = s.vid_lo, span = s.vid_span;
    uint2 b[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const uint32_t id = cur[k] - lo;
        has[k] = has[k] & (id < span);
        b[k] = __ldg(dir + (has[k] ? id >> 5 : 0u));
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const uint32_t id = cur[k] - lo;
        has[k] = has[k] & dir_has(b[k], id);
        at[k] = has[k] ? dir_place(b[k], id) : 0u;
    }
}

// Lists of cur[k] in the step's segment for the live rows (deg 0 elsewhere).
template <int K>
__device__ __forceinline__ void pipe_lists(const PipeArgs& a, const StepRow& s, const PipeOp& o,
                                           const uint32_t (&cur)[K], const bool (&live)[K],
                                           uint64_t (&off)[K], uint32_t (&deg)[K]) {
    uint64_t p[K];
    bool zero = false;
#pragma unroll
    for (int k = 0; k < K; ++k) zero |= live[k] && cur[k] == 0;
    if (s.how <= kHowWord && !zero) {
        uint32_t at[K];
        bool has[K];
#pragma unroll
        for (int k = 0; k < K; ++k) has[k] = live[k];
        dir_places(s, cur, has, at);
        if (s.how == kHowValue) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const uint64_t e = make_inline_ptr(__ldg(static_cast<const uint32_t*>(s.words) + at[k]));
                p[k] = has[k] ? e : 0;
            }
        } else {
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const uint64_t e = __ldg(static_cast<const unsigned long long*>(s.words) + at[k]);
                p[k] = has[k] ? e : 0;
            }
        }
    } else {
        unsigned m = 0;
        SlowIds<K> ids;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            m |= (unsigned)live[k] << k;
            ids.id[k] = cur[k];
        }
        const SlowWords<K> w = slow_words<K>(a, o, ids, m);
#pragma unroll
        for (int k = 0; k < K; ++k) p[k] = w.p[k];
    }
    bool corrupt = false;   // (list_of_ptr, without its branches)
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const bool one = ptr_is_inline(p[k]);
        deg[k] = (uint32_t)ptr_size(p[k]);
        off[k] = one ? kInlineTag | (uint32_t)(p[k] >> kNbitsSize) : ptr_off(p[k]);
        const bool bad = !one & (off[k] + deg[k] > a.store.n_edges);
        corrupt |= bad & (deg[k] != 0);
        if (bad) deg[k] = 0;
    }
    if (corrupt) atomicOr(&a.ctl->err, kErrCorrupt);
}

// Bytes and list entries the steps run one launch each would account for (StepCtl), of a thread's
// rows; kept only for a profile.
struct Acc {
    unsigned long long alg, sd;
};

// The steps of the pass over a round; `live` keeps the rows that survive.  Without `test`: rows known
// to survive, of which only the appended columns are wanted.
template <bool kList, int K>
__device__ __forceinline__ void pipe_ops(const PipeArgs& a, const StepRow* steps, const Rows<kList>& v,
                                         bool (&live)[K], bool test, Acc* acc) {
    int w = a.w_in;   // columns of a row at this step
#pragma unroll 1
    for (int i = 0; i < a.n_ops; ++i) {
        const StepRow& s = steps[i];
        const uint32_t op = s.op, how = s.how;
        if (!test && op != kXK2U) continue;
        uint32_t cur[K], n_in = 0, sd = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const uint32_t x = v.col_if(live[k], k, s.col);
            cur[k] = live[k] ? x : kBlankId;
        }
        bool zero = false;
#pragma unroll
        for (int k = 0; k < K; ++k) zero |= cur[k] == 0;
        if (acc) {
#pragma unroll
            for (int k = 0; k < K; ++k) n_in += live[k] && (how == kHowOne || cur[k] != kBlankId);
        }
        if (how == kHowValue && !zero) {
            // every list has one entry and the directory holds it (a blank id is outside it)
            uint32_t at[K], e[K];
            dir_places(s, cur, live, at);
            const uint32_t* words = static_cast<const uint32_t*>(s.words);
#pragma unroll
            for (int k = 0; k < K; ++k) e[k] = __ldg(words + at[k]);
            if (acc) {
#pragma unroll
                for (int k = 0; k < K; ++k) sd += live[k];
            }
            if (op == kXK2U) {
#pragma unroll
                for (int k = 0; k < K; ++k) v.at(k, w) = e[k];   // (a lost row's word is not read)
            } else if (op == kXK2K) {
#pragma unroll
                for (int k = 0; k < K; ++k) live[k] = live[k] & (e[k] == v.col_if(live[k], k, s.tcol));
            } else {
                const uint32_t target = s.end_const;
#pragma unroll
                for (int k = 0; k < K; ++k) live[k] = live[k] & (e[k] == target);
            }
        } else {
            uint64_t off[K];
            uint32_t deg[K];
            if (how == kHowOne) {
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    off[k] = s.one_off;
                    deg[k] = live[k] ? s.one_deg : 0;
                }
            } else {
#pragma unroll
                for (int k = 0; k < K; ++k) live[k] = live[k] && cur[k] != kBlankId;
                pipe_lists(a, s, a.ops[i], cur, live, off, deg);
            }
#pragma unroll
            for (int k = 0; k < K; ++k) {
                sd += deg[k];
                live[k] = deg[k] != 0;
            }
            if (op == kXK2U) {
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    if (deg[k] > 1) atomicOr(&a.ctl->err, kErrUnfuse);   // (vid 0 only)
                    if (live[k]) v.at(k, w) = list_at(a.store.edges, off[k], 0);
                }
            } else {
                uint32_t target[K];
                bool found[K];
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    target[k] = how == kHowOne ? cur[k] : s.end_const;
                    if (op == kXK2K) target[k] = v.col_if(live[k], k, s.tcol);
                }
                pipe_member(a, off, deg, target, live, found);
#pragma unroll
                for (int k = 0; k < K; ++k) live[k] = found[k];
            }
        }
        const int w0 = w;
        if (op == kXK2U) ++w;
        if (acc) {
            uint32_t left = 0;
#pragma unroll
            for (int k = 0; k < K; ++k) left += live[k];
            acc->sd += sd;
            acc->alg += n_in * (w0 * 4 + 16) + left * w * 4 + sd * 4ull;
        }
    }
}

// Count and list of the last step for a round.
template <bool kList, int K>
__device__ __forceinline__ void pipe_last(const PipeArgs& a, const StepRow& s, const Rows<kList>& v,
                                          bool (&live)[K], int w, uint32_t (&cnt)[K],
                                          uint64_t (&off)[K], Acc* acc) {
    uint32_t cur[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const uint32_t x = v.col_if(live[k], k, s.col);
        cur[k] = live[k] ? x : kBlankId;
        live[k] = live[k] && cur[k] != kBlankId && !(a.last.type_index && cur[k] >= (1u << kNbitsIdx));
    }
    pipe_lists(a, s, a.last, cur, live, off, cnt);
    if (acc) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            acc->sd += cnt[k];
            acc->alg += live[k] * (w * 4 + 16) + cnt[k] * (unsigned long long)((w + 2) * 4);
        }
    }
}

// Copy `words` staged words to `dst` (coalesced); the warp's lanes all call this.
__device__ __forceinline__ void flush_words(uint32_t* dst, const uint32_t* s, uint32_t words) {
    __syncwarp();
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll 4
    for (uint32_t i = lane; i < words; i += 32) dst[i] = s[i];
    __syncwarp();
}

// kLast: the pass ends with a step that multiplies rows.  kList: the rows are the entries of one
// list.
template <bool kLast, bool kList>
__global__ void __launch_bounds__(kPipeThreads, kPipeCtas) pipe_kernel(const __grid_constant__ PipeArgs a) {
    constexpr int K = kPipeRows<kLast, kList>, kMaxRounds = kMaxGroups / K;
    extern __shared__ __align__(16) unsigned char smem[];   // pipe_smem_bytes
    // the lists of the kept rounds and their counts, then positions (a last step)
    uint64_t* const s_off = reinterpret_cast<uint64_t*>(smem);
    uint32_t* const s_pos = reinterpret_cast<uint32_t*>(s_off + (kLast ? kKeepRounds * K * kPipeThreads : 0));
    uint32_t* const s_stage = s_pos + (kLast ? kKeepRounds * K * kPipeThreads : 0);
    uint32_t* const s_held = s_stage + kPipeWarps * kStageWords;
    // which rows of each round survive (no last step)
    __shared__ unsigned char s_live[kLast ? 1 : kMaxRounds][kPipeThreads];
    __shared__ uint64_t s_warp[kPipeWarps];
    __shared__ OneList s_src;
    __shared__ StepRow s_steps[kMaxPipeOps + 1];
    __shared__ unsigned long long s_claim, s_excl;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned epoch = *(volatile unsigned*)&a.ctl->epoch;

    // the steps, and the lists of those that read one list for every row
    if (lane == 0 && warp <= kMaxPipeOps && (warp < a.n_ops || (warp == kMaxPipeOps && kLast))) {
        const PipeOp& o = warp < kMaxPipeOps ? a.ops[warp] : a.last;
        StepRow s{};
        s.dir = reinterpret_cast<const uint2*>(o.seg.dir);
        s.words = o.seg.dir_words;
        s.vid_lo = o.seg.vid_lo;
        s.vid_span = o.seg.vid_span;
        s.end_const = o.end_const;
        s.op = o.op;
        s.col = o.cs;
        s.tcol = o.ce;
        if (o.op == kXC2K || o.op == kXI2K) {
            const OneList l = one_list(a, o.seg, o.start_key, o.op == kXI2K ? o.mt : 0, false);
            s.how = kHowOne;
            s.col = o.ce;
            s.one_off = l.off;
            s.one_deg = (uint32_t)l.deg;
        } else {
            s.how = o.seg.vid_span && !o.type_index ? (o.seg.dir_values ? kHowValue : kHowWord) : kHowHash;
        }
        s_steps[warp] = s;
    }
    uint64_t R = 0;
    const uint32_t* in = a.in;
    uint32_t only = 0;   // the entry of a one-entry list kept in its pointer word (in is null)
    if (kList) {
        if (threadIdx.x == kPipeThreads - 1) {
            s_src = OneList{a.src_off, a.src_len};
            if (!a.src_known) s_src = one_list(a, a.src_seg, a.src_key, 0, true);
        }
        __syncthreads();
        const uint64_t sz = s_src.deg;
        // mt_factor slice (sparql.hpp:213-224)
        const uint64_t f = a.mt_factor > 0 ? (uint64_t)a.mt_factor : 1;
        uint64_t b = 0, e = sz;
        if (f > 1) {
            const uint64_t start = (uint64_t)a.mt_tid % f, len = sz / f;
            b = start * len;
            if (start != f - 1) e = b + len;
        }
        R = e - b;
        if (s_src.off & kInlineTag) {
            in = nullptr;
            only = (uint32_t)s_src.off;
        } else {
            in = a.store.edges + s_src.off + b;
        }
        if (a.account && blockIdx.x == 0 && threadIdx.x == 0) {
            atomicAdd(&a.ctl->sum_deg, (unsigned long long)sz);
            atomicAdd(&a.ctl->alg_bytes, 16ull + (unsigned long long)R * 8);
        }
    } else {
        R = *(volatile const uint64_t*)a.in_rows;
        if (R > a.in_cap_rows) R = 0;   // past capacity: the step before overflowed
        __syncthreads();
    }
    // A chunk per CTA: the rows split evenly, in groups of 32 per warp, at most kMaxGroups of them
    // (on larger inputs CTAs take several chunks).
    const uint64_t cta_rows = (R + gridDim.x - 1) / gridDim.x;
    const int groups = (int)min((unsigned long long)kMaxGroups,
                                (unsigned long long)((cta_rows + kPipeThreads - 1) / kPipeThreads));
    const int rounds = (groups + K - 1) / K;
    const uint32_t warp_rows = 32 * groups, tile_rows = warp_rows * kPipeWarps;
    uint64_t ntiles = groups ? (R + tile_rows - 1) / tile_rows : 0;
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
    const int wo = a.w_out, w_row = kLast ? wo - 1 : wo;   // columns of a surviving row
    uint32_t* stage = s_stage + warp * kStageWords;
    Acc sums{0, 0};
    Acc* acc = a.account ? &sums : nullptr;

    Rows<kList> v;
    v.w_in = kList ? 0 : a.w_in;
    v.safe = in;
    // small chunks keep what they count; the rows of a larger one are run again to be written
    const int held_cols = w_row - v.w_in;
    const bool keep = rounds <= (kLast ? kKeepRounds : kMaxRounds) && held_cols * K * rounds <= kHeldSlots<kLast>;
    v.stride = (keep ? rounds : 1) * K * kPipeThreads;
    bool live[K];
    uint32_t done = 0;   // chunks this CTA has written
    bool pushed = false;
    if (threadIdx.x == 0) s_claim = atomicAdd(&a.ctl->tile_counter, 1ull);
    __syncthreads();
    for (uint64_t tile = s_claim; tile < ntiles; ++done) {
        const uint64_t w0 = tile * tile_rows + (uint64_t)warp * warp_rows + lane;   // the warp's rows
        uint64_t total = 0;           // output rows of the warp
        uint64_t o0 = 0;              // its next output row
        // t < 0 counts round t + rounds, t >= 0 writes round t (one body for both); the look-back
        // lies between
#pragma unroll 1
        for (int t = -rounds; t < rounds; ++t) {
            if (t == 0) {
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) total += __shfl_xor_sync(kFull, total, d);
                if (lane == 0) s_warp[warp] = total;
                __syncthreads();
                uint64_t before = 0, all = 0;
#pragma unroll
                for (int w = 0; w < kPipeWarps; ++w) {
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
            const int round = count ? t + rounds : t;
            const uint64_t r0 = w0 + 32 * K * round;
            const int n_groups = min(K, groups - K * round);
            unsigned mask = ~0u;
            if (!kLast && !count) {
                mask = s_live[round][threadIdx.x];
                if (!__any_sync(kFull, mask)) continue;
            }
            const int slot = keep ? round : 0;
            uint64_t* loff = s_off + (slot * kPipeWarps + warp) * 32 * K;   // of the warp's rows
            uint32_t* pos = s_pos + (slot * kPipeWarps + warp) * 32 * K;
            v.held = s_held + slot * K * kPipeThreads + threadIdx.x;
            v.src = in + r0 * (uint64_t)a.w_in;
            if (count || !keep) {
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    live[k] = k < n_groups && (mask >> k & 1) && r0 + 32 * k < R;
                    if (kList) {
                        uint32_t x = only;
                        if (in) x = __ldg(live[k] ? v.src + 32 * k : in);
                        v.at(k, 0) = x;
                    }
                }
                // (rows known to survive: only their appended columns are wanted)
                if (kLast || count || w_row > a.w_in)
                    pipe_ops<kList>(a, s_steps, v, live, kLast || count, count ? acc : nullptr);
                if (kLast) {
                    uint32_t cnt[K];
                    uint64_t off[K];
                    pipe_last<kList>(a, s_steps[kMaxPipeOps], v, live, w_row, cnt, off, count ? acc : nullptr);
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        loff[32 * k + lane] = off[k];
                        pos[32 * k + lane] = cnt[k];
                        if (count) total += cnt[k];
                    }
                }
            }
            if (count) {
                if (!kLast) {
                    unsigned m = 0;
#pragma unroll
                    for (int k = 0; k < K; ++k) m |= (unsigned)live[k] << k;
                    s_live[round][threadIdx.x] = (unsigned char)m;
                    total += __popc(m);
                }
                continue;
            }
            if (!kLast) {
                // each surviving row into the stage, then out
                const uint32_t fit = kStageWords / wo;
#pragma unroll 1
                for (int k = 0; k < n_groups; ++k) {
                    const unsigned m = __ballot_sync(kFull, mask >> k & 1);
                    const uint32_t n = __popc(m), at = __popc(m & ((1u << lane) - 1));
                    for (uint32_t c0 = 0; c0 < n; c0 += fit) {
                        if ((mask >> k & 1) && at >= c0 && at < c0 + fit) {
                            uint32_t* d = stage + (at - c0) * wo;
                            for (int c = 0; c < wo; ++c) d[c] = v.col(k, c);
                        }
                        flush_words(a.out + (o0 + c0) * wo, stage, min(n - c0, fit) * wo);
                    }
                    o0 += n;
                }
                continue;
            }
            uint32_t mx = 0;
#pragma unroll
            for (int k = 0; k < K; ++k) mx = max(mx, pos[32 * k + lane]);
            mx = __reduce_max_sync(kFull, mx);
            if (mx <= kLaneList) {
                // Short lists: each lane lays its row's outputs out in the stage, as many rows as fit
                // at a time.  (Spread over the lanes as below they took 300 instructions per 32
                // output rows, and the expansion of 1 M rows 94 us.)
                const uint32_t fit = kStageWords / wo;
#pragma unroll 1
                for (int k = 0; k < n_groups; ++k) {
                    const uint32_t cnt = pos[32 * k + lane];
                    const uint64_t off = loff[32 * k + lane];
                    uint32_t st = cnt;
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const uint32_t y = __shfl_up_sync(kFull, st, d);
                        if (lane >= d) st += y;
                    }
                    const uint32_t n = __shfl_sync(kFull, st, 31);
                    st -= cnt;
                    for (uint32_t c0 = 0; c0 < n; c0 += fit) {
                        const uint32_t lo = max(st, c0), hi = min(st + cnt, c0 + fit);
                        if (lo < hi) {
                            const int m = (int)(hi - lo);
                            uint32_t* d = stage + (lo - c0) * wo;
                            if (off & kInlineTag) {
                                d[w_row] = (uint32_t)off;
                            } else {
                                const uint32_t* p = a.store.edges + off + (lo - st);
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
                            for (int c = 0; c < w_row; ++c) {
                                const uint32_t x = v.col(k, c);
                                uint32_t* y = d + c;
                                for (int j = 0; j < m; ++j, y += wo) *y = x;
                            }
                        }
                        flush_words(a.out + (o0 + c0) * wo, stage, min(n - c0, fit) * wo);
                    }
                    o0 += n;
                }
                continue;
            }
            if (mx <= kWarpList) {
                // Output rows spread over the lanes: an output row finds its input row by a binary
                // search of the positions of the warp's rows, so lists are read and rows written in
                // output order, through the stage, whatever the lists' lengths.
                uint32_t n = 0;
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    const uint32_t cnt = pos[32 * k + lane];
                    uint32_t st = cnt;
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const uint32_t y = __shfl_up_sync(kFull, st, d);
                        if (lane >= d) st += y;
                    }
                    pos[32 * k + lane] = n + st - cnt;
                    n += __shfl_sync(kFull, st, 31);
                }
                __syncwarp();
                const uint32_t fit = spread_rows(wo);   // output rows staged at once
                for (uint32_t c0 = 0; c0 < n; c0 += fit) {
                    const uint32_t c1 = min(n, c0 + fit);
                    int row[4];
                    uint32_t e[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const uint32_t o = c0 + 32 * u + lane;
                        row[u] = 0;
                        e[u] = 0;
                        if (o >= c1) continue;
                        int lo = 0;   // the last row whose position is <= o
#pragma unroll
                        for (int step = 16 * K; step > 0; step >>= 1)
                            if (pos[lo + step] <= o) lo += step;
                        row[u] = lo;
                        e[u] = list_at(a.store.edges, loff[lo], o - pos[lo]);
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const uint32_t o = c0 + 32 * u + lane;
                        if (o >= c1) continue;
                        uint32_t* d = stage + (o - c0) * wo;
                        for (int c = 0; c < w_row; ++c) d[c] = v.col_of(row[u] >> 5, c, row[u] & 31);
                        d[w_row] = e[u];
                    }
                    flush_words(a.out + (o0 + c0) * wo, stage, (c1 - c0) * wo);
                }
                o0 += n;
                continue;
            }
            // a long list among them: row by row, the warp over each row's list; past the threshold,
            // slices for the queue
            __syncwarp();
#pragma unroll 1
            for (int r = 0; r < 32 * n_groups; ++r) {
                const uint32_t n = pos[r];
                const uint64_t lo = loff[r];
                if (n > thr) {
                    if (lane == 0) push_slices(a.ctl, a.heavy, a.heavy_cap, epoch, r0 - lane + r, lo, o0, n, 0);
                    pushed = true;
                } else if (n) {
                    uint32_t* dst = a.out + o0 * wo;
                    for (int c = 0; c < w_row; ++c) {
                        const uint32_t x = v.col_of(r >> 5, c, r & 31);
                        for (uint32_t j = lane; j < n; j += 32) dst[j * (uint64_t)wo + c] = x;
                    }
                    for (uint32_t j = lane; j < n; j += 32) dst[j * (uint64_t)wo + w_row] = list_at(a.store.edges, lo, j);
                }
                o0 += n;
            }
            __syncwarp();
        }
        // The next chunk: claimed only now, since the CTAs behind it wait for its count (claimed a
        // look-back ahead it held them up by this one's writing), and whatever the grid, so that a
        // launch never needs its last CTAs to be resident.
        if (threadIdx.x == 0) s_claim = atomicAdd(&a.ctl->tile_counter, 1ull);
        __syncthreads();
        tile = s_claim;
    }

    if (kLast) {
        // Out of chunks: every warp says how many it has written (its slices are reserved by
        // then); then write queued slices until every chunk is done and the queue is drained.
        if (lane == 0 && done) {
            if (pushed) __threadfence();
            atomicAdd(&a.ctl->tiles_done, (unsigned long long)done);
        }
        for (;;) {
            __syncthreads();
            if (threadIdx.x == 0) s_claim = claim_slice(a.ctl, a.heavy, a.heavy_cap, ntiles * kPipeWarps, epoch, spin);
            __syncthreads();
            const unsigned long long idx = s_claim;
            if (idx == ~0ull) break;
            const HeavyItem* it = a.heavy + idx;
            const uint64_t in_row = __ldcg((const unsigned long long*)&it->in_row);
            const uint64_t l_off = __ldcg((const unsigned long long*)&it->off);
            const uint64_t out_pos = __ldcg((const unsigned long long*)&it->out_pos);
            const uint32_t count = __ldcg((const unsigned int*)&it->count);
            // the row's appended columns again: its steps are the same for every thread
            v.src = in + in_row * (uint64_t)a.w_in;
            v.held = s_held + threadIdx.x;
            if (kList) v.at(0, 0) = in ? __ldg(v.src) : only;
#pragma unroll
            for (int k = 0; k < K; ++k) live[k] = k == 0;
            pipe_ops<kList>(a, s_steps, v, live, false, nullptr);
            const uint64_t ne = (uint64_t)count * wo;
            uint32_t* dst = a.out + out_pos * wo;
            for (uint64_t e = threadIdx.x; e < ne; e += kPipeThreads) {
                const uint64_t j = e / wo;
                const int c = (int)(e - j * wo);
                dst[e] = c < w_row ? v.col(0, c) : __ldg(a.store.edges + l_off + j);
            }
        }
    }
    if (acc) {
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
                  a.heavy ? a.heavy_cap : 0, active);
}

using PipeKernel = void (*)(const PipeArgs);
constexpr int kPipeKernels = 4;
PipeKernel pipe_kernel_of(int k) {
    static const PipeKernel kernels[kPipeKernels] = {pipe_kernel<false, false>, pipe_kernel<false, true>,
                                                     pipe_kernel<true, false>, pipe_kernel<true, true>};
    return kernels[k];
}

}  // namespace

static size_t pipe_smem_bytes(bool last) {
    return (last ? kKeepRounds * kPipeRows<true, false> * kPipeThreads * 12 : 0) + kPipeWarps * kStageWords * 4 +
           (last ? kHeldSlots<true> : kHeldSlots<false>) * kPipeThreads * 4;
}
static bool kernel_has_last(int k) { return k >= 2; }

int pipe_grid(int sm_count) { return sm_count * kPipeCtas; }

int pipe_grid_beside(int sm_count, const CtaUse& other, int other_ctas) {
    int regs = 0, dev = 0, reserved = 0;
    size_t smem = 0;
    for (int k = 0; k < kPipeKernels; ++k) {
        cudaFuncAttributes fa{};
        if (cudaFuncGetAttributes(&fa, pipe_kernel_of(k)) != cudaSuccess) fa.numRegs = 255;
        regs = std::max(regs, fa.numRegs);
        smem = std::max(smem, fa.sharedSizeBytes + pipe_smem_bytes(kernel_has_last(k)));
    }
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
    CtaUse me{smem + (size_t)reserved, ((regs * 32 + 255) / 256) * 256 * kPipeWarps, kPipeThreads};
    return blocks_beside(me, kPipeCtas, other, other_ctas) * sm_count;
}

cudaError_t launch_pipe(const PipeArgs& a, int grid, cudaStream_t s) {
    pipe_kernel_of((a.has_last ? 2 : 0) + (a.from_list ? 1 : 0))<<<std::max(grid, 1), kPipeThreads,
                                                                       pipe_smem_bytes(a.has_last != 0), s>>>(a);
    return cudaGetLastError();
}

cudaError_t pipe_kernel_attrs() {
    for (int k = 0; k < kPipeKernels; ++k) {
        cudaError_t e = cudaFuncSetAttribute(pipe_kernel_of(k), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)pipe_smem_bytes(kernel_has_last(k)));
        if (e == cudaSuccess) e = use_max_shared_carveout(pipe_kernel_of(k));
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace wk
