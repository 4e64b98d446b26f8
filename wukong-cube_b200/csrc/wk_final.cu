// Post-pattern stage on the device: DISTINCT, OFFSET, LIMIT and the projection onto the
// required variables, as SPARQLEngine::final_process applies them (sparql.hpp:1419-1546), so a
// query's table can be finished without leaving the GPU.  ORDER BY is not here: the reference
// orders by the strings of the ids (sparql.hpp:1378-1400), which needs the string server.
//
// DISTINCT follows the reference step for step: the rows are sorted by all their columns,
// compared as signed 32-bit values (ReduceCmp over an int table, sparql.hpp:1403-1417), then
// of each run of neighbours equal on the required columns the first is kept.  The sort is an
// LSD radix sort of packed keys over only the bits in which the rows differ (see "DISTINCT sort"
// below).  Only the columns up to the last required one are looked at: the columns behind it order
// rows that are equal in all that is output.  Rows equal in every column looked at are
// interchangeable, so the result does not depend on how the reference's std::sort orders them.  A
// table found to be in that order already (one pass over it, scan_rows_kernel) skips the sort.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "wk_ctx.h"
#include "wk_device.cuh"
#include "wk_radix.cuh"

namespace wk {
namespace {
using namespace dev;

#define WKF_CUDA(ctx, call)                                        \
    do {                                                           \
        cudaError_t e_ = (call);                                   \
        if (e_ != cudaSuccess) return (ctx)->cuda_fail(e_, #call); \
    } while (0)

constexpr int kFinThreads = 256;
constexpr int kDigits = radix::kDigits;

// ---------------------------------------------------------------- DISTINCT sort
// The sort orders rows by their columns as signed 32-bit values.  A column is first mapped
// to its offset from the column's smallest value (in signed order), so a column spanning d
// distinct-order values needs only ceil(log2(d)) bits, and a constant column none.  Columns are
// packed, last column in the lowest bits, into 64-bit keys ("chunks" of consecutive columns that
// fit in 64 bits); the LSD sort runs the chunks from the last columns to the first, and within a
// chunk one stable counting pass per byte of the chunk's bits.
//
// Where one chunk holds all the columns, the key is the row: the passes move the keys alone (16
// bytes a row and pass instead of 24), and the compaction compares neighbouring keys and writes the
// required columns out of them, so no index array is kept and no row is gathered.  Else every
// pass moves the row indices with the keys, and the table is read once per chunk.
// Measured on 3,000,000 rows of three columns (63 bits, 39 of them up to the second column), the
// first two required: 598 -> 265 us a call.

// One chunk's key layout: columns ccol[0..nc), most significant first, ccol[j] in cbits[j]
// bits above the next, offset by cmin[j].
struct ChunkDesc {
    int nc;
    int ccol[32];
    int cbits[32];
    uint32_t cmin[32];
};

// keys[i] = the chunk key of row idx_in[i] (row i when idx_in is null); idx_out[i] = that row.
__global__ void __launch_bounds__(kFinThreads) key_kernel(const uint32_t* table, int cols, ChunkDesc cd,
                                                          const uint32_t* idx_in, uint32_t n,
                                                          unsigned long long* keys, uint32_t* idx_out) {
    for (uint32_t i = blockIdx.x * kFinThreads + threadIdx.x; i < n; i += gridDim.x * kFinThreads) {
        const uint32_t r = idx_in ? idx_in[i] : i;
        const uint32_t* row = table + (uint64_t)r * cols;
        unsigned long long k = 0;
        for (int j = 0; j < cd.nc; ++j)
            k = (k << cd.cbits[j]) | (unsigned long long)((__ldg(row + cd.ccol[j]) ^ 0x80000000u) - cd.cmin[j]);
        keys[i] = k;
        idx_out[i] = r;
    }
}

// One pass over the rows: *flag = 0 (all ones before) when some row is greater than the next one,
// its first `cmp` columns compared as signed 32-bit values in column order (ReduceCmp), and the
// smallest and largest value of each of these columns (in signed order, stored with the sign bit
// flipped; the largest as its complement, so that both begin as all ones).  A table already in that
// order is what the sort would return (rows equal in these columns are interchangeable), so the
// sort is skipped for it: the exploration writes rows in input order and each row's new column
// from a sorted list, so a table started from an index or a constant with unique rows comes out in
// this order.
// A CTA stages `tile_rows` consecutive rows and the row after them in shared memory with
// coalesced loads, eight in flight per thread, then each thread compares rows with the next ones
// and takes the columns' extremes out of shared memory.  Bound by the read of the table: 14.9 us at
// 36 MB, where two kernels that each read it took 22.
constexpr int kCheckWords = 8192;   // 32 KiB of rows per tile

__global__ void __launch_bounds__(kFinThreads) scan_rows_kernel(const uint32_t* table, int cols, int cmp,
                                                                uint32_t n, uint32_t tile_rows, unsigned* flag,
                                                                uint32_t* mm /* [2 * cmp] */) {
    __shared__ uint32_t s_t[kCheckWords];
    __shared__ uint32_t s_lo[32], s_hi[32];
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        s_lo[threadIdx.x] = 0xFFFFFFFFu;
        s_hi[threadIdx.x] = 0;
    }
    const uint32_t pairs = n - 1;   // pair i is rows (i, i + 1); n >= 2
    bool bad = false;
    for (uint64_t t0 = (uint64_t)blockIdx.x * tile_rows; t0 < pairs; t0 += (uint64_t)gridDim.x * tile_rows) {
        const uint32_t here = (uint32_t)min((uint64_t)tile_rows, pairs - t0);   // pairs of this tile
        const uint32_t words = (here + 1) * (uint32_t)cols;                     // <= kCheckWords
        const uint32_t* src = table + t0 * cols;
        constexpr int kPer = 8;
        uint32_t w = threadIdx.x;
        for (; w + (kPer - 1) * kFinThreads < words; w += kPer * kFinThreads) {
            uint32_t v[kPer];
#pragma unroll
            for (int r = 0; r < kPer; ++r) v[r] = __ldg(src + w + r * kFinThreads);
#pragma unroll
            for (int r = 0; r < kPer; ++r) s_t[w + r * kFinThreads] = v[r] ^ 0x80000000u;
        }
        for (; w < words; w += kFinThreads) s_t[w] = __ldg(src + w) ^ 0x80000000u;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < here; i += kFinThreads) {
            const uint32_t* r = s_t + i * cols;
            for (int c = 0; c < cmp; ++c) {
                const uint32_t x = r[c], y = r[cols + c];
                if (x != y) {
                    bad |= x > y;
                    break;
                }
            }
        }
        for (int c = 0; c < cmp; ++c) {
            uint32_t lo = 0xFFFFFFFFu, hi = 0;
            for (uint32_t i = threadIdx.x; i <= here; i += kFinThreads) {
                const uint32_t x = s_t[i * cols + c];
                lo = min(lo, x);
                hi = max(hi, x);
            }
            lo = __reduce_min_sync(kFull, lo);
            hi = __reduce_max_sync(kFull, hi);
            if (lane == 0 && lo <= hi) {
                atomicMin(&s_lo[c], lo);
                atomicMax(&s_hi[c], hi);
            }
        }
        __syncthreads();   // before the next tile overwrites s_t
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0) *flag = 0;
    if ((int)threadIdx.x < cmp && s_lo[threadIdx.x] <= s_hi[threadIdx.x]) {
        atomicMin(&mm[2 * threadIdx.x], s_lo[threadIdx.x]);
        atomicMin(&mm[2 * threadIdx.x + 1], ~s_hi[threadIdx.x]);
    }
}

struct SortPass {
    const unsigned long long* key_in;
    const uint32_t* idx_in;
    unsigned long long* key_out;
    uint32_t* idx_out;
    int shift;
    uint32_t n;
    uint32_t per_cta;        // elements of a CTA
    uint32_t* hist;          // [kDigits][grid]: digit-major, so one scan gives the offsets
    uint32_t* dtot;          // [kDigits]: elements of each digit
};
static_assert(kFinThreads == radix::kThreads);

__device__ __forceinline__ void chunk(uint32_t n, uint32_t* lo, uint32_t* hi) {
    const uint32_t c = (n + gridDim.x - 1) / gridDim.x;
    *lo = min(n, blockIdx.x * c);
    *hi = min(n, *lo + c);
}

template <class A>
__device__ __forceinline__ void span(const A& a, uint32_t* lo, uint32_t* hi) {
    *lo = (uint32_t)min((uint64_t)a.n, (uint64_t)blockIdx.x * a.per_cta);
    *hi = (uint32_t)min((uint64_t)a.n, (uint64_t)*lo + a.per_cta);
}

// Digit counts of each CTA's chunk.  A thread loads eight keys before it counts any of them, so
// eight loads per thread are in flight instead of one.
__global__ void __launch_bounds__(kFinThreads) hist_kernel(const SortPass a) {
    constexpr int kPer = 8;
    __shared__ uint32_t s_h[kDigits];
    s_h[threadIdx.x] = 0;
    __syncthreads();
    uint32_t lo, hi;
    span(a, &lo, &hi);
    uint64_t i = lo + threadIdx.x;
    for (; i + (kPer - 1) * kFinThreads < hi; i += kPer * kFinThreads) {
        unsigned long long k[kPer];
#pragma unroll
        for (int r = 0; r < kPer; ++r) k[r] = a.key_in[i + r * kFinThreads];
#pragma unroll
        for (int r = 0; r < kPer; ++r) atomicAdd(&s_h[(uint32_t)(k[r] >> a.shift) & 0xFFu], 1u);
    }
    for (; i < hi; i += kFinThreads) atomicAdd(&s_h[(uint32_t)(a.key_in[i] >> a.shift) & 0xFFu], 1u);
    __syncthreads();
    a.hist[threadIdx.x * gridDim.x + blockIdx.x] = s_h[threadIdx.x];
}

// Exclusive scan of n words in place by one CTA of 1,024 threads.
__global__ void __launch_bounds__(1024) scan_kernel(uint32_t* v, uint32_t n, uint32_t* total) {
    __shared__ uint64_t s_warp[32];
    __shared__ uint64_t s_carry;
    if (threadIdx.x == 0) s_carry = 0;
    __syncthreads();
    for (uint32_t r0 = 0; r0 < n; r0 += 1024) {
        const uint32_t i = r0 + threadIdx.x;
        const uint64_t x = i < n ? v[i] : 0;
        const uint64_t ex = block_exclusive_sum<1024>(x, s_warp);
        const uint64_t carry = s_carry;
        if (i < n) v[i] = (uint32_t)(carry + ex);
        __syncthreads();
        if (threadIdx.x == 1023) s_carry = carry + ex + x;
        __syncthreads();
    }
    if (threadIdx.x == 0 && total) *total = (uint32_t)s_carry;
}

// The scatter of a pass (radix_scatter).  With the row indices: 4 CTAs per SM (64 registers, no
// spills; 43 KB of shared memory each), so the pass's 4 CTAs per SM run in one wave.  Keys alone:
// 5 CTAs per SM, each over whole tiles.
template <bool kIdx>
__global__ void __launch_bounds__(kFinThreads, kIdx ? 4 : 5) scatter_kernel(const SortPass a) {
    __shared__ radix::Tile<kIdx> s_tile;
    // thread d: digit d's first place for this CTA = the elements of smaller digits plus the
    // digit-d elements of the CTAs before this one
    const uint32_t smaller = (uint32_t)block_exclusive_sum<kFinThreads>(a.dtot[threadIdx.x], s_tile.warp);
    const uint32_t first = smaller + a.hist[threadIdx.x * gridDim.x + blockIdx.x];
    uint32_t lo, hi;
    span(a, &lo, &hi);
    radix::radix_scatter<kIdx>(s_tile, a.key_in, a.idx_in, a.key_out, a.idx_out, lo, hi, first,
                        [&](unsigned long long k, uint32_t) { return (uint32_t)(k >> a.shift) & 0xFFu; });
}

// ---- one chunk holds all the columns looked at: keys alone

// The rows' keys and the first pass's digit counts, a CTA over the span it has in that pass: the
// table is read once, eight rows in flight per thread.
__global__ void __launch_bounds__(kFinThreads) key_hist_kernel(const uint32_t* table, int cols,
                                                               const __grid_constant__ ChunkDesc cd, const SortPass a,
                                                               unsigned long long* keys) {
    constexpr int kPer = 8;
    __shared__ uint32_t s_h[kDigits];
    s_h[threadIdx.x] = 0;
    __syncthreads();
    uint32_t lo, hi;
    span(a, &lo, &hi);
    for (uint64_t i0 = lo + threadIdx.x; i0 < hi; i0 += kPer * kFinThreads) {
        unsigned long long k[kPer];
#pragma unroll
        for (int r = 0; r < kPer; ++r) k[r] = 0;
        for (int j = 0; j < cd.nc; ++j) {
            const int c = cd.ccol[j], bits = cd.cbits[j];
            const uint32_t lowest = cd.cmin[j];
            uint32_t v[kPer];
#pragma unroll
            for (int r = 0; r < kPer; ++r) {
                const uint64_t i = i0 + r * kFinThreads;
                v[r] = i < hi ? __ldg(table + i * cols + c) : 0;
            }
#pragma unroll
            for (int r = 0; r < kPer; ++r)
                k[r] = (k[r] << bits) | (unsigned long long)((v[r] ^ 0x80000000u) - lowest);
        }
#pragma unroll
        for (int r = 0; r < kPer; ++r) {
            const uint64_t i = i0 + r * kFinThreads;
            if (i >= hi) continue;
            keys[i] = k[r];
            atomicAdd(&s_h[(uint32_t)k[r] & 0xFFu], 1u);
        }
    }
    __syncthreads();
    a.hist[threadIdx.x * gridDim.x + blockIdx.x] = s_h[threadIdx.x];
}

// The required columns of a key: column k is the `bits[k]` bits at `shift[k]`, above `lowest[k]`.
struct KeyCols {
    int n;
    unsigned long long mask;   // their bits: neighbours that differ in none of them are one row
    int shift[32], bits[32];
    uint32_t lowest[32];
};

struct KeyRuns {
    const unsigned long long* keys;   // sorted
    uint32_t n;
    uint32_t per_cta;                 // keys of a CTA
    uint32_t* part;                   // [grid + 1] kept keys per CTA, then their exclusive scan
};

__device__ __forceinline__ bool starts_key_run(const KeyRuns& a, const KeyCols& kc, uint32_t i) {
    return i == 0 || ((a.keys[i] ^ a.keys[i - 1]) & kc.mask) != 0;
}

__global__ void __launch_bounds__(kFinThreads) key_count_kernel(const KeyRuns a, const __grid_constant__ KeyCols kc) {
    __shared__ uint64_t s_warp[kFinThreads / 32];
    uint32_t lo, hi;
    span(a, &lo, &hi);
    uint64_t c = 0;
#pragma unroll 4
    for (uint64_t i = (uint64_t)lo + threadIdx.x; i < hi; i += kFinThreads) c += starts_key_run(a, kc, (uint32_t)i);
    const uint64_t ex = block_exclusive_sum<kFinThreads>(c, s_warp);
    if (threadIdx.x == kFinThreads - 1) a.part[blockIdx.x] = (uint32_t)(ex + c);
}

// Kept key number r goes to output row r - start where that lies in [0, count).  A warp takes four
// runs of 32 keys a round, so one scan serves 1,024 keys; a round's kept keys are packed in shared
// memory and written out column by column, consecutive threads on consecutive words.
// The rows kept (*total) are known on the device only: a result that does not fit `cap` words is
// left out whole, and the host, which reads *total, makes room and runs this again.
__global__ void __launch_bounds__(kFinThreads) key_write_kernel(const KeyRuns a, const __grid_constant__ KeyCols kc,
                                                                const uint32_t* total, uint64_t offset,
                                                                int64_t limit, uint32_t* out, uint64_t cap,
                                                                uint64_t* out_rows) {
    constexpr int kPer = 4;
    __shared__ uint32_t s_n[kFinThreads / 32];
    __shared__ unsigned long long s_key[kPer * kFinThreads];
    __shared__ uint4 s_col[32];   // a column's shift, mask, smallest value
    if (threadIdx.x < 32)
        s_col[threadIdx.x] = make_uint4(kc.shift[threadIdx.x],
                                        kc.bits[threadIdx.x] ? 0xFFFFFFFFu >> (32 - kc.bits[threadIdx.x]) : 0,
                                        kc.lowest[threadIdx.x], 0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t m = *total, start = min(offset, m);
    const uint64_t count = limit < 0 ? m - start : min((uint64_t)limit, m - start);
    if (count * kc.n > cap) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) *out_rows = count;
    uint32_t lo, hi;
    span(a, &lo, &hi);
    uint64_t carry = a.part[blockIdx.x];
    for (uint64_t base = lo; base < hi; base += kPer * kFinThreads) {
        unsigned long long key[kPer];
        unsigned m32[kPer];
        uint32_t mine = 0;
#pragma unroll
        for (int r = 0; r < kPer; ++r) {
            const uint64_t i = base + (warp * kPer + r) * 32 + lane;
            key[r] = i < hi ? a.keys[i] : 0;
        }
        const uint64_t w0 = base + warp * kPer * 32;   // the key before the warp's
        unsigned long long before = lane == 0 && w0 > 0 && w0 < hi ? a.keys[w0 - 1] : 0;
#pragma unroll
        for (int r = 0; r < kPer; ++r) {
            const uint64_t i = w0 + r * 32 + lane;
            const unsigned long long up = __shfl_up_sync(kFull, key[r], 1);
            const unsigned long long prev = lane == 0 ? before : up;
            before = __shfl_sync(kFull, key[r], 31);
            m32[r] = __ballot_sync(kFull, i < hi && (i == 0 || ((key[r] ^ prev) & kc.mask) != 0));
            mine += __popc(m32[r]);
        }
        // the warp's kept keys go before those of the warps behind it
        if (lane == 0) s_n[warp] = mine;
        __syncthreads();
        uint32_t at = 0, kept = 0;
#pragma unroll
        for (int w = 0; w < kFinThreads / 32; ++w) {
            if (w < warp) at += s_n[w];
            kept += s_n[w];
        }
#pragma unroll
        for (int r = 0; r < kPer; ++r) {
            if (m32[r] >> lane & 1u) s_key[at + __popc(m32[r] & ((1u << lane) - 1))] = key[r];
            at += __popc(m32[r]);
        }
        __syncthreads();
        // the packed keys [from, to) are output rows carry + from - start ...
        const uint32_t from = carry < start ? (uint32_t)min((uint64_t)kept, start - carry) : 0;
        const uint32_t to = (uint32_t)min((uint64_t)kept, start + count > carry ? start + count - carry : 0);
        if (from < to) {
            uint32_t* dst = out + (carry + from - start) * kc.n;
            const uint32_t words = (to - from) * kc.n, n = (uint32_t)kc.n;
            uint32_t j = threadIdx.x / n, c = threadIdx.x - j * n;
            const uint32_t dj = kFinThreads / n, dc = kFinThreads - dj * n;
            for (uint32_t e = threadIdx.x; e < words; e += kFinThreads) {
                const uint4 col = s_col[c];
                dst[e] = (((uint32_t)(s_key[from + j] >> col.x) & col.y) + col.z) ^ 0x80000000u;
                j += dj;
                c += dc;
                if (c >= n) {
                    c -= n;
                    ++j;
                }
            }
        }
        carry += kept;
        __syncthreads();
    }
}

// out row i = table row idx[i]: the table in sorted order, so the run compaction and the
// projection read consecutive rows instead of gathering each row (and its neighbour) through
// the index array.  One thread per element, consecutive threads on consecutive elements.
__global__ void __launch_bounds__(kFinThreads) gather_rows_kernel(const uint32_t* table, int cols,
                                                                  const uint32_t* idx, uint32_t n, uint32_t* out) {
    const uint64_t total = (uint64_t)n * cols;
    for (uint64_t e = blockIdx.x * (uint64_t)kFinThreads + threadIdx.x; e < total;
         e += (uint64_t)gridDim.x * kFinThreads) {
        const uint64_t i = e / cols;
        const int c = (int)(e - i * cols);
        out[e] = __ldg(table + (uint64_t)__ldg(idx + i) * cols + c);
    }
}

struct UniqueArgs {
    const uint32_t* table;
    int cols;
    const int32_t* keep;   // required columns
    int n_keep;
    const uint32_t* idx;   // sorted row indices
    uint32_t n;
    uint32_t* part;        // [grid + 1] kept rows per CTA, then their exclusive scan
    uint32_t* out;         // kept row indices
};

// Row i of the sorted order (idx null: the table was in order already).
__device__ __forceinline__ uint32_t sorted_row(const UniqueArgs& a, uint32_t i) { return a.idx ? a.idx[i] : i; }

__device__ __forceinline__ bool starts_run(const UniqueArgs& a, uint32_t i) {
    if (i == 0) return true;
    const uint32_t* r = a.table + (uint64_t)sorted_row(a, i) * a.cols;
    const uint32_t* p = a.table + (uint64_t)sorted_row(a, i - 1) * a.cols;
    for (int k = 0; k < a.n_keep; ++k)
        if (r[a.keep[k]] != p[a.keep[k]]) return true;
    return false;
}

__global__ void __launch_bounds__(kFinThreads) unique_count_kernel(const UniqueArgs a) {
    __shared__ uint64_t s_warp[kFinThreads / 32];
    uint32_t lo, hi;
    chunk(a.n, &lo, &hi);
    uint64_t c = 0;
    for (uint32_t i = lo + threadIdx.x; i < hi; i += kFinThreads) c += starts_run(a, i);
    const uint64_t ex = block_exclusive_sum<kFinThreads>(c, s_warp);
    if (threadIdx.x == kFinThreads - 1) a.part[blockIdx.x] = (uint32_t)(ex + c);
}

__global__ void __launch_bounds__(kFinThreads) unique_place_kernel(const UniqueArgs a) {
    __shared__ uint64_t s_warp[kFinThreads / 32];
    __shared__ uint64_t s_carry;
    uint32_t lo, hi;
    chunk(a.n, &lo, &hi);
    if (threadIdx.x == 0) s_carry = a.part[blockIdx.x];
    __syncthreads();
    for (uint32_t base = lo; base < hi; base += kFinThreads) {
        const uint32_t i = base + threadIdx.x;
        const uint64_t m = i < hi ? starts_run(a, i) : 0;
        const uint64_t ex = block_exclusive_sum<kFinThreads>(m, s_warp);
        const uint64_t carry = s_carry;
        if (m) a.out[carry + ex] = sorted_row(a, i);
        __syncthreads();
        if (threadIdx.x == kFinThreads - 1) s_carry = carry + ex + m;
        __syncthreads();
    }
}

// out row j = the required columns of input row idx[start + j] (idx null: row start + j).
__global__ void __launch_bounds__(kFinThreads) project_kernel(const uint32_t* table, int cols,
                                                              const int32_t* keep, int n_keep,
                                                              const uint32_t* idx, uint64_t start,
                                                              uint64_t count, uint32_t* out,
                                                              uint64_t* out_rows) {
    const uint64_t total = count * n_keep;
    for (uint64_t e = blockIdx.x * (uint64_t)kFinThreads + threadIdx.x; e < total;
         e += (uint64_t)gridDim.x * kFinThreads) {
        const uint64_t j = e / n_keep;
        const int k = (int)(e - j * n_keep);
        const uint64_t row = idx ? idx[start + j] : start + j;
        out[e] = table[row * cols + keep[k]];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *out_rows = count;
}

// ---------------------------------------------------------------- BOUND filter
// SPARQLEngine::bound_filter (sparql.hpp:1222-1234) for every BOUND(?x) of a query at once, as
// execute_filter ANDs them (:1356-1376): a row survives when none of the named columns holds
// BLANK_ID, and the survivors keep their order (append_row_to in row order).
struct BoundArgs {
    const uint32_t* table;
    int cols;
    const int32_t* bcols;   // columns that must be bound
    int nb;
    uint32_t n;
    uint32_t* part;         // [grid + 1] survivors per CTA, then their exclusive scan
    uint32_t* out;
};

__device__ __forceinline__ bool row_bound(const BoundArgs& a, uint32_t i) {
    const uint32_t* r = a.table + (uint64_t)i * a.cols;
    for (int k = 0; k < a.nb; ++k)
        if (__ldg(r + a.bcols[k]) == kBlankId) return false;
    return true;
}

__global__ void __launch_bounds__(kFinThreads) bound_count_kernel(const BoundArgs a) {
    __shared__ uint64_t s_warp[kFinThreads / 32];
    uint32_t lo, hi;
    chunk(a.n, &lo, &hi);
    uint64_t c = 0;
    for (uint32_t i = lo + threadIdx.x; i < hi; i += kFinThreads) c += row_bound(a, i);
    const uint64_t ex = block_exclusive_sum<kFinThreads>(c, s_warp);
    if (threadIdx.x == kFinThreads - 1) a.part[blockIdx.x] = (uint32_t)(ex + c);
}

// Each CTA walks its chunk 256 rows at a time; a surviving row goes to its CTA's offset plus the
// survivors before it, and its words are copied by consecutive threads.
__global__ void __launch_bounds__(kFinThreads) bound_place_kernel(const BoundArgs a) {
    __shared__ uint64_t s_warp[kFinThreads / 32];
    __shared__ uint64_t s_carry;
    __shared__ uint32_t s_src[kFinThreads], s_dst[kFinThreads];
    __shared__ uint32_t s_m;
    uint32_t lo, hi;
    chunk(a.n, &lo, &hi);
    if (threadIdx.x == 0) s_carry = a.part[blockIdx.x];
    __syncthreads();
    for (uint32_t base = lo; base < hi; base += kFinThreads) {
        const uint32_t i = base + threadIdx.x;
        const uint64_t m = i < hi ? row_bound(a, i) : 0;
        const uint64_t ex = block_exclusive_sum<kFinThreads>(m, s_warp);
        const uint64_t carry = s_carry;
        if (m) {
            s_src[ex] = i;
            s_dst[ex] = (uint32_t)(carry + ex);
        }
        if (threadIdx.x == kFinThreads - 1) s_m = (uint32_t)(ex + m);
        __syncthreads();
        const uint32_t cnt = s_m;
        for (uint32_t e = threadIdx.x; e < cnt * (uint32_t)a.cols; e += kFinThreads) {
            const uint32_t j = e / a.cols, c = e - j * a.cols;
            a.out[(uint64_t)s_dst[j] * a.cols + c] = __ldg(a.table + (uint64_t)s_src[j] * a.cols + c);
        }
        __syncthreads();
        if (threadIdx.x == 0) s_carry = carry + cnt;
        __syncthreads();
    }
}

}  // namespace

cudaError_t final_kernel_attrs() {
    cudaError_t e = use_max_shared_carveout(scan_rows_kernel);
    if (e == cudaSuccess) e = use_max_shared_carveout(key_kernel);
    if (e == cudaSuccess) e = use_max_shared_carveout(hist_kernel);
    if (e == cudaSuccess) e = use_max_shared_carveout(scan_kernel);
    if (e == cudaSuccess) e = use_max_shared_carveout(radix::digit_rows_kernel);
    if (e == cudaSuccess) e = use_max_shared_carveout(scatter_kernel<true>);
    if (e == cudaSuccess) e = use_max_shared_carveout(scatter_kernel<false>);
    if (e == cudaSuccess) e = use_max_shared_carveout(key_hist_kernel);
    if (e == cudaSuccess) e = use_max_shared_carveout(key_count_kernel);
    if (e == cudaSuccess) e = use_max_shared_carveout(key_write_kernel);
    if (e == cudaSuccess) e = use_max_shared_carveout(unique_count_kernel);
    if (e == cudaSuccess) e = use_max_shared_carveout(unique_place_kernel);
    if (e == cudaSuccess) e = use_max_shared_carveout(project_kernel);
    if (e == cudaSuccess) e = use_max_shared_carveout(bound_count_kernel);
    if (e == cudaSuccess) e = use_max_shared_carveout(bound_place_kernel);
    return e;
}

}  // namespace wk

extern "C" int wk_table_final_process(wk_ctx* ctx, const wk_table* in, const int32_t* keep_cols,
                                      int32_t n_keep, int32_t distinct, int64_t offset, int64_t limit,
                                      wk_table* out) {
    using namespace wk;
    if (!ctx || !in || !out || in == out || (!keep_cols && n_keep) || n_keep < 0 || offset < 0)
        return WK_E_BADARG;
    std::lock_guard<std::mutex> lk(ctx->mu);
    const int cols = in->cols;
    cudaStream_t s = ctx->stream;
    uint64_t R = 0;
    int rrc = table_rows(ctx, in, &R);
    if (rrc) return rrc;
    // a row count past the capacity marks a table whose writing step overflowed: refused before
    // any launch (and before any scratch is sized from it), as wk_table_download refuses it
    if (cols > 0 && R > in->cap / (uint64_t)cols)
        return ctx->fail(WK_E_CORRUPT, "row count beyond table capacity");
    if (R == 0) {   // an empty table is left as it is, columns included (sparql.hpp:1420-1421)
        int rc = ctx->table_reserve(out, 1);
        if (rc) return rc;
        out->cols = cols;
        out->written();
        WKF_CUDA(ctx, cudaMemsetAsync(out->d_rows, 0, 8, s));
        WKF_CUDA(ctx, cudaStreamSynchronize(s));
        return WK_SUCCESS;
    }
    if (n_keep == 0) return ctx->fail(WK_NO_REQUIRED_VAR, "no required variable");
    // tables hold at most 32 columns (the context's column limit); the sort's chunk layout and
    // the order check's row tiles are sized for that
    if (cols > 32) return ctx->fail(WK_E_CAPACITY, "more than 32 columns");
    for (int k = 0; k < n_keep; ++k)
        if (keep_cols[k] < 0 || keep_cols[k] >= cols) return ctx->fail(WK_E_BADARG, "required column out of range");
    if (R >= (1ull << 32)) return ctx->fail(WK_E_CAPACITY, "table too long for the post-pattern stage");
    const uint32_t n = (uint32_t)R;
    const int grid = std::max(1, std::min<int>(ctx->sm_count * 4, (int)((n + 2047) / 2048)));
    // the passes over keys alone: whole tiles for each CTA, and one wave of CTAs (a part
    // that ends within a tile leaves the rest of the CTA idle in it)
    const radix::Split ksplit = radix::split(n, (uint64_t)ctx->sm_count * 5);
    const int hgrid = std::max(grid, ksplit.grid);        // the histogram's rows
    const int pgrid1 = std::max(grid, ctx->sm_count * 8);   // the CTA counts
    // scratch: the required columns, two index arrays, two key arrays (DISTINCT only), the
    // digit histogram, the CTA counts and the distinct total, the column ranges, the digit totals
    const bool sort = distinct && n > 1;
    const size_t keep_bytes = ((size_t)n_keep * 4 + 255) & ~(size_t)255;
    const size_t idx_bytes = ((2 * (size_t)n * 4) + 255) & ~(size_t)255;
    // the two key arrays; once the sort is done the same room holds the table in sorted order
    const size_t key_bytes = sort ? std::max(2 * (size_t)n * 8, (size_t)n * cols * 4) : 0;
    const size_t bytes = keep_bytes + idx_bytes + key_bytes + (size_t)kDigits * hgrid * 4 +
                         ((size_t)pgrid1 + 2) * 4 + (size_t)cols * 8 + (size_t)kDigits * 4 + 64;
    // the context keeps the scratch between calls (grown, never shrunk): an allocation and a
    // cudaFree per call would cost more than the stage's own kernels
    int src = ctx->final_scratch_reserve(bytes);
    if (src) return src;
    char* scratch = static_cast<char*>(ctx->d_final_scratch);
    auto done = [&](int rc) {   // after what was enqueued; a success is one only if that was
        const cudaError_t w = cudaStreamSynchronize(s);
        if (w != cudaSuccess) cudaGetLastError();   // (reported here, not by the next launch)
        return rc == WK_SUCCESS && w != cudaSuccess ? ctx->cuda_fail(w, "post-pattern stage") : rc;
    };
    int32_t* d_keep = reinterpret_cast<int32_t*>(scratch);
    uint32_t* idx0 = reinterpret_cast<uint32_t*>(scratch + keep_bytes);
    uint32_t* idx1 = idx0 + n;
    unsigned long long* key0 = reinterpret_cast<unsigned long long*>(scratch + keep_bytes + idx_bytes);
    unsigned long long* key1 = key0 + (sort ? n : 0);
    uint32_t* hist = reinterpret_cast<uint32_t*>(scratch + keep_bytes + idx_bytes + key_bytes);
    uint32_t* part = hist + (size_t)kDigits * hgrid;
    uint32_t* d_total = part + pgrid1 + 1;
    uint32_t* d_mm = d_total + 1;
    uint32_t* dtot = d_mm + 2 * (size_t)cols;
    cudaError_t e = cudaSuccess;
    const uint32_t* idx = nullptr;   // null: rows in table order
    const uint32_t* table_src = in->d;   // the rows idx refers to (the sorted copy after a sort)
    uint64_t m = n;
    // the columns up to the last required one order and tell apart all that is output
    int cmp = 0;
    for (int k = 0; k < n_keep; ++k) cmp = std::max(cmp, keep_cols[k] + 1);
    bool in_order = false;
    std::vector<uint32_t> mm(2 * (size_t)cols);
    if (sort) {   // a table already in the sort's order keeps it; else each column's range, in signed order
        const uint32_t max_rows = (uint32_t)(kCheckWords / cols - 1);   // cols <= 32: >= 255 rows
        const uint64_t ctas = (uint64_t)ctx->sm_count * 6, turns = (n - 1 + ctas * max_rows - 1) / (ctas * max_rows);
        const uint32_t tile_rows = (uint32_t)std::max<uint64_t>(255, (n - 1 + ctas * turns - 1) / (ctas * turns));
        const int cgrid = (int)std::min<uint64_t>(ctas, ((uint64_t)n - 1 + tile_rows - 1) / tile_rows);
        // (d_total is free until the scan: the order check's word, with the ranges behind it)
        if ((e = cudaMemsetAsync(d_total, 0xFF, (1 + mm.size()) * 4, s)) == cudaSuccess) {
            scan_rows_kernel<<<cgrid, kFinThreads, 0, s>>>(in->d, cols, cmp, n, tile_rows, d_total, d_mm);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(ctx->h_small, d_total, (1 + mm.size()) * 4, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return done(ctx->cuda_fail(e, "order check"));
        in_order = ctx->h_small[0] != 0;
        for (int c = 0; c < cols; ++c) {
            mm[2 * c] = ctx->h_small[1 + 2 * c];
            mm[2 * c + 1] = ~ctx->h_small[2 + 2 * c];
        }
        int bits = 0;
        for (int c = 0; c < cmp; ++c)
            if (mm[2 * c] < mm[2 * c + 1]) bits += 32 - __builtin_clz(mm[2 * c + 1] - mm[2 * c]);
        // one key per row holds all that matters of it (bits > 0: rows equal in these columns are in order)
        if (!in_order && bits <= 64 && n_keep <= 32) {
            ChunkDesc cd{};
            KeyCols kc{};
            kc.n = n_keep;
            std::vector<int> shift_of(cmp, 0), bits_of(cmp, 0);
            int left = bits;
            for (int c = 0; c < cmp; ++c) {
                if (mm[2 * c] >= mm[2 * c + 1]) continue;   // constant: orders nothing
                bits_of[c] = 32 - __builtin_clz(mm[2 * c + 1] - mm[2 * c]);
                left -= bits_of[c];
                shift_of[c] = left;
                cd.ccol[cd.nc] = c;
                cd.cbits[cd.nc] = bits_of[c];
                cd.cmin[cd.nc++] = mm[2 * c];
            }
            for (int k = 0; k < n_keep; ++k) {
                const int c = keep_cols[k];
                kc.shift[k] = shift_of[c];
                kc.bits[k] = bits_of[c];
                kc.lowest[k] = mm[2 * c];
                if (bits_of[c]) kc.mask |= (unsigned long long)(0xFFFFFFFFu >> (32 - bits_of[c])) << shift_of[c];
            }
            unsigned long long *ka = key0, *kb = key1;
            for (int shift = 0; shift < bits; shift += 8) {
                SortPass p{ka, nullptr, kb, nullptr, shift, n, ksplit.per_cta, hist, dtot};
                if (shift == 0)
                    key_hist_kernel<<<ksplit.grid, kFinThreads, 0, s>>>(in->d, cols, cd, p, ka);
                else
                    hist_kernel<<<ksplit.grid, kFinThreads, 0, s>>>(p);
                radix::digit_rows_kernel<<<kDigits, kFinThreads, 0, s>>>(hist, (uint32_t)ksplit.grid, dtot);
                scatter_kernel<false><<<ksplit.grid, kFinThreads, 0, s>>>(p);
                std::swap(ka, kb);
            }
            // whole rounds of key_write_kernel for each CTA, and one wave of CTAs
            const uint32_t rounds = (uint32_t)(((uint64_t)n + 1023) / 1024);
            const uint32_t cta_rounds = (rounds + ctx->sm_count * 8 - 1) / (ctx->sm_count * 8);
            const int ugrid = (int)((rounds + cta_rounds - 1) / cta_rounds);
            KeyRuns u{ka, n, cta_rounds * 1024, part};
            key_count_kernel<<<ugrid, kFinThreads, 0, s>>>(u, kc);
            scan_kernel<<<1, 1024, 0, s>>>(part, (uint32_t)ugrid, d_total);
            // written right away where the room that `out` has turns out to be enough
            auto write = [&] {
                key_write_kernel<<<ugrid, kFinThreads, 0, s>>>(u, kc, d_total, (uint64_t)offset, limit, out->d,
                                                               out->cap, out->d_rows);
                return cudaGetLastError();
            };
            if (!out->d || !out->d_rows) {   // (a table that an earlier call could not grow)
                const int rc = ctx->table_reserve(out, 1);
                if (rc) return done(rc);
            }
            out->written();
            if ((e = write()) != cudaSuccess) return done(ctx->cuda_fail(e, "distinct launches"));
            if ((e = cudaMemcpyAsync(ctx->h_small, d_total, 4, cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
                (e = cudaStreamSynchronize(s)) != cudaSuccess)
                return done(ctx->cuda_fail(e, "distinct count"));
            m = ctx->h_small[0];
            const uint64_t start = std::min<uint64_t>((uint64_t)offset, m);
            const uint64_t count = limit < 0 ? m - start : std::min<uint64_t>((uint64_t)limit, m - start);
            if (count * n_keep > out->cap) {
                const int rc = ctx->table_reserve(out, std::max<uint64_t>(count * n_keep, 1));
                if (rc) return done(rc);
                if ((e = write()) != cudaSuccess || (e = cudaStreamSynchronize(s)) != cudaSuccess)
                    return done(ctx->cuda_fail(e, "distinct rows"));
            }
            out->cols = n_keep;
            out->rows = count;
            out->rows_known = true;
            return WK_SUCCESS;
        }
    }
    e = cudaMemcpyAsync(d_keep, keep_cols, (size_t)n_keep * 4, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return done(ctx->cuda_fail(e, "post-pattern columns"));
    if (sort) {
        const uint32_t* sorted = nullptr;   // the sorted row order (null: the table's own)
        if (!in_order) {
            // chunks of columns, last column first; a constant column orders nothing and is left out
            std::vector<ChunkDesc> chunks;
            std::vector<int> chunk_bits;
            ChunkDesc cur{};
            int cur_bits = 0;
            auto flush = [&]() {
                if (!cur.nc) return;
                // columns were added least significant first; the key wants the most significant first
                std::reverse(cur.ccol, cur.ccol + cur.nc);
                std::reverse(cur.cbits, cur.cbits + cur.nc);
                std::reverse(cur.cmin, cur.cmin + cur.nc);
                chunks.push_back(cur);
                chunk_bits.push_back(cur_bits);
                cur = ChunkDesc{};
                cur_bits = 0;
            };
            for (int c = cmp - 1; c >= 0; --c) {
                const uint32_t lo = mm[2 * c], hi = mm[2 * c + 1];
                if (lo >= hi) continue;
                const int b = 32 - __builtin_clz(hi - lo);
                if (cur_bits + b > 64) flush();
                cur.ccol[cur.nc] = c;
                cur.cbits[cur.nc] = b;
                cur.cmin[cur.nc] = lo;
                cur.nc++;
                cur_bits += b;
            }
            flush();
            const int kgrid = std::max(1, std::min(ctx->sm_count * 8, (int)((n + 255) / 256)));
            uint32_t* ia = idx0;
            uint32_t* ib = idx1;
            unsigned long long* ka = key0;
            unsigned long long* kb = key1;
            for (size_t k = 0; k < chunks.size(); ++k) {
                key_kernel<<<kgrid, kFinThreads, 0, s>>>(in->d, cols, chunks[k], sorted, n, ka, ia);
                for (int shift = 0; shift < chunk_bits[k]; shift += 8) {
                    SortPass p{ka, ia, kb, ib, shift, n, (uint32_t)(((uint64_t)n + grid - 1) / grid), hist, dtot};
                    hist_kernel<<<grid, kFinThreads, 0, s>>>(p);
                    radix::digit_rows_kernel<<<kDigits, kFinThreads, 0, s>>>(hist, (uint32_t)grid, dtot);
                    scatter_kernel<true><<<grid, kFinThreads, 0, s>>>(p);
                    std::swap(ka, kb);
                    std::swap(ia, ib);
                }
                sorted = ia;
                std::swap(ia, ib);   // the next chunk's keys go to the other index array
            }
        }
        uint32_t* kept = sorted == idx0 ? idx1 : idx0;
        // rows gathered into sorted order once (into the key arrays' room): the compaction then
        // compares consecutive rows and the projection reads the kept ones from this copy
        const uint32_t* rows_src = in->d;
        if (sorted) {
            uint32_t* sorted_rows = reinterpret_cast<uint32_t*>(key0);
            const int ggrid = std::max(1, std::min<int>(ctx->sm_count * 8, (int)(((uint64_t)n * cols + 255) / 256)));
            gather_rows_kernel<<<ggrid, kFinThreads, 0, s>>>(in->d, cols, sorted, n, sorted_rows);
            rows_src = sorted_rows;
            sorted = nullptr;
        }
        UniqueArgs u{rows_src, cols, d_keep, n_keep, sorted, n, part, kept};
        unique_count_kernel<<<grid, kFinThreads, 0, s>>>(u);
        scan_kernel<<<1, 1024, 0, s>>>(part, (uint32_t)grid, d_total);
        unique_place_kernel<<<grid, kFinThreads, 0, s>>>(u);
        if ((e = cudaGetLastError()) != cudaSuccess) return done(ctx->cuda_fail(e, "distinct launches"));
        uint32_t h_total = 0;
        if ((e = cudaMemcpyAsync(&h_total, d_total, 4, cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
            (e = cudaStreamSynchronize(s)) != cudaSuccess)
            return done(ctx->cuda_fail(e, "distinct count"));
        m = h_total;
        idx = kept;
        table_src = rows_src;
    }
    const uint64_t start = std::min<uint64_t>((uint64_t)offset, m);
    const uint64_t count = limit < 0 ? m - start : std::min<uint64_t>((uint64_t)limit, m - start);
    const int rc = ctx->table_reserve(out, std::max<uint64_t>(count * n_keep, 1));
    if (rc) return done(rc);
    out->cols = n_keep;
    out->written();
    const int pgrid = std::max(1, std::min<int>(ctx->sm_count * 8, (int)((count * n_keep + 255) / 256)));
    project_kernel<<<pgrid, kFinThreads, 0, s>>>(table_src, cols, d_keep, n_keep, idx, start, count, out->d,
                                                 out->d_rows);
    if ((e = cudaGetLastError()) != cudaSuccess) return done(ctx->cuda_fail(e, "projection launch"));
    const int wrc = done(WK_SUCCESS);
    if (wrc) return wrc;
    out->rows = count;
    out->rows_known = true;
    return WK_SUCCESS;
}

extern "C" int wk_table_filter_bound(wk_ctx* ctx, const wk_table* in, const int32_t* bound_cols,
                                     int32_t n_bound, wk_table* out) {
    using namespace wk;
    if (!ctx || !in || !out || in == out || (!bound_cols && n_bound) || n_bound < 0) return WK_E_BADARG;
    std::lock_guard<std::mutex> lk(ctx->mu);
    if (n_bound > 64) return ctx->fail(WK_E_BADARG, "at most 64 bound columns");
    const int cols = in->cols;
    cudaStream_t s = ctx->stream;
    uint64_t R = 0;
    int rc = table_rows(ctx, in, &R);
    if (rc) return rc;
    if (cols > 0 && R > in->cap / (uint64_t)cols)
        return ctx->fail(WK_E_CORRUPT, "row count beyond table capacity");
    for (int k = 0; k < n_bound; ++k)
        if (bound_cols[k] < 0 || bound_cols[k] >= cols) return ctx->fail(WK_E_BADARG, "bound column out of range");
    if (R >= (1ull << 32)) return ctx->fail(WK_E_CAPACITY, "table too long for the filter stage");
    rc = ctx->table_reserve(out, std::max<uint64_t>(R * (uint64_t)std::max(cols, 1), 1));
    if (rc) return rc;
    out->cols = cols;
    out->written();
    if (R == 0 || n_bound == 0) {   // nothing to drop: the table as it is
        if (R) WKF_CUDA(ctx, cudaMemcpyAsync(out->d, in->d, R * (uint64_t)cols * 4, cudaMemcpyDeviceToDevice, s));
        WKF_CUDA(ctx, cudaMemcpyAsync(out->d_rows, in->d_rows, 8, cudaMemcpyDeviceToDevice, s));
        WKF_CUDA(ctx, cudaStreamSynchronize(s));
        return WK_SUCCESS;
    }
    const uint32_t n = (uint32_t)R;
    const int grid = std::max(1, std::min<int>(ctx->sm_count * 4, (int)((n + 2047) / 2048)));
    const size_t bytes = 256 + ((size_t)grid + 2) * 4 + 64;
    int src = ctx->final_scratch_reserve(bytes);
    if (src) return src;
    char* scratch = static_cast<char*>(ctx->d_final_scratch);
    auto done = [&](int code) {
        const cudaError_t w = cudaStreamSynchronize(s);
        if (w != cudaSuccess) cudaGetLastError();
        return code == WK_SUCCESS && w != cudaSuccess ? ctx->cuda_fail(w, "filter stage") : code;
    };
    int32_t* d_cols = reinterpret_cast<int32_t*>(scratch);
    uint32_t* part = reinterpret_cast<uint32_t*>(scratch + 256);
    uint32_t* d_total = part + grid + 1;
    cudaError_t e = cudaMemcpyAsync(d_cols, bound_cols, (size_t)n_bound * 4, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return done(ctx->cuda_fail(e, "filter columns"));
    BoundArgs b{in->d, cols, d_cols, n_bound, n, part, out->d};
    bound_count_kernel<<<grid, kFinThreads, 0, s>>>(b);
    scan_kernel<<<1, 1024, 0, s>>>(part, (uint32_t)grid, d_total);
    bound_place_kernel<<<grid, kFinThreads, 0, s>>>(b);
    if ((e = cudaGetLastError()) != cudaSuccess) return done(ctx->cuda_fail(e, "filter launches"));
    uint32_t h_total = 0;
    if ((e = cudaMemcpyAsync(&h_total, d_total, 4, cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
        (e = cudaStreamSynchronize(s)) != cudaSuccess)
        return done(ctx->cuda_fail(e, "filter count"));
    ctx->h_rows[1] = h_total;
    e = cudaMemcpyAsync(out->d_rows, ctx->h_rows + 1, 8, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return done(ctx->cuda_fail(e, "filter row count"));
    return done(WK_SUCCESS);
}
