// Flat passes of a batch level: count -> place -> expand.
//
// The tile launch (wk_explore.cu) keeps a whole level in one persistent launch, which suits many
// small tables but pays per-tile barriers and look-back waits, and runs at the occupancy its shared
// memory allows.  A level whose tables are large together can run (knob 5) as three short launches
// at full occupancy instead:
//   1. count: one thread per input row looks its step's key up, records the row's output count
//      (list size for a start or known_to_unknown, 0/1 membership for the filters) and its list
//      offset; each CTA owns a contiguous chunk of rows and publishes the chunk total, and the last
//      CTA to finish scans the totals, checks the output capacity (overflow sets kErrOverflow and
//      the rows needed, as the tile launch does) and sets the row count;
//   2. place: each CTA scans its chunk into per-row output positions and records the queries'
//      ranges; filters copy their surviving rows straight to the output here;
//   3. expand: the output rows are split evenly over the CTAs; each CTA finds its first input row
//      by a 32-way search of the positions and writes its rows in row-major then edge order
//      (sparql.hpp:328-370), consecutive threads on consecutive rows.
// Row counts are read on the device, so the launches chain without a host round trip and can be
// captured in a graph.
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/wukong_b200.h"
#include "wk_device.cuh"
#include "wk_flat.h"

namespace wk {
namespace {
using namespace dev;

constexpr int kFlatThreads = 256;
constexpr int kWindow = 256;   // input rows staged per expand round
__device__ __forceinline__ void chunk_of(uint64_t R, uint64_t* lo, uint64_t* hi) {
    const uint64_t chunk = (R + gridDim.x - 1) / gridDim.x;
    *lo = min(R, (uint64_t)blockIdx.x * chunk);
    *hi = min(R, *lo + chunk);
}

__device__ __forceinline__ uint64_t block_sum(uint64_t x, uint64_t* s_warp) {
    const uint64_t ex = block_exclusive_sum<kFlatThreads>(x, s_warp);
    __shared__ uint64_t s_tot;
    if (threadIdx.x == kFlatThreads - 1) s_tot = ex + x;
    __syncthreads();
    const uint64_t t = s_tot;
    __syncthreads();
    return t;
}

// Called by every thread of a count CTA once its chunk total is in part[blockIdx.x]: true in the
// last CTA to get here, which then runs the scan (and leaves the counter at 0 for the next pass).
__device__ __forceinline__ bool last_count_cta(StepCtl* ctl) {
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        s_last = atomicAdd(&ctl->flat_done, 1u) == gridDim.x - 1;
        if (s_last) ctl->flat_done = 0;
    }
    __syncthreads();
    if (s_last) __threadfence();
    return s_last != 0;
}

constexpr int kCountCtas = 8;   // count CTAs per SM (32 registers): resident warps set the lookups' rate

// Every row carries its owner query, whose step at this level (start, known_to_unknown,
// known_to_known, known_to_const or done) comes from the level's descriptor array.  Rows keep
// their order, so each query's output rows stay contiguous and its range is recorded from the
// runs of its rows.

__device__ __forceinline__ uint64_t level_rows(const FlatLevelArgs& a) {
    if (a.virtual_rows) return a.n_queries;
    uint64_t R = *(volatile const uint64_t*)a.in_rows;
    return R > a.in_cap_rows ? 0 : R;   // past capacity: the step before overflowed
}

__device__ __forceinline__ uint32_t level_owner(const FlatLevelArgs& a, uint64_t r) {
    return a.virtual_rows ? (uint32_t)r : __ldg(a.owner_in + r);
}

// Scan of the count CTAs' chunk totals, run by the last count CTA to finish: part[] becomes the
// exclusive scan, part[nparts] the total; the capacity check sets the output row count or the
// overflow bit.  The totals of other CTAs are read from L2 (they were written by other SMs).
__device__ void flat_level_scan_parts(const FlatLevelArgs& a, uint32_t nparts, uint64_t R,
                                      uint64_t* s_warp) {
    __shared__ uint64_t s_carry;
    if (threadIdx.x == 0) s_carry = 0;
    __syncthreads();
    for (uint32_t r0 = 0; r0 < nparts; r0 += kFlatThreads) {
        const uint32_t i = r0 + threadIdx.x;
        const uint64_t x = i < nparts ? __ldcg((const unsigned long long*)a.part + i) : 0;
        const uint64_t ex = block_exclusive_sum<kFlatThreads>(x, s_warp);
        const uint64_t carry = s_carry;
        if (i < nparts) a.part[i] = carry + ex;
        __syncthreads();
        if (threadIdx.x == kFlatThreads - 1) s_carry = carry + ex + x;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const uint64_t total = s_carry;
        a.part[nparts] = total;
        a.pos[R] = total;
        if (total > a.out_cap_rows) {
            atomicOr(&a.ctl->err, kErrOverflow);
            atomicMax(&a.ctl->need, (unsigned long long)total);
            *a.out_rows = 0;
        } else {
            *a.out_rows = total;
        }
    }
}

__global__ void __launch_bounds__(kFlatThreads, kCountCtas) flat_level_count_kernel(const FlatLevelArgs a) {
    __shared__ uint64_t s_warp[kFlatThreads / 32];
    const uint64_t R = level_rows(a);
    uint64_t lo, hi;
    chunk_of(R, &lo, &hi);
    uint64_t sum = 0, sd = 0, alg = 0;
    for (uint64_t r = lo + threadIdx.x; r < hi; r += kFlatThreads) {
        const StepDesc* d = a.desc + level_owner(a, r);
        const uint32_t op = d->op;
        const uint32_t* row = a.in + r * (uint64_t)a.w_in;
        const SegDesc* sg = a.store.segs + d->seg;
        bool valid = op != kXDone;
        uint64_t key = 0;
        uint32_t target = d->end_const;
        if (valid && op == kXStart) {
            key = d->start_key;
        } else if (valid && (op == kXC2K || op == kXI2K)) {   // one list for every row
            key = d->start_key;
            target = __ldg(row + d->ce);
        } else if (valid) {
            const uint32_t cur = __ldg(row + d->cs);
            if (op == kXK2K) target = __ldg(row + d->ce);
            if (cur == kBlankId) valid = false;
            if (op == kXK2U && d->type_index) {
                // get_index(cur, IN) (sparql.hpp:342-345); only 17-bit ids can be keys
                key = make_key(0, cur, kIn);
                sg = a.store.segs + a.seg_index[kIn];
                if (cur >= (1u << kNbitsIdx)) valid = false;
            } else {
                key = make_key(cur, d->pid, d->dir);
                if (cur == 0) sg = a.store.segs + (d->dir & 1 ? a.seg_index[1] : a.seg_index[0]);   // vid 0 names the index
            }
        }
        uint64_t off = 0, deg = 0;
        if (valid && sg->num_buckets != 0 && key != 0) {
            const uint64_t p = seg_lookup(a.store, *sg, key, (uint32_t)key_vid(key), &a.ctl->err);
            list_of_ptr(p, a.store.n_edges, &a.ctl->err, &off, &deg);
            if (op == kXI2K) {
                uint64_t s_lo, s_hi;
                mt_slice(d->mt, deg, &s_lo, &s_hi);
                off += s_lo;
                deg = s_hi - s_lo;
            }
        }
        const bool filt = is_filter_op(op);
        uint32_t c = (uint32_t)deg;
        if (filt) c = (valid && deg && thread_member(a.store.edges, off, deg, target, a.sorted_lists != 0)) ? 1u : 0u;
        if (!valid) c = 0;
        a.pos[r] = c;   // the count; flat_level_place_kernel turns it into the row's position
        a.off[r] = off;
        sum += c;
        if (valid) {
            const uint32_t cin = op == kXStart ? 0u : d->cin;
            sd += deg;
            alg += cin * 4ull + 16 + deg * 4 + (uint64_t)c * d->cout * 4;
        }
    }
    sum = block_sum(sum, s_warp);
    sd = block_sum(sd, s_warp);
    alg = block_sum(alg, s_warp);
    if (threadIdx.x == 0) {
        a.part[blockIdx.x] = sum;
        if (alg) {
            atomicAdd(&a.ctl->sum_deg, (unsigned long long)sd);
            atomicAdd(&a.ctl->alg_bytes, (unsigned long long)alg);
        }
    }
    if (last_count_cta(a.ctl)) flat_level_scan_parts(a, gridDim.x, R, s_warp);
}

__global__ void __launch_bounds__(kFlatThreads) flat_level_place_kernel(const FlatLevelArgs a, uint32_t nparts) {
    __shared__ uint64_t s_warp[kFlatThreads / 32];
    __shared__ uint64_t s_carry;
    const uint64_t R = level_rows(a);
    if (a.part[nparts] > a.out_cap_rows) return;
    uint64_t lo, hi;
    chunk_of(R, &lo, &hi);
    if (threadIdx.x == 0) s_carry = a.part[blockIdx.x];
    __syncthreads();
    for (uint64_t r0 = lo; r0 < hi; r0 += kFlatThreads) {
        const uint64_t r = r0 + threadIdx.x;
        const uint64_t c = r < hi ? a.pos[r] : 0;
        const uint64_t ex = block_exclusive_sum<kFlatThreads>(c, s_warp);
        const uint64_t p = s_carry + ex;
        if (r < hi) {
            a.pos[r] = p;
            const uint32_t q = level_owner(a, r);
            // the query's output range: (end - start) of every run of its rows
            const bool first = r == lo || level_owner(a, r - 1) != q;
            const bool last = r + 1 == hi || level_owner(a, r + 1) != q;
            if (first) {
                atomicMin(a.qfirst + q, (unsigned long long)p);
                atomicAdd(a.qcount + q, (unsigned long long)(0 - p));
            }
            if (last) atomicAdd(a.qcount + q, (unsigned long long)(p + c));
            const uint32_t op = a.desc[q].op;
            if (c && is_filter_op(op)) {   // a surviving row keeps its columns
                const int cin = a.desc[q].cin;
                const uint32_t* src = a.in + r * (uint64_t)a.w_in;
                uint32_t* dst = a.out + p * (uint64_t)a.w_out;
                for (int k = 0; k < cin; ++k) dst[k] = __ldg(src + k);
                a.owner_out[p] = q;
            }
        }
        __syncthreads();
        if (threadIdx.x == kFlatThreads - 1) s_carry = p + c;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kFlatThreads) flat_level_expand_kernel(const FlatLevelArgs a) {
    __shared__ uint64_t s_pos[kWindow + 1];
    __shared__ uint64_t s_off[kWindow];
    __shared__ uint32_t s_q[kWindow];
    __shared__ int32_t s_ecol[kWindow];   // column the edge goes to; -1: not an expanding row
    __shared__ uint64_t s_i0;
    const uint64_t R = level_rows(a);
    const uint64_t total = a.pos[R];
    if (total > a.out_cap_rows || total == 0) return;
    const uint64_t per = (total + gridDim.x - 1) / gridDim.x;
    const uint64_t j0 = min(total, (uint64_t)blockIdx.x * per), j1 = min(total, j0 + per);
    if (j0 >= j1) return;
    if (threadIdx.x < 32) {   // the last r with pos[r] <= j0 (pos[R] = total > j0)
        uint64_t lo = 0, hi = R;
        while (hi - lo > 1) {
            const uint64_t step = (hi - lo + 31) / 32;
            const uint64_t probe = min(hi, lo + (uint64_t)(threadIdx.x + 1) * step);
            const bool le = probe < hi && a.pos[probe] <= j0;
            const unsigned m = __ballot_sync(0xffffffffu, le);
            const int k = m ? 31 - __clz(m) : -1;
            const uint64_t nlo = k >= 0 ? min(hi, lo + (uint64_t)(k + 1) * step) : lo;
            const uint64_t nhi = min(hi, nlo + step);
            lo = nlo;
            hi = max(nhi, lo + 1);
        }
        if (threadIdx.x == 0) s_i0 = lo;
    }
    __syncthreads();
    const int wo = a.w_out;
    uint64_t i = s_i0;
    uint64_t j = j0;
    while (j < j1 && i < R) {
        const uint64_t n = min((uint64_t)kWindow, R - i);
        for (int t = threadIdx.x; t <= (int)n; t += kFlatThreads) s_pos[t] = a.pos[i + t];
        for (int t = threadIdx.x; t < (int)n; t += kFlatThreads) {
            // the window's rows once: list offset, owner, and where its step puts the edge
            s_off[t] = a.off[i + t];
            const uint32_t q = level_owner(a, i + t);
            s_q[t] = q;
            const StepDesc* d = a.desc + q;
            const uint32_t op = d->op;
            s_ecol[t] = op == kXStart ? 0 : op == kXK2U ? (int32_t)d->cin : -1;   // filters: -1
        }
        __syncthreads();
        const uint64_t wend = min(j1, s_pos[n]);
        constexpr int U = 4;   // output rows per thread with their neighbour loads in flight
        for (uint64_t jb = j + threadIdx.x; jb < wend; jb += (uint64_t)U * kFlatThreads) {
            int row[U];
            uint32_t nb[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint64_t jj = jb + (uint64_t)u * kFlatThreads;
                row[u] = -1;
                if (jj >= wend) continue;
                int lo = 0, hi = (int)n;   // last t with s_pos[t] <= jj
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (s_pos[mid] <= jj) lo = mid; else hi = mid;
                }
                if (s_ecol[lo] < 0) continue;   // filters wrote their rows already
                row[u] = lo;
                nb[u] = list_at(a.store.edges, s_off[lo], jj - s_pos[lo]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (row[u] < 0) continue;
                const uint64_t jj = jb + (uint64_t)u * kFlatThreads;
                const int lo = row[u], ecol = s_ecol[lo];
                const uint32_t* src = a.in + (i + lo) * (uint64_t)a.w_in;
                uint32_t* dst = a.out + jj * (uint64_t)wo;
                for (int k = 0; k < ecol; ++k) dst[k] = __ldg(src + k);
                dst[ecol] = nb[u];
                a.owner_out[jj] = s_q[lo];
            }
        }
        j = max(j, wend);
        i += n;
        __syncthreads();
    }
}

}  // namespace

int flat_grid(int sm_count) { return sm_count * (2048 / kFlatThreads); }

cudaError_t launch_flat_level(const FlatLevelArgs& a, int grid, cudaStream_t s) {
    flat_level_count_kernel<<<grid, kFlatThreads, 0, s>>>(a);   // its last CTA scans the totals
    flat_level_place_kernel<<<grid, kFlatThreads, 0, s>>>(a, (uint32_t)grid);
    flat_level_expand_kernel<<<grid, kFlatThreads, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t flat_kernel_attrs() {
    cudaError_t e;
    if ((e = use_max_shared_carveout(flat_level_count_kernel)) != cudaSuccess) return e;
    if ((e = use_max_shared_carveout(flat_level_place_kernel)) != cudaSuccess) return e;
    return use_max_shared_carveout(flat_level_expand_kernel);
}

}  // namespace wk
