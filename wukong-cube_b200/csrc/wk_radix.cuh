// Parts of a stable 8-bit counting pass by CTAs of 256 threads, shared by the DISTINCT sort
// (wk_final.cu) and the store build's sorts (wk_gbuild.cu).  A pass counts each CTA's digits into a
// histogram (digit-major: one row of `grid` words per digit), scans the rows (digit_rows), and
// scatters (radix_scatter).
#pragma once
#include "wk_device.cuh"

namespace wk {
namespace {
namespace radix {

constexpr int kThreads = 256, kWarps = kThreads / 32;
constexpr int kDigits = 256;                  // one thread per digit
constexpr int kPer = 8;                       // elements per thread per tile
constexpr int kTile = kThreads * kPer;        // 2,048

// Offsets of a pass: digit d of CTA b starts at the elements of smaller digits plus the digit-d
// elements of CTAs before b.  CTA d of this launch scans digit d's row of hist in place into
// exclusive offsets within the digit, with coalesced loads, and writes the digit's total to dtot[d];
// each scatter CTA then adds the elements of smaller digits (an exclusive scan of dtot) itself.
__global__ void __launch_bounds__(kThreads) digit_rows_kernel(uint32_t* hist, uint32_t grid, uint32_t* dtot) {
    __shared__ uint64_t s_warp[kWarps];
    __shared__ uint64_t s_carry;
    uint32_t* row = hist + (size_t)blockIdx.x * grid;
    if (threadIdx.x == 0) s_carry = 0;
    __syncthreads();
    constexpr uint32_t kWords = 4;   // a row of a full grid in one round
    for (uint32_t b0 = 0; b0 < grid; b0 += kWords * kThreads) {
        const uint32_t b = b0 + kWords * threadIdx.x;
        uint32_t x[kWords], sum = 0;
#pragma unroll
        for (uint32_t j = 0; j < kWords; ++j) x[j] = b + j < grid ? row[b + j] : 0;
#pragma unroll
        for (uint32_t j = 0; j < kWords; ++j) sum += x[j];
        const uint64_t ex = dev::block_exclusive_sum<kThreads>(sum, s_warp);
        const uint64_t carry = s_carry;
        uint32_t at = (uint32_t)(carry + ex);
#pragma unroll
        for (uint32_t j = 0; j < kWords; ++j) {
            if (b + j < grid) row[b + j] = at;
            at += x[j];
        }
        __syncthreads();
        if (threadIdx.x == kThreads - 1) s_carry = carry + ex + sum;
        __syncthreads();
    }
    if (threadIdx.x == 0) dtot[blockIdx.x] = (uint32_t)s_carry;
}

template <bool kVal>
struct Tile {
    uint32_t cnt[kWarps][kDigits];
    uint32_t peers[kWarps][kDigits];
    uint32_t off[kDigits];
    unsigned long long key[kTile];
    uint32_t val[kVal ? kTile : 1];
    uint64_t warp[kWarps];
};

// Stable scatter of a CTA's elements [lo, hi) in 2,048-element tiles, keys alone or with 32-bit
// values; `run` (thread d) is digit d's first place for this CTA, digit(key, value) an element's.
// Warp w takes elements [w * 256, w * 256 + 256) of the tile in 8 rounds of 32 consecutive ones, so
// the warp's rounds follow the elements' order.  Within a round, an element's rank among the lanes
// with its digit comes from a mask per digit in shared memory, into which the lanes set their bits
// (a match takes time with the number of different digits, 32 us a pass of eight bits where one
// with a third of the digits took 17; eight ballots were bound by their own pipe at 24), and the
// warp's running count of each digit (updated by one lane per digit) gives its place in the warp;
// one barrier then turns the warps' counts into per-warp digit offsets.  The tile is placed in
// shared memory sorted by digit (stable), and then written out in that order, consecutive threads
// on consecutive elements, so each digit's run goes to global memory in contiguous stores.  Bound by
// the shared-memory chain within a tile and its barriers: 3,000,000 keys alone take 22 us a pass
// (with row indices and a match it took 35).
template <bool kVal, class Digit>
__device__ __forceinline__ void radix_scatter(Tile<kVal>& s, const unsigned long long* key_in,
                                              const uint32_t* val_in, unsigned long long* key_out,
                                              uint32_t* val_out, uint64_t lo, uint64_t hi, uint32_t run,
                                              Digit digit) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int w = 0; w < kWarps; ++w) s.peers[w][threadIdx.x] = 0;
    for (uint64_t base = lo; base < hi; base += kTile) {
        for (int w = 0; w < kWarps; ++w) s.cnt[w][threadIdx.x] = 0;
        __syncthreads();
        unsigned long long key[kPer];
        uint32_t val[kPer], dg[kPer], at[kPer];
        const uint64_t wbase = base + (uint32_t)warp * (32 * kPer);
#pragma unroll
        for (int r = 0; r < kPer; ++r) {
            const uint64_t i = wbase + r * 32 + lane;
            const bool live = i < hi;
            key[r] = live ? key_in[i] : 0;
            val[r] = kVal && live ? val_in[i] : 0;
            dg[r] = live ? digit(key[r], val[r]) : (uint32_t)kDigits;
        }
#pragma unroll
        for (int r = 0; r < kPer; ++r) {
            const bool live = dg[r] < kDigits;
            if (live) atomicOr(&s.peers[warp][dg[r]], 1u << lane);
            __syncwarp();
            const unsigned peers = live ? s.peers[warp][dg[r]] : 0;   // the lanes with this lane's digit
            const int rank = __popc(peers & ((1u << lane) - 1));
            at[r] = live ? s.cnt[warp][dg[r]] + rank : 0;
            __syncwarp();
            if (live && rank == 0) {
                s.cnt[warp][dg[r]] += __popc(peers);
                s.peers[warp][dg[r]] = 0;
            }
            __syncwarp();
        }
        __syncthreads();
        uint32_t cnt[kWarps], tile_cnt = 0;   // per digit (thread = digit): prefix over the warps
#pragma unroll
        for (int w = 0; w < kWarps; ++w) cnt[w] = s.cnt[w][threadIdx.x];
#pragma unroll
        for (int w = 0; w < kWarps; ++w) tile_cnt += cnt[w];
        // the tile sorted by digit in shared memory: digit d's elements start at tbase, warp w's
        // at cnt[w][d]; off[d] takes a place in the tile to its place in the output
        const uint32_t tbase = (uint32_t)dev::block_exclusive_sum<kThreads>(tile_cnt, s.warp);
        s.off[threadIdx.x] = run - tbase;
        run += tile_cnt;
        uint32_t wat = tbase;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            s.cnt[w][threadIdx.x] = wat;
            wat += cnt[w];
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kPer; ++r) {
            if (dg[r] >= kDigits) continue;
            const uint32_t lp = s.cnt[warp][dg[r]] + at[r];
            s.key[lp] = key[r];
            if constexpr (kVal) s.val[lp] = val[r];
        }
        __syncthreads();
        // consecutive threads write consecutive elements: each digit's run goes out contiguous
        const uint32_t m = (uint32_t)min((uint64_t)kTile, hi - base);
        for (uint32_t j = threadIdx.x; j < m; j += kThreads) {
            const unsigned long long k = s.key[j];
            const uint32_t v = kVal ? s.val[j] : 0;
            const uint32_t pos = s.off[digit(k, v)] + j;
            key_out[pos] = k;
            if constexpr (kVal) val_out[pos] = v;
        }
        __syncthreads();
    }
}

// Elements of a CTA and CTAs of a pass over n: whole tiles, at most `ctas` CTAs.
struct Split {
    uint32_t per_cta;
    int grid;
};
inline Split split(uint64_t n, uint64_t ctas) {
    const uint64_t tiles = (n + kTile - 1) / kTile, each = (tiles + ctas - 1) / ctas;
    if (!tiles) return {kTile, 1};
    return {(uint32_t)(each * kTile), (int)((tiles + each - 1) / each)};
}

}  // namespace radix
}  // namespace
}  // namespace wk
