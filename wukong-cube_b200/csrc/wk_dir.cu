// Load-time passes over a store on the device.
//
// A key table in the reference's layout spreads a segment's keys over 128-byte buckets by hash:
// a probe of a distinct key moves a whole DRAM line for the 16 bytes it reads, however near the
// vertex ids are to each other.  Wukong's ids are dense (its string server hands them out in
// order of appearance), so each (predicate, direction) segment also gets a directory by vertex id
// on the device: one 8-byte block per 32 ids (which of them have a key, and where the first one's
// word is) and the keys' words in vertex order: their pointer words, or, for a segment whose lists
// all have one entry, those entries.  A lookup reads its block and, where the bit is set, one word.
// Neighbouring vertices share both, absent keys are settled by the bit, and at 10,000 organisations
// a segment's blocks (11 MB) stay in L2.  The words are the slots' own, so a lookup answers what
// the probe answers; segments whose ids are too thin for
// one (see dir_plan in wk_ctx.cpp) keep the hash probe.  Measured against probing by hash, whole
// calls: the triangle at 10,000 organisations 868 -> 449 us (its first two count passes 305 and
// 119 -> 103 us each, where the writes now bound them), the star over a Zipf graph of 3,001 198 ->
// 168 us, a batch of 16,384 light queries at 2,000 1.73 -> 1.58 ms.
//
// The directory holds exactly the keys a probe finds: the builder walks each main bucket's chain
// as thread_probe does and stops where it stops.  A store with a chain that leaves the slot array
// or does not end, or with a key twice in one chain, gets no directory, so such stores answer as
// before.
#include <cuda_runtime.h>

#include <algorithm>

#include "wk_device.cuh"
#include "wk_dir.h"

namespace wk {
namespace {
using namespace dev;

constexpr int kLoadThreads = 256;
constexpr uint64_t kSerialList = 32;   // a longer list is checked by its whole warp

// Entry of the predicate segment table (sorted by key) with this key, or n.
__device__ __forceinline__ uint32_t pseg_find(const PredSeg* ps, uint32_t n, uint32_t key) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(&ps[mid].key) < key) lo = mid + 1; else hi = mid;
    }
    return lo < n && __ldg(&ps[lo].key) == key ? lo : n;
}

__device__ __forceinline__ void flush_range(SegScan* out, uint32_t seg, uint32_t n_pseg, uint32_t lo, uint32_t hi,
                                            uint32_t longest) {
    if (seg >= n_pseg) return;
    if (longest) atomicMax(&out[seg].longest, longest);
    if (lo > hi) return;
    atomicMin(&out[seg].vid_lo, lo);
    atomicMax(&out[seg].vid_hi, hi);
}

// One thread per slot, a warp over shares of 1,024 slots, four slots loaded before any is looked
// at.  The shares are dealt round: a segment's keys lie together, and with one contiguous share a
// warp the few warps that met the segments with lists of hundreds of entries (the members of 9,000
// departments) ran long after the others (1.78 -> 0.49 ms at 500 organisations).  Bound by the read
// of the table (16 bytes a slot, most of them empty at the default load factor) and by the short
// lists' sectors.  Lists past kChunkList entries (the type and predicate indexes: 1.5e6 entries in one list at 500 organisations) go to a
// queue as chunks that a second kernel checks with every warp; walked by the one warp that met
// them, they took 21 of the 22 ms this check cost on that store.
constexpr int kScanUnroll = 4;
__global__ void __launch_bounds__(kLoadThreads)
store_scan_kernel(const DevStore st, const PredSeg* pseg, uint32_t n_pseg, SegScan* per_seg, StoreScan* out,
                  ulonglong2* chunks, uint32_t max_chunks) {
    const uint64_t n_slots = st.n_buckets * kAssoc;
    const int lane = threadIdx.x & 31;
    const uint64_t warps = (uint64_t)gridDim.x * (kLoadThreads / 32);
    const uint64_t w = (uint64_t)blockIdx.x * (kLoadThreads / 32) + threadIdx.x / 32;
    constexpr uint64_t kStep = 32 * kScanUnroll, kShare = 8 * kStep;
    uint32_t flags = 0, seg = n_pseg, seg_key = 0xFFFFFFFFu, vlo = 0xFFFFFFFFu, vhi = 0, longest = 0;
    unsigned long long ones = 0;
    // one set of atomics a warp where its lanes met one segment or none; leaves the lanes' range empty
    auto flush = [&] {
        const unsigned any = __ballot_sync(kFull, seg < n_pseg);
        if (!any) return;
        const uint32_t seg0 = __shfl_sync(kFull, seg, __ffs(any) - 1);
        if (__all_sync(kFull, seg == seg0 || seg >= n_pseg)) {
            const uint32_t l = __reduce_min_sync(kFull, vlo), h = __reduce_max_sync(kFull, vhi);
            const uint32_t len = __reduce_max_sync(kFull, longest);
            if (lane == 0) flush_range(per_seg, seg0, n_pseg, l, h, len);
        } else {
            flush_range(per_seg, seg, n_pseg, vlo, vhi, longest);
        }
        vlo = 0xFFFFFFFFu;
        vhi = longest = 0;
        seg = n_pseg;
        seg_key = 0xFFFFFFFFu;
    };
    for (uint64_t b0 = w * kShare; b0 < n_slots; b0 += warps * kShare) {
        const uint64_t hi = min(n_slots, b0 + kShare);
        for (uint64_t b = b0; b < hi; b += kStep) {
            Slot sl[kScanUnroll];
#pragma unroll
            for (int u = 0; u < kScanUnroll; ++u) {
                const uint64_t i = b + 32 * u + lane;
                sl[u] = i < hi ? st.slots[i] : Slot{0, 0};
            }
#pragma unroll
            for (int u = 0; u < kScanUnroll; ++u) {
                const uint64_t i = b + 32 * u + lane;
                uint64_t off = 0, sz = 0;
                if (sl[u].key != 0 && (i & (kAssoc - 1)) == kAssoc - 1) {   // chain link
                    if (key_vid(sl[u].key) >= st.n_buckets) flags |= kStoreBadChain;
                } else if (sl[u].key != 0) {
                    const uint64_t v = key_vid(sl[u].key);
                    const uint32_t k = key_pid(sl[u].key) * 2 + key_dir(sl[u].key);
                    if (k != seg_key) {
                        flush_range(per_seg, seg, n_pseg, vlo, vhi, longest);
                        seg_key = k;
                        seg = pseg_find(pseg, n_pseg, k);
                        vlo = 0xFFFFFFFFu;
                        vhi = longest = 0;
                    }
                    if (v != 0) longest = max(longest, (uint32_t)ptr_size(sl[u].ptr));   // vid 0: an index list
                    if (v != 0 && v < kBlankId) {
                        vlo = min(vlo, (uint32_t)v);
                        vhi = max(vhi, (uint32_t)v);
                    }
                    off = ptr_off(sl[u].ptr);
                    sz = ptr_size(sl[u].ptr);
                    if ((sl[u].ptr >> 62) == 0 && sz == 1 && off < st.n_edges) ++ones;
                    if (ptr_is_inline(sl[u].ptr)) {
                        flags |= kStoreInlineType;
                        sz = 0;
                    } else if (off + sz > st.n_edges) {
                        flags |= kStoreBadList;
                        sz = 0;
                    } else if (sz <= kSerialList) {
                        uint32_t prev = 0;
                        const int n = (int)sz;
                        // (a one-entry list of the plain type is read when it goes into its slot)
                        for (int e0 = 0; (n > 1 || sl[u].ptr >> 62) && e0 < n; e0 += 8) {   // eight entries in flight
                            uint32_t x[8];
#pragma unroll
                            for (int j = 0; j < 8; ++j)
                                if (e0 + j < n) x[j] = __ldg(st.edges + off + e0 + j);
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                if (e0 + j >= n) continue;
                                if (e0 + j && prev >= x[j]) flags |= kStoreUnsorted;
                                if (x[j] == 0) flags |= kStoreZeroId;
                                prev = x[j];
                            }
                        }
                        sz = 0;
                    }
                }
                // the long lists of the warp's slots, one after the other, 32 entries at a time
                for (unsigned m = __ballot_sync(kFull, sz > 0); m; m &= m - 1) {
                    const int src = __ffs(m) - 1;
                    const uint64_t o = __shfl_sync(kFull, off, src), n = __shfl_sync(kFull, sz, src);
                    if (n > kChunkList) {
                        const uint32_t nc = (uint32_t)((n + kChunkList - 1) / kChunkList);
                        unsigned at = 0;
                        if (lane == 0) at = atomicAdd(&out->n_chunks, nc);
                        at = __shfl_sync(kFull, at, 0);
                        if (at + nc <= max_chunks) {   // (lists that overlap may ask for more)
                            for (uint32_t c = lane; c < nc; c += 32) {
                                // a chunk begins with the last entry of the one before it
                                const uint64_t c0 = (uint64_t)c * kChunkList - (c ? 1 : 0);
                                chunks[at + c] = make_ulonglong2(o + c0, min(n, (uint64_t)(c + 1) * kChunkList) - c0);
                            }
                            continue;
                        }
                        for (uint32_t c = lane; c < nc && at + c < max_chunks; c += 32)
                            chunks[at + c] = make_ulonglong2(0, 0);
                    }
                    bool bad = false, zero = false;
#pragma unroll 8
                    for (uint64_t e = 1 + lane; e < n; e += 32) {
                        const uint32_t x = __ldg(st.edges + o + e - 1), y = __ldg(st.edges + o + e);
                        bad |= x >= y;
                        zero |= x == 0 || y == 0;
                    }
                    if (bad) flags |= kStoreUnsorted;
                    if (zero) flags |= kStoreZeroId;
                }
            }
        }
        flush();
    }
    flags = __reduce_or_sync(kFull, flags);
    for (int o = 16; o > 0; o >>= 1) ones += __shfl_xor_sync(kFull, ones, o);
    if (lane == 0 && flags) atomicOr(&out->flags, flags);
    if (lane == 0 && ones) atomicAdd(&out->n_inline, ones);
}

// The long lists' chunks, one warp each, eight pairs in flight per lane.
__global__ void __launch_bounds__(kLoadThreads)
chunk_check_kernel(const uint32_t* edges, const ulonglong2* chunks, uint32_t max_chunks, StoreScan* out) {
    const uint32_t n = min(out->n_chunks, max_chunks);
    const int lane = threadIdx.x & 31;
    const uint32_t warps = gridDim.x * (kLoadThreads / 32);
    bool bad = false, zero = false;
    for (uint32_t i = blockIdx.x * (kLoadThreads / 32) + threadIdx.x / 32; i < n; i += warps) {
        const ulonglong2 c = chunks[i];
        const uint32_t* p = edges + c.x;
#pragma unroll 8
        for (uint64_t e = 1 + lane; e < c.y; e += 32) {
            const uint32_t x = __ldg(p + e - 1), y = __ldg(p + e);
            bad |= x >= y;
            zero |= x == 0 || y == 0;
        }
    }
    const unsigned flags = (__any_sync(kFull, bad) ? kStoreUnsorted : 0u) | (__any_sync(kFull, zero) ? kStoreZeroId : 0u);
    if (flags && lane == 0) atomicOr(&out->flags, flags);
}

// One-entry lists into their keys' own pointer words (see kInlinePtrType): for every data slot
// (slots 0-6) whose list has one entry, the original pointer word goes to the side table
// `orig` (slot index, pointer word; wk_store_export puts them back) and the slot's pointer word
// becomes the entry with the inline type.  The places in `orig` are taken a warp at a time.
__global__ void __launch_bounds__(kLoadThreads)
inline_kernel(Slot* slots, uint64_t n_slots, const uint32_t* edges, uint64_t n_edges, StoreScan* out,
              uint64_t* orig) {
    const int lane = threadIdx.x & 31;
    bool zero = false;
    const uint64_t stride = (uint64_t)gridDim.x * kLoadThreads * kScanUnroll;
    for (uint64_t b = ((uint64_t)blockIdx.x * kLoadThreads + (threadIdx.x & ~31)) * kScanUnroll; b < n_slots;
         b += stride) {
        Slot sl[kScanUnroll];
        bool one[kScanUnroll];
        unsigned m[kScanUnroll];
        uint32_t total = 0;
#pragma unroll
        for (int u = 0; u < kScanUnroll; ++u) {
            const uint64_t i = b + 32 * u + lane;
            sl[u] = i < n_slots ? slots[i] : Slot{0, 0};
        }
#pragma unroll
        for (int u = 0; u < kScanUnroll; ++u) {
            const uint64_t i = b + 32 * u + lane;
            one[u] = (i & (kAssoc - 1)) != kAssoc - 1 && sl[u].key != 0 && (sl[u].ptr >> 62) == 0 &&
                     ptr_size(sl[u].ptr) == 1 && ptr_off(sl[u].ptr) < n_edges;
            m[u] = __ballot_sync(kFull, one[u]);
            total += __popc(m[u]);
        }
        if (!total) continue;
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(&out->n_inline, (unsigned long long)total);
        at = __shfl_sync(kFull, at, 0);
#pragma unroll
        for (int u = 0; u < kScanUnroll; ++u) {
            if (one[u]) {
                const uint64_t i = b + 32 * u + lane;
                const uint64_t k = at + __popc(m[u] & ((1u << lane) - 1));
                *reinterpret_cast<ulonglong2*>(orig + 2 * k) = make_ulonglong2(i, sl[u].ptr);
                const uint32_t entry = __ldg(edges + ptr_off(sl[u].ptr));
                zero |= entry == 0;
                slots[i].ptr = make_inline_ptr(entry);
            }
            at += __popc(m[u]);
        }
    }
    if (zero) atomicOr(&out->flags, (unsigned)kStoreZeroId);
}

// Every key a probe of its segment finds, from the segment's main buckets: f(vid, pointer word).
// One thread per main bucket, walking it and its chain in the probe's order up to the first empty
// slot; a key is reported by its home bucket only.
template <class F>
__device__ __forceinline__ void dir_walk(const DevStore& st, const DirSeg* segs, uint32_t n_segs, uint64_t n_buckets,
                                         unsigned* flags, F f) {
    for (uint64_t t = (uint64_t)blockIdx.x * kLoadThreads + threadIdx.x; t < n_buckets;
         t += (uint64_t)gridDim.x * kLoadThreads) {
        uint32_t lo = 0, hi = n_segs - 1;   // the last segment whose first bucket is <= t
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1) >> 1;
            if (__ldg(&segs[mid].first) <= t) lo = mid; else hi = mid - 1;
        }
        const DirSeg& d = segs[lo];
        const uint64_t home = d.seg.bucket_start + (t - d.first);
        uint64_t bucket = home;
        int hop = 0;
        for (; hop < kMaxProbeIters; ++hop) {
            // (a chain this long may be one that does not end; where one has been found there is no
            // directory, so the walks of a store full of them are cut short)
            if (hop >= 64 && *(volatile unsigned*)flags & kStoreBadChain) return;
            if (bucket >= st.n_buckets) {
                atomicOr(flags, kStoreBadChain);
                break;
            }
            const Slot* b = st.slots + bucket * kAssoc;
            bool end = true;
            for (int s = 0; s < kAssoc; s += 2) {
                const ulonglong2* q = reinterpret_cast<const ulonglong2*>(b + s);
                const ulonglong2 s0 = q[0], s1 = q[1];
                bool stop = false;
                for (int j = 0; j < 2 && !stop; ++j) {
                    const uint64_t key = j ? s1.x : s0.x, ptr = j ? s1.y : s0.y;
                    if (key == 0) {
                        stop = true;
                    } else if (s + j == kAssoc - 1) {   // the chain link
                        bucket = key_vid(key);
                        end = false;
                    } else {
                        const uint64_t v = key_vid(key);
                        if (v != 0 && v < kBlankId && key_pid(key) * 2 + key_dir(key) == d.key &&
                            bucket_of(key, d.seg) == home)
                            f(d, (uint32_t)v, ptr);
                    }
                }
                if (stop) break;
            }
            if (end) break;
        }
        if (hop == kMaxProbeIters) atomicOr(flags, kStoreBadChain);
    }
}

__global__ void __launch_bounds__(kLoadThreads)
dir_bits_kernel(const DevStore st, const DirSeg* segs, uint32_t n_segs, uint64_t n_buckets, DirBlock* blocks,
                unsigned* flags) {
    dir_walk(st, segs, n_segs, n_buckets, flags, [&](const DirSeg& d, uint32_t vid, uint64_t ptr) {
        if (ptr_size(ptr) == 0) return;   // an empty list is no key to any step
        const uint32_t i = vid - d.seg.vid_lo;
        if (i >= d.seg.vid_span) return;   // the scan saw every key, so none is outside
        const unsigned bit = 1u << (i & 31);
        if (atomicOr(&blocks[d.block0 + (i >> 5)].bits, bit) & bit) atomicOr(flags, (unsigned)kStoreDupKey);
    });
}

__global__ void __launch_bounds__(kLoadThreads)
dir_fill_kernel(const DevStore st, const DirSeg* segs, uint32_t n_segs, uint64_t n_buckets, unsigned* flags) {
    dir_walk(st, segs, n_segs, n_buckets, flags, [&](const DirSeg& d, uint32_t vid, uint64_t ptr) {
        const uint32_t i = vid - d.seg.vid_lo;
        if (i >= d.seg.vid_span || ptr_size(ptr) == 0) return;
        const uint32_t at = dir_place(dir_block(d.seg, i), i);
        if (d.seg.dir_values)
            static_cast<uint32_t*>(const_cast<void*>(d.seg.dir_words))[at] =
                ptr_is_inline(ptr) ? (uint32_t)(ptr >> kNbitsSize) : __ldg(st.edges + ptr_off(ptr));
        else
            static_cast<uint64_t*>(const_cast<void*>(d.seg.dir_words))[at] = ptr;
    });
}

// Each block's base: the keys of its segment's blocks before it.  kDirScanBlocks blocks per CTA
// (segments start at multiples of that many blocks); the CTAs' sums are scanned by one CTA in
// between.
__global__ void __launch_bounds__(kLoadThreads) dir_sum_kernel(const DirBlock* blocks, uint64_t* sums) {
    __shared__ uint64_t s_warp[kLoadThreads / 32];
    const uint64_t b0 = (uint64_t)blockIdx.x * kDirScanBlocks;
    uint64_t c = 0;
    for (uint32_t i = threadIdx.x; i < kDirScanBlocks; i += kLoadThreads) c += __popc(blocks[b0 + i].bits);
    const uint64_t ex = block_exclusive_sum<kLoadThreads>(c, s_warp);
    if (threadIdx.x == kLoadThreads - 1) sums[blockIdx.x] = ex + c;
}

__global__ void __launch_bounds__(kLoadThreads) dir_scan_kernel(uint64_t* sums, uint32_t n) {
    __shared__ uint64_t s_warp[kLoadThreads / 32];
    __shared__ uint64_t s_carry;
    if (threadIdx.x == 0) s_carry = 0;
    __syncthreads();
    for (uint32_t r0 = 0; r0 < n; r0 += kLoadThreads) {
        const uint32_t i = r0 + threadIdx.x;
        const uint64_t x = i < n ? sums[i] : 0;
        const uint64_t ex = block_exclusive_sum<kLoadThreads>(x, s_warp);
        const uint64_t carry = s_carry;
        if (i < n) sums[i] = carry + ex;
        __syncthreads();
        if (threadIdx.x == kLoadThreads - 1) s_carry = carry + ex + x;
        __syncthreads();
    }
    if (threadIdx.x == 0) sums[n] = s_carry;
}

__global__ void __launch_bounds__(kLoadThreads)
dir_base_kernel(DirBlock* blocks, const uint64_t* sums, const DirSeg* segs, uint32_t n_segs) {
    __shared__ uint64_t s_warp[kLoadThreads / 32];
    constexpr int kPer = kDirScanBlocks / kLoadThreads;   // consecutive blocks per thread
    const uint64_t b0 = (uint64_t)blockIdx.x * kDirScanBlocks + threadIdx.x * kPer;
    uint32_t lo = 0, hi = n_segs - 1;   // the segment these blocks belong to
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (__ldg(&segs[mid].block0) <= b0) lo = mid; else hi = mid - 1;
    }
    const uint64_t first = sums[segs[lo].block0 / kDirScanBlocks];
    uint32_t c[kPer], sum = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        c[k] = __popc(blocks[b0 + k].bits);
        sum += c[k];
    }
    uint32_t at = (uint32_t)(sums[blockIdx.x] - first + block_exclusive_sum<kLoadThreads>(sum, s_warp));
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        blocks[b0 + k].base = at;
        at += c[k];
    }
}

int load_grid(int sm_count) { return sm_count * (2048 / kLoadThreads); }

}  // namespace

cudaError_t launch_store_scan(const DevStore& st, const PredSeg* pseg, uint32_t n_pseg, SegScan* per_seg,
                              StoreScan* out, ulonglong2* chunks, uint32_t max_chunks, int sm_count, cudaStream_t s) {
    store_scan_kernel<<<load_grid(sm_count), kLoadThreads, 0, s>>>(st, pseg, n_pseg, per_seg, out, chunks, max_chunks);
    chunk_check_kernel<<<load_grid(sm_count), kLoadThreads, 0, s>>>(st.edges, chunks, max_chunks, out);
    return cudaGetLastError();
}

cudaError_t launch_inline(const DevStore& st, StoreScan* out, uint64_t* orig, int sm_count, cudaStream_t s) {
    inline_kernel<<<load_grid(sm_count), kLoadThreads, 0, s>>>(const_cast<Slot*>(st.slots), st.n_buckets * kAssoc,
                                                               st.edges, st.n_edges, out, orig);
    return cudaGetLastError();
}

cudaError_t launch_dir_bits(const DevStore& st, const DirSeg* segs, uint32_t n_segs, uint64_t n_buckets,
                            DirBlock* blocks, uint64_t n_blocks, uint64_t* sums, StoreScan* out, int sm_count,
                            cudaStream_t s) {
    const uint32_t n_sums = (uint32_t)(n_blocks / kDirScanBlocks);
    dir_bits_kernel<<<load_grid(sm_count), kLoadThreads, 0, s>>>(st, segs, n_segs, n_buckets, blocks, &out->flags);
    dir_sum_kernel<<<n_sums, kLoadThreads, 0, s>>>(blocks, sums);
    dir_scan_kernel<<<1, kLoadThreads, 0, s>>>(sums, n_sums);
    dir_base_kernel<<<n_sums, kLoadThreads, 0, s>>>(blocks, sums, segs, n_segs);
    return cudaGetLastError();
}

cudaError_t launch_dir_fill(const DevStore& st, const DirSeg* segs, uint32_t n_segs, uint64_t n_buckets,
                            StoreScan* out, int sm_count, cudaStream_t s) {
    dir_fill_kernel<<<load_grid(sm_count), kLoadThreads, 0, s>>>(st, segs, n_segs, n_buckets, &out->flags);
    return cudaGetLastError();
}

}  // namespace wk
