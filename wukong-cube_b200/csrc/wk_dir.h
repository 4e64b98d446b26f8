// Load-time passes over a store on the device (wk_dir.cu): the checks of its lists, the
// one-entry lists moved into their keys' slots, and the vertex directories.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "wk_kernels.h"
#include "wk_versatile.h"

namespace wk {

// What the first pass finds.
enum : uint32_t {
    kStoreUnsorted = 1u,   // a list is not strictly ascending
    kStoreBadList = 2u,    // a list lies outside the edge array
    kStoreInlineType = 4u, // a pointer word already carries the inline type
    kStoreBadChain = 8u,   // a chain link past the slot array, or a chain that does not end
    kStoreDupKey = 16u,    // a key twice in one chain
    kStoreZeroId = 32u,    // a list holds id 0, which as a row's vertex names an index list
};
struct StoreScan {
    unsigned long long n_inline;   // keys whose list has one entry
    unsigned int flags;
    unsigned int n_chunks;         // chunks of long lists
};
constexpr uint64_t kChunkList = 8192;   // entries of a long list checked by one warp
inline uint32_t store_scan_chunks(uint64_t n_edges) {   // room for every chunk of disjoint lists
    return (uint32_t)(2 * n_edges / kChunkList) + 1;
}

// What it finds of each predicate segment.
struct SegScan {
    uint32_t vid_lo, vid_hi;   // lowest and highest vertex id of its keys (the blank id and
                               // above left out); 0xFFFFFFFF and 0 when there is none
    uint32_t longest;          // entries of its longest list
    uint32_t pad;
};

// Pass over every slot: the checks, the one-entry lists counted, and per_seg[i] for pseg[i] (set
// by the caller to no key, 0).  `chunks`: store_scan_chunks(n_edges) entries of scratch.
cudaError_t launch_store_scan(const DevStore& st, const PredSeg* pseg, uint32_t n_pseg, SegScan* per_seg,
                              StoreScan* out, ulonglong2* chunks, uint32_t max_chunks, int sm_count, cudaStream_t s);
// One-entry lists into their keys' pointer words; the original words (slot index, word) go to
// orig, counted in out->n_inline (0 on entry).  (Their entries are looked at here, all others by the scan.)
cudaError_t launch_inline(const DevStore& st, StoreScan* out, uint64_t* orig, int sm_count, cudaStream_t s);

// A segment whose directory is built: its main buckets (disjoint from every other's), the keys'
// predicate and direction, and where its blocks start among all blocks.
struct DirSeg {
    uint64_t first;          // main buckets of the segments before it in the table
    uint64_t block0;
    SegDesc seg;             // vid_lo, vid_span, dir, dir_values and (for the fill) dir_words set
    uint32_t key;            // pid * 2 + dir
    uint32_t pad;
};
// Set the presence bits of every key a probe of its segment finds (flags: kStoreBadChain,
// kStoreDupKey), then each block's base.  block0 and n_blocks are multiples of kDirScanBlocks;
// sums[k] becomes the keys of the blocks before k * kDirScanBlocks (n_blocks / kDirScanBlocks + 1
// entries).
constexpr uint32_t kDirScanBlocks = 512;
cudaError_t launch_dir_bits(const DevStore& st, const DirSeg* segs, uint32_t n_segs, uint64_t n_buckets,
                            DirBlock* blocks, uint64_t n_blocks, uint64_t* sums, StoreScan* out, int sm_count,
                            cudaStream_t s);
// Put every key's word in its place (seg.dir_words).
cudaError_t launch_dir_fill(const DevStore& st, const DirSeg* segs, uint32_t n_segs, uint64_t n_buckets,
                            StoreScan* out, int sm_count, cudaStream_t s);

}  // namespace wk
