// Decode attention over long contexts and for several rows: the keys stream once for all query rows of a kv head.
//
// A ring of K/V tiles (16 keys: 8 KB of K, 8 KB of V) in shared memory is filled by cp.async one tile ahead of the warps that
// read it, so the loads of the next tile are in flight while a tile is multiplied; with tiles read straight into registers
// a warp waited for one DRAM round trip per tile (3.4 TB/s at 200K keys).  A warp holds 8 or 16 query rows (NTR = 1, 2) in
// the mma fragments of attn_mma.cuh (same arithmetic: Q and P as bf16 hi + lo); WR warps share a ring, so up to 32 rows - an
// eight-row step over the four heads of a rank - read K and V from memory once instead of in four passes.  No ring waits
// for another; their partials and those of the CTAs are merged by attn_merge_kernel.
#pragma once

#include "attn_mma.cuh"

namespace nexrt {

constexpr int kStreamHd = 256;
constexpr int kTileKeys = 16;
constexpr int kTileRow = kStreamHd * 2 + 16;                    // bytes between two rows of a tile: fragment reads do not conflict
constexpr int kTileHalf = kTileKeys * kTileRow;                 // K or V of one tile
constexpr int kTileStage = 2 * kTileHalf;
constexpr int kTileDepth = 2;                                   // stages of a ring
template <int WR> constexpr int stream_rings() { return WR == 1 ? 6 : 4; }

// Shared memory: the rings, the query fragments of the WR row groups, the new K rows, a scratch row per warp, the rotations.
template <int NTR, int WR> constexpr size_t attn_stream_smem(int M, int rotary) {
    return static_cast<size_t>(stream_rings<WR>()) * kTileDepth * kTileStage + static_cast<size_t>(WR) * 16 * 32 * 16 * NTR +
           static_cast<size_t>(M) * kStreamHd * 2 + sizeof(float) * (static_cast<size_t>(kStreamHd) * stream_rings<WR>() * WR + static_cast<size_t>(M) * rotary);
}

__device__ __forceinline__ void cp_async16_zfill(void* dst, const void* src, bool valid) {
    const unsigned int d = static_cast<unsigned int>(__cvta_generic_to_shared(dst));
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

}  // namespace nexrt
