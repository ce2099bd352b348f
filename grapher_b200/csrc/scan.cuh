// scan.cuh -- single-pass scans over tiles of GVIZ_SCAN_TILE entries: a tile
// takes its index from a ticket counter, so every lower tile has started
// before it, publishes its count, adds those of the tiles before it by
// decoupled look-back and publishes its prefix. state: [0] ticket, [1 + t]
// status word of tile t (flag in the high half, count in the low half), zero
// at the start. Shared by sort.cu and tree.cu.
#pragma once
#include "internal.cuh"

namespace {

constexpr uint64_t kFlagAggregate = 1ull << 32;
constexpr uint64_t kFlagPrefix = 2ull << 32;
constexpr uint32_t kLookbackSpin = 1u << 22;  // reads of a status word before giving up

__device__ __forceinline__ uint64_t ld_status(const uint64_t *p) {
  uint64_t v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_status(uint64_t *p, uint64_t v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// The scan's look-back by one warp: lane l reads the word of the l-th tile
// before, so a step covers 32 tiles; the result is in every lane.
__device__ __forceinline__ uint32_t lookback_warp(const uint64_t *st, uint32_t tile,
                                                  uint32_t *status) {
  const uint32_t lane = lane_id();
  uint32_t excl = 0;
  uint32_t spins = 0;
  for (int64_t p = (int64_t)tile - 1; p >= 0; p -= 32) {
    uint64_t w = p - lane >= 0 ? ld_status(st + (size_t)(p - lane)) : kFlagPrefix;
    uint32_t have;
    for (;;) {
      // enough once every word up to the nearest prefix is published
      have = __ballot_sync(0xffffffffu, (w >> 32) != 0);
      const uint32_t pre = __ballot_sync(0xffffffffu, (w & ~0xffffffffull) == kFlagPrefix);
      const uint32_t need = pre ? (pre ^ (pre - 1u)) : 0xffffffffu;
      if ((have & need) == need) {
        uint32_t c = (need >> lane) & 1u ? (uint32_t)w : 0u;
        excl += __reduce_add_sync(0xffffffffu, c);
        if (pre) return excl;
        break;
      }
      if (++spins > kLookbackSpin) {
        if (lane == 0) atomicOr(status, GVIZ_ST_TREE);
        return excl;
      }
      if ((w >> 32) == 0) w = ld_status(st + (size_t)(p - lane));
    }
  }
  return excl;
}

// Block-wide exclusive scan of one value per thread; returns the block total.
template <int THREADS>
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v,
                                                         uint32_t &excl) {
  __shared__ uint32_t warpTot[THREADS / 32];
  const unsigned lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= (unsigned)o) inc += t;
  }
  if (lane == 31) warpTot[w] = inc;
  __syncthreads();
  if (w == 0) {
    uint32_t t = lane < THREADS / 32 ? warpTot[lane] : 0;
    uint32_t ti = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t u = __shfl_up_sync(0xffffffffu, ti, o);
      if (lane >= (unsigned)o) ti += u;
    }
    if (lane < THREADS / 32) warpTot[lane] = ti - t;  // exclusive warp offsets
  }
  __syncthreads();
  excl = warpTot[w] + inc - v;
  __shared__ uint32_t blockTot;
  if (threadIdx.x == THREADS - 1) blockTot = excl + v;
  __syncthreads();
  uint32_t bt = blockTot;
  __syncthreads();
  return bt;
}

__device__ __forceinline__ uint32_t scan_ticket(uint64_t *state) {
  return (uint32_t)atomicAdd(reinterpret_cast<unsigned long long *>(state), 1ull);
}

// The sum of the tiles before `tile`, whose own count is `tot` (the same in
// every thread); the last tile writes the whole sum to *total (may be null).
// For the whole block.
__device__ __forceinline__ uint32_t scan_publish(uint64_t *state, uint32_t tile, uint32_t tot,
                                                 uint32_t nTiles, uint32_t *total,
                                                 uint32_t *status) {
  __shared__ uint32_t sExcl;
  uint64_t *st = state + 1;
  if (threadIdx.x < 32) {
    if (tile != 0 && threadIdx.x == 0) st_status(st + tile, kFlagAggregate | tot);
    const uint32_t before = lookback_warp(st, tile, status);
    if (threadIdx.x == 0) {
      st_status(st + tile, kFlagPrefix | (before + tot));
      sExcl = before;
      if (total && tile == nTiles - 1) *total = before + tot;
    }
  }
  __syncthreads();
  return sExcl;
}

// The same for a count per warp (the same in every lane of it): the sum of
// the tiles and of this tile's warps before the caller's.
template <int THREADS>
__device__ __forceinline__ uint32_t scan_tile_prefix(uint64_t *state, uint32_t tile,
                                                     uint32_t warpCount, uint32_t nTiles,
                                                     uint32_t *total, uint32_t *status) {
  __shared__ uint32_t warpTot[THREADS / 32];
  const uint32_t w = threadIdx.x >> 5;
  if ((threadIdx.x & 31u) == 0u) warpTot[w] = warpCount;
  __syncthreads();
  uint32_t before = 0, tot = 0;
#pragma unroll
  for (uint32_t k = 0; k < THREADS / 32; k++) {
    before += k < w ? warpTot[k] : 0u;
    tot += warpTot[k];
  }
  return before + scan_publish(state, tile, tot, nTiles, total, status);
}

}  // namespace
