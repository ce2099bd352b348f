// sort.cu -- hand-written device primitives: exclusive scan and a stable
// LSD radix sort of (uint64 key, uint32 value) pairs.
//
// The quadtree build sorts vertices by their quadrant path; stability keeps
// equal paths in vertex-index order, which is the arrival order of points in
// a reference leaf (src/ds/gvizQuadtree.c:129-131).
//
// Both are single-pass over their input per digit (per scan): a tile takes
// its index from a ticket counter, so every lower tile has started before
// it; it publishes its count (flag AGGREGATE), then adds the counts of the
// tiles before it, walking back until one has published its inclusive
// prefix (flag PREFIX), and publishes its own prefix (decoupled look-back).
// The first pass's digit counts come from the kernel that makes the keys; each
// pass counts the next pass's digits of the keys it holds.
// Status words are 64 bits in the scan (flag in the high half, count in the
// low half) and 32 bits in the sort, written and read with single relaxed
// accesses; a wait that outlasts its iteration limit sets GVIZ_ST_TREE and
// ends.
#include <algorithm>

#include "internal.cuh"
#include "scan.cuh"

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
static_assert(kScanThreads * kScanItems == GVIZ_SCAN_TILE, "the scan state is sized by it");
constexpr int kScanTile = GVIZ_SCAN_TILE;
constexpr int kTopThreads = 1024;

constexpr int kLookbackWidth = 8;
constexpr int kSortThreads = 512;
constexpr int kSortPasses = (64 - GVIZ_SORT_SKIP_BITS) / 8;
static_assert(kSortPasses % 2 == 0, "the sorted pairs must end in the input buffers");

// the sort's status words: flag in the top two bits, count below (n < 2^30)
constexpr uint32_t kAggregate32 = 1u << 30;
constexpr uint32_t kPrefix32 = 1u << 31;
constexpr uint32_t kCount32 = kAggregate32 - 1u;

__device__ __forceinline__ uint32_t ld_status32(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_status32(uint32_t *p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// The sort's look-back, one thread per digit: the sum of the counts of tiles
// [0, tile) in the status column `st` of stride 256 (tile t's word is
// st[256 t]), WIDTH tiles per step (independent loads). The tiles of a pass
// run side by side and publish their counts at about the same time, so the
// walk is a chain of L2 round trips; its length, not its traffic, sets the
// pass's time, hence the wide step. Tile 0 publishes its prefix without
// waiting, so the walk always ends.
template <int WIDTH>
__device__ __forceinline__ uint32_t lookback_digit(const uint32_t *st, uint32_t tile,
                                                   uint32_t *status) {
  uint32_t excl = 0;
  uint32_t spins = 0;
  for (int64_t p = (int64_t)tile - 1; p >= 0; p -= WIDTH) {
    uint32_t w[WIDTH];
#pragma unroll
    for (int i = 0; i < WIDTH; i++)
      w[i] = p - i >= 0 ? ld_status32(st + (size_t)(p - i) * 256) : kPrefix32;
#pragma unroll
    for (int i = 0; i < WIDTH; i++) {
      while ((w[i] & ~kCount32) == 0) {  // not published yet
        if (++spins > kLookbackSpin) {
          atomicOr(status, GVIZ_ST_TREE);
          return excl;
        }
        w[i] = ld_status32(st + (size_t)(p - i) * 256);
      }
      excl += w[i] & kCount32;
      if (w[i] & kPrefix32) return excl;
    }
  }
  return excl;
}

// Single-pass exclusive scan: tile = ticket, 2048 entries per tile.
// state: [0] ticket, [1 + t] status of tile t.
__global__ __launch_bounds__(kScanThreads) void k_scan_onepass(
    const uint32_t *in, uint32_t *out, uint32_t n, uint64_t *state, uint32_t *total,
    uint32_t *status) {
  step_order();
  __shared__ uint32_t sTile;
  if (threadIdx.x == 0) sTile = scan_ticket(state);
  __syncthreads();
  const uint32_t tile = sTile;
  const uint32_t base = tile * kScanTile + threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  uint32_t s = 0;
#pragma unroll
  for (int j = 0; j < kScanItems; j++) {
    const uint32_t i = base + j;
    v[j] = i < n ? in[i] : 0u;
    s += v[j];
  }
  uint32_t excl;
  const uint32_t tot = block_exclusive_scan<kScanThreads>(s, excl);
  excl += scan_publish(state, tile, tot, (n + kScanTile - 1) / kScanTile, total, status);
#pragma unroll
  for (int j = 0; j < kScanItems; j++) {
    const uint32_t i = base + j;
    if (i < n) out[i] = excl;
    excl += v[j];
  }
}

// Whole scan in one block: each thread owns a contiguous run of ceil(n/1024)
// entries (n <= kSingleMax), one launch instead of three.
constexpr uint32_t kSingleMax = 1u << 13;  // one SM: only for small arrays

__global__ __launch_bounds__(kTopThreads) void k_scan_single(
    const uint32_t *in, uint32_t *out, uint32_t n, uint32_t *total) {
  step_order();
  const uint32_t per = (n + kTopThreads - 1) / kTopThreads;
  const uint32_t b = threadIdx.x * per;
  uint32_t s = 0;
  for (uint32_t j = 0; j < per; j++) {
    const uint32_t i = b + j;
    if (i < n) s += in[i];
  }
  uint32_t excl;
  const uint32_t tot = block_exclusive_scan<kTopThreads>(s, excl);
  for (uint32_t j = 0; j < per; j++) {
    const uint32_t i = b + j;
    if (i < n) {
      const uint32_t t = in[i];
      out[i] = excl;
      excl += t;
    }
  }
  if (threadIdx.x == 0 && total) *total = tot;
}

// The lanes holding valid keys of the same 8-bit digit d: eight ballots, one
// per bit, which do not depend on each other.
__device__ __forceinline__ uint32_t digit_peers(uint32_t d, bool valid) {
  uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
  for (int b = 0; b < 8; b++) {
    const uint32_t set = __ballot_sync(0xffffffffu, (d >> b) & 1u);
    peers &= ((d >> b) & 1u) ? set : ~set;
  }
  return peers;
}

// Stable scatter: warp w of a tile owns 32 * ROUNDS consecutive keys, taken
// in rounds of 32; ballots rank equal digits inside a round. A pass moves
// 24 B per key but is bound by latency: the ticket, the ranking rounds (each
// reads and writes its warp's counters) and the look-back. __match_any_sync
// in place of the ballots and 16 rounds of 256 threads took 23.5 us per pass
// at 1,048,576 keys and 14.5 us at 1,024 (one tile); this takes 17 and 5.5.
// Shared memory of the scatter beyond its static arrays: the tile's keys
// and values reordered by digit.
constexpr size_t scatter_dyn(size_t tile) { return tile * (sizeof(uint64_t) + sizeof(uint32_t)); }

// One pass over digit `pass`: tile = ticket; each digit's start in the
// output is its global start (a scan of ghist) plus its count in the tiles
// before (look-back over the status words state[tile * 256 + digit]).
template <int THREADS, int ROUNDS>
__global__ __launch_bounds__(THREADS) void k_radix_onesweep(
    const uint64_t *__restrict__ kin, const uint32_t *__restrict__ vin,
    uint64_t *__restrict__ kout, uint32_t *__restrict__ vout, uint32_t n,
    int pass, uint32_t *ghist, uint32_t *state, uint32_t *ticket,
    uint32_t *status) {
  step_order();
  constexpr int kWarps = THREADS / 32;
  constexpr uint32_t kTile = THREADS * ROUNDS;
  extern __shared__ __align__(16) unsigned char dyn[];
  uint64_t *sk = reinterpret_cast<uint64_t *>(dyn);
  uint32_t *sv = reinterpret_cast<uint32_t *>(sk + kTile);
  __shared__ uint32_t wcnt[kWarps][256];
  __shared__ uint32_t base[256];
  __shared__ uint32_t start[256];  // first in-tile position of each digit
  __shared__ uint32_t sTile;
  __shared__ uint32_t nextCnt[256];  // the next pass's digit counts of this tile
  const unsigned tid = threadIdx.x, w = tid >> 5, lane = tid & 31u;
  const int shift = GVIZ_SORT_SKIP_BITS + 8 * pass;
  const bool countNext = pass + 1 < kSortPasses;
  const bool digitThread = tid < 256;  // thread d looks after digit d
  if (tid == 0) sTile = atomicAdd(ticket, 1u);
  for (unsigned d = tid; d < kWarps * 256; d += THREADS) (&wcnt[0][0])[d] = 0;
  if (digitThread) nextCnt[tid] = 0u;
  // the digit's first output position: exclusive scan of the global counts
  uint32_t gstart;
  block_exclusive_scan<THREADS>(digitThread ? ghist[pass * 256 + tid] : 0u, gstart);
  const uint32_t tile = sTile;
  const uint32_t tileBase = tile * kTile + w * (ROUNDS * 32);
  uint64_t k[ROUNDS];
  uint32_t v[ROUNDS];
  uint32_t rank[ROUNDS];
  // all of the tile's loads are in flight before the first is ranked: the
  // ranking rounds below are ordered by warp barriers, which no load crosses
#pragma unroll
  for (int r = 0; r < ROUNDS; r++) {
    const uint32_t i = tileBase + r * 32 + lane;
    k[r] = i < n ? kin[i] : 0ull;
    v[r] = i < n ? vin[i] : 0u;
  }
#pragma unroll
  for (int r = 0; r < ROUNDS; r++) {
    const bool valid = tileBase + r * 32 + lane < n;
    const uint32_t d = (uint32_t)(k[r] >> shift) & 255u;
    if (countNext && valid) atomicAdd(&nextCnt[(uint32_t)(k[r] >> (shift + 8)) & 255u], 1u);
    const uint32_t peers = digit_peers(d, valid);
    const uint32_t lt = peers & ((1u << lane) - 1u);
    const uint32_t before = valid ? wcnt[w][d] : 0u;
    rank[r] = before + __popc(lt);
    __syncwarp();
    if (valid && lt == 0) wcnt[w][d] = before + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // per digit: warps' offsets, then this tile's count of the digit and the
  // counts of the tiles before; the tile's digit starts by a block-wide
  // exclusive scan of the digit totals
  uint32_t run = 0;
  if (digitThread) {
#pragma unroll
    for (int ww = 0; ww < kWarps; ww++) {
      const uint32_t t = wcnt[ww][tid];
      wcnt[ww][tid] = run;
      run += t;
    }
    st_status32(state + tid + (size_t)tile * 256, (tile == 0 ? kPrefix32 : kAggregate32) | run);
    if (countNext && nextCnt[tid]) atomicAdd(ghist + (pass + 1) * 256 + tid, nextCnt[tid]);
  }
  uint32_t first;
  block_exclusive_scan<THREADS>(run, first);
  if (digitThread) start[tid] = first;
  __syncthreads();
  // the tile reordered by digit in shared memory (stable: warp, round, lane
  // is input order) ...
#pragma unroll
  for (int r = 0; r < ROUNDS; r++) {
    if (tileBase + r * 32 + lane >= n) continue;
    const uint32_t d = (uint32_t)(k[r] >> shift) & 255u;
    const uint32_t pos = start[d] + wcnt[w][d] + rank[r];
    sk[pos] = k[r];
    sv[pos] = v[r];
  }
  if (digitThread) {
    uint32_t *col = state + tid;
    const uint32_t before = tile ? lookback_digit<kLookbackWidth>(col, tile, status) : 0u;
    if (tile) st_status32(col + (size_t)tile * 256, kPrefix32 | (before + run));
    base[tid] = gstart + before;
  }
  __syncthreads();
  // ... then written out in order: each digit's run lands contiguously
  const uint32_t t0 = tile * kTile;
  const uint32_t cnt = n - t0 < kTile ? n - t0 : kTile;
#pragma unroll
  for (int r = 0; r < ROUNDS; r++) {
    const uint32_t j = r * THREADS + tid;
    if (j >= cnt) break;
    const uint64_t kk = sk[j];
    const uint32_t d = (uint32_t)(kk >> shift) & 255u;
    const uint32_t dst = base[d] + (j - start[d]);
    kout[dst] = kk;
    vout[dst] = sv[j];
  }
}

// The whole sort of n <= THREADS * ROUNDS keys by one block: the pairs stay in
// shared memory through all passes, so there are no launches, counts or
// look-backs between them.
template <int THREADS, int ROUNDS>
struct SmallSortSmem {
  uint64_t k[THREADS * ROUNDS];
  uint32_t v[THREADS * ROUNDS];
  uint32_t wcnt[THREADS / 32][256];
  uint32_t start[256];
};

template <int THREADS, int ROUNDS>
__global__ __launch_bounds__(THREADS) void k_radix_small(uint64_t *keys, uint32_t *vals,
                                                         uint32_t n) {
  step_order();
  constexpr int kWarps = THREADS / 32;
  extern __shared__ __align__(16) unsigned char dyn[];
  SmallSortSmem<THREADS, ROUNDS> &s = *reinterpret_cast<SmallSortSmem<THREADS, ROUNDS> *>(dyn);
  const unsigned tid = threadIdx.x, w = tid >> 5, lane = tid & 31u;
  const uint32_t at = w * (ROUNDS * 32) + lane;
  uint64_t k[ROUNDS];
  uint32_t v[ROUNDS], rank[ROUNDS];
#pragma unroll
  for (int r = 0; r < ROUNDS; r++) {
    const uint32_t i = at + r * 32;
    k[r] = i < n ? keys[i] : 0ull;
    v[r] = i < n ? vals[i] : 0u;
  }
  for (int pass = 0; pass < kSortPasses; pass++) {
    const int shift = GVIZ_SORT_SKIP_BITS + 8 * pass;
    for (unsigned d = tid; d < kWarps * 256; d += THREADS) (&s.wcnt[0][0])[d] = 0;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
      const bool valid = at + r * 32 < n;
      const uint32_t d = (uint32_t)(k[r] >> shift) & 255u;
      const uint32_t peers = digit_peers(d, valid);
      const uint32_t lt = peers & ((1u << lane) - 1u);
      const uint32_t before = valid ? s.wcnt[w][d] : 0u;
      rank[r] = before + __popc(lt);
      __syncwarp();
      if (valid && lt == 0) s.wcnt[w][d] = before + __popc(peers);
      __syncwarp();
    }
    __syncthreads();
    uint32_t run = 0;
    if (tid < 256) {
#pragma unroll
      for (int ww = 0; ww < kWarps; ww++) {
        const uint32_t t = s.wcnt[ww][tid];
        s.wcnt[ww][tid] = run;
        run += t;
      }
    }
    uint32_t first;
    block_exclusive_scan<THREADS>(run, first);
    if (tid < 256) s.start[tid] = first;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
      if (at + r * 32 >= n) continue;
      const uint32_t d = (uint32_t)(k[r] >> shift) & 255u;
      const uint32_t to = s.start[d] + s.wcnt[w][d] + rank[r];
      s.k[to] = k[r];
      s.v[to] = v[r];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
      const uint32_t i = at + r * 32;
      k[r] = i < n ? s.k[i] : 0ull;
      v[r] = i < n ? s.v[i] : 0u;
    }
  }
#pragma unroll
  for (int r = 0; r < ROUNDS; r++) {
    const uint32_t i = at + r * 32;
    if (i < n) {
      keys[i] = k[r];
      vals[i] = v[r];
    }
  }
}

template <int THREADS, int ROUNDS>
void small_sort_limit() {
  cudaFuncSetAttribute(k_radix_small<THREADS, ROUNDS>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)sizeof(SmallSortSmem<THREADS, ROUNDS>));
}

template <int THREADS, int ROUNDS>
void small_sort(gvizCudaForce *h, uint64_t *keys, uint32_t *vals, size_t n) {
  launch_after(h->stream, k_radix_small<THREADS, ROUNDS>, 1, THREADS,
               sizeof(SmallSortSmem<THREADS, ROUNDS>), keys, vals, (uint32_t)n);
}

}  // namespace

size_t scan_state_entries(size_t n) {
  return (n + kScanTile - 1) / kScanTile + 1;
}

struct SortShape {
  int threads, rounds;
  size_t tile() const { return (size_t)threads * rounds; }
};

// Tile of a pass: small tiles keep a short array's passes spread over the
// GPU and their serial ranking rounds few; large ones shorten the look-back's
// chain of tiles. Whole step in us, tiles of 512 x 2 / 512 x 4 / 512 x 8 keys
// (256 x 16 with __match_any_sync before): 1,024 vertices 169 / 172 / 179
// (196), 65,537 311 / 316 / 323 (358), 262,144 639 / 636 / 635 (669), 0.75M
// in 512 graphs 974 / 972 / 951 (983), 1,048,576 1583 / 1570 / 1534 (1575).
constexpr size_t kSmallSort = 1u << 17;
// k_radix_small up to here: whole step in us, one block / six launches: 300
// vertices 72 / 84, 1,024 82 / 96, 2,000 94 / 106, 3,000 104 / 107, 4,000 110
// / 111; eight rounds for 8,192 keys would take 143 / 125.
constexpr size_t kBlockSort = 4096;

static SortShape sort_shape(size_t n) {
  if (n <= kSmallSort) return {kSortThreads, 2};
  return {kSortThreads, 8};
}

static size_t sort_tiles(size_t n) {
  const size_t t = sort_shape(n).tile();
  return (n + t - 1) / t;
}

size_t sort_state_entries(size_t n) {
  const size_t tiles = sort_tiles(n);
  // per pass the global counts of 256 digits and a ticket, then per pass and
  // tile 256 status words (all 32 bits)
  return (size_t)kSortPasses * (256 * (tiles ? tiles : 1) + 256 + 1);
}

// Where the caller counts the first sorted digit (GVIZ_SORT_SKIP_BITS up) of
// the keys before radix_sort_pairs, in the zeroed sort state.
uint32_t *sort_digit_counts(gvizCudaForce *h) { return h->d_sortState; }

// Exclusive scan of n uint32 (n <= 2^31); in == out allowed. total may be
// nullptr or a device pointer receiving the sum.
void scan_exclusive(gvizCudaForce *h, const uint32_t *in, uint32_t *out,
                    size_t n, uint32_t *total) {
  if (n == 0) {
    if (total) cudaMemsetAsync(total, 0, sizeof(uint32_t), h->stream);
    return;
  }
  if (n <= kSingleMax) {
    launch_after(h->stream, k_scan_single, 1, kTopThreads, 0, in, out, (uint32_t)n, total);
    return;
  }
  const uint32_t tiles = (uint32_t)((n + kScanTile - 1) / kScanTile);
  cudaMemsetAsync(h->d_scanState, 0, (tiles + 1) * sizeof(uint64_t), h->stream);
  k_scan_onepass<<<tiles, kScanThreads, 0, h->stream>>>(in, out, (uint32_t)n, h->d_scanState,
                                                        total, h->d_status);
}

// The scatter's shared memory exceeds the default per-block budget: opted
// into once per device, at handle creation (outside any stream capture).
void sort_set_smem_limits() {
  small_sort_limit<512, 2>();
  small_sort_limit<1024, 2>();
  small_sort_limit<1024, 4>();
  cudaFuncSetAttribute(k_radix_onesweep<kSortThreads, 8>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)scatter_dyn(kSortThreads * 8));
}

// Stable sort by the key bits above GVIZ_SORT_SKIP_BITS (an even number of
// 8-bit passes, so the result ends in (keys, vals)); keys equal in those bits
// keep their input order. The sort state is zero but for the first digit's
// counts.
void radix_sort_pairs(gvizCudaForce *h, uint64_t *keys, uint32_t *vals,
                      uint64_t *keysAlt, uint32_t *valsAlt, size_t n) {
  if (n <= 1) return;
  if (n <= kBlockSort) {
    if (n <= 1024) small_sort<512, 2>(h, keys, vals, n);
    else if (n <= 2048) small_sort<1024, 2>(h, keys, vals, n);
    else small_sort<1024, 4>(h, keys, vals, n);
    prof_mark(h, "radix_sort");
    return;
  }
  const SortShape shape = sort_shape(n);
  const uint32_t tiles = (uint32_t)sort_tiles(n);
  uint32_t *ghist = sort_digit_counts(h);
  uint32_t *tickets = ghist + kSortPasses * 256;
  uint32_t *state = tickets + kSortPasses;
  uint64_t *ka = keys, *kb = keysAlt;
  uint32_t *va = vals, *vb = valsAlt;
  for (int pass = 0; pass < kSortPasses; pass++) {
    const auto kernel =
        shape.rounds == 2 ? k_radix_onesweep<kSortThreads, 2> : k_radix_onesweep<kSortThreads, 8>;
    launch_after(h->stream, kernel, tiles, shape.threads, scatter_dyn(shape.tile()), ka, va, kb,
                 vb, (uint32_t)n, pass, ghist, state + (size_t)pass * 256 * tiles,
                 tickets + pass, h->d_status);
    std::swap(ka, kb);
    std::swap(va, vb);
  }
  prof_mark(h, "radix_sort");
}
