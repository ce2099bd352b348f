// tree.cu -- device rebuild of gviz's quadtree (src/ds/gvizQuadtree.c) as a
// compressed, preorder-laid-out tree whose leaves hold exactly the point
// sets of the reference's leaves.
//
// Pipeline (one launch each, no host synchronisation):
//   bounding box per graph (gvizQuadtree.c:165-178)
//   per point: root box and quadrant path by replaying the reference's FP64
//     descent (QuadrantFor :65-73 against centres cx +/- halfSize/2,
//     Subdivide :75-92)
//   stable radix sort of (graph, path) -> fix-up sort of equal-prefix runs
//   buckets = identical full paths -> Karras binary radix tree (2012)
//   binary nodes merged into quadtree nodes (two path bits per level)
//   bottom-up mass / centre-of-mass / subtree sizes (arrival counters)
//     through shared memory: blocks of 256 buckets, then blocks of 4,096 for
//     the few nodes spanning those, then one block for the rest; the last two
//     also give those nodes' preorder positions
//   every node record at its preorder position, its own walk up weighted
//   parent links stopping at the first ancestor above blocks
//
// Why the compressed tree walks like the reference's: a chain of single-child
// nodes shares one point set, hence one mass and centre of mass; the
// reference accepts some chain node iff it accepts the deepest one (the
// ratio only shrinks going down), so one node per chain, tested with the
// deepest chain halfSize, gives the same pseudo-bodies. Leaves are never
// tested (gvizForceEmbedder.c:41-53); an overflow leaf below a chain is
// tested with its parent's halfSize. Empty children are skipped there too
// (mass == 0, :38-39).
#include <math.h>

#include <algorithm>

#include <cuda/atomic>

#include "internal.cuh"
#include "scan.cuh"

// Super-ranges such that neither level's lists outgrow k_top's shared memory:
// about 8 nodes span a block's edge, so 2^12, 2^14, 2^15 and 2^16 buckets have
// level-1 lists of ~120, ~500, ~1,000 and ~2,000 nodes, and level 2 has as many
// per 16, 64, 128 and 256 super-ranges. Node phase in us with 14 / 15 / 16 bits:
// BA 1,500,000 371 / 358 / 596, 3,000,000 869 / 679 / 893, R-MAT 4,194,304 1,634
// / 1,342 / 1,601.
static int super_bits(size_t V) {
  return V <= (1u << 17) ? 12 : (V <= (1u << 20) ? 14 : (V <= (1u << 22) ? 15 : 16));
}

// super-ranges of the tree build's nodes above blocks (see node_level)
size_t top_count_entries(size_t V) { return (V >> super_bits(V)) + 1; }

namespace {

constexpr int kThreads = 256;


// ---------------------------------------------------------------------------
// bounding boxes and roots
// ---------------------------------------------------------------------------

// A double as an unsigned integer of the same order, for atomic min and max.
__device__ __forceinline__ uint64_t ordered_bits(double x) {
  const uint64_t b = (uint64_t)__double_as_longlong(x);
  return b >> 63 ? ~b : b | 0x8000000000000000ull;
}
__device__ __forceinline__ double from_ordered_bits(uint64_t u) {
  return __longlong_as_double((long long)(u >> 63 ? u ^ 0x8000000000000000ull : ~u));
}

// Bounding box of every graph: box[4g..] = the largest ordered bits of -min x,
// max x, -min y, max y over its points (zero at the start: below every
// double's). Minimum and maximum are order-free, so the box is exact however
// the chunks' atomics interleave.
__global__ __launch_bounds__(kThreads) void k_bbox_chunks(
    const double2 *__restrict__ pos, const uint32_t *__restrict__ cb,
    const uint32_t *__restrict__ ce, const uint32_t *__restrict__ cg, unsigned long long *box,
    uint32_t *status) {
  step_order();
  const uint32_t b = cb[blockIdx.x], e = ce[blockIdx.x];
  double mnx = INFINITY, mxx = -INFINITY, mny = INFINITY, mxy = -INFINITY;
  int bad = 0;
  double2 p[GVIZ_CHUNK / kThreads];  // the chunk's loads, all in flight at once
#pragma unroll
  for (int r = 0; r < GVIZ_CHUNK / kThreads; r++) {
    const uint32_t i = b + r * kThreads + threadIdx.x;
    p[r] = pos[min(i, e - 1u)];
  }
#pragma unroll
  for (int r = 0; r < GVIZ_CHUNK / kThreads; r++) {
    if (!isfinite(p[r].x) || !isfinite(p[r].y)) bad = 1;
    mnx = fmin(mnx, p[r].x);
    mxx = fmax(mxx, p[r].x);
    mny = fmin(mny, p[r].y);
    mxy = fmax(mxy, p[r].y);
  }
  for (int o = 16; o > 0; o >>= 1) {
    mnx = fmin(mnx, __shfl_xor_sync(0xffffffffu, mnx, o));
    mxx = fmax(mxx, __shfl_xor_sync(0xffffffffu, mxx, o));
    mny = fmin(mny, __shfl_xor_sync(0xffffffffu, mny, o));
    mxy = fmax(mxy, __shfl_xor_sync(0xffffffffu, mxy, o));
  }
  __shared__ double4 wb[kThreads / 32];
  if (lane_id() == 0) wb[threadIdx.x >> 5] = make_double4(mnx, mxx, mny, mxy);
  if (bad) atomicOr(status, GVIZ_ST_NONFINITE);
  __syncthreads();
  if (threadIdx.x < 4) {
    const double *w = reinterpret_cast<const double *>(wb) + threadIdx.x;
    double r = w[0];
    for (int k = 1; k < kThreads / 32; k++)
      r = (threadIdx.x & 1u) ? fmax(r, w[4 * k]) : fmin(r, w[4 * k]);
    atomicMax(box + 4 * (size_t)cg[blockIdx.x] + threadIdx.x,
              (unsigned long long)ordered_bits((threadIdx.x & 1u) ? r : -r));
  }
}

// The root box of gvizQuadtreeBuild (src/ds/gvizQuadtree.c:165-178) from a
// graph's bounding box. D, the first depth whose half size is at most 1e-9,
// follows from the exponents (halving is exact).
__device__ __forceinline__ GraphRoot graph_root(const unsigned long long *box) {
  const double mnx = -from_ordered_bits(box[0]), mxx = from_ordered_bits(box[1]);
  const double mny = -from_ordered_bits(box[2]), mxy = from_ordered_bits(box[3]);
  GraphRoot R;
  R.cx = R.cy = 0.0;
  R.h0 = 1.0;
  R.D = R.capped = 0;
  if (!(mnx <= mxx)) return R;  // every position NaN: an error that the status reports
  const double sx = mxx - mnx, sy = mxy - mny;
  const double span = sx > sy ? sx : sy;
  R.h0 = span > 0.0 ? span / 2.0 : 1.0;
  R.cx = (mnx + mxx) / 2.0;
  R.cy = (mny + mxy) / 2.0;
  const long long hb = __double_as_longlong(R.h0), lb = __double_as_longlong(1e-9);
  const int up = (int)(hb >> 52) - (int)(lb >> 52);  // h0 > 0: no sign bit
  const int d = up + ((hb & 0xfffffffffffffll) > (lb & 0xfffffffffffffll) ? 1 : 0);
  R.D = min(max(d, 0), 64);
  R.capped = d > 64 ? 1 : 0;
  return R;
}

// Sixteen levels (or n < 16) of the descent from centre (cx, cy) and half
// size h: the digits of 16 levels, the first in the top bits. The sign of
// p - c, which is exact, gives the side: QuadrantFor's p >= c is its clear
// sign bit unless p is -0.0 (-0.0 - 0.0 is -0.0), which p must not be; c moves
// by h / 2 with that sign. Halving subtracts one from h's exponent (h > 1e-9
// here).
__device__ __forceinline__ uint32_t path_digits(double2 p, double &cx, double &cy, double &h,
                                                int n) {
  uint32_t w = 0;
  auto level = [&]() {
    const uint32_t tx = (uint32_t)__double2hiint(p.x - cx);
    const uint32_t ty = (uint32_t)__double2hiint(p.y - cy);
    const uint32_t hh = (uint32_t)__double2hiint(h) - 0x00100000u;
    const int hl = __double2loint(h);
    w = __funnelshift_l(ty, w, 1);  // south
    w = __funnelshift_l(tx, w, 1);  // west
    cx += __hiloint2double((int)(hh | (tx & 0x80000000u)), hl);
    cy += __hiloint2double((int)(hh | (ty & 0x80000000u)), hl);
    h = __hiloint2double((int)hh, hl);
  };
  if (n >= 16) {
#pragma unroll
    for (int d = 0; d < 16; d++) level();
    return w ^ 0x55555555u;  // west to east
  }
#pragma unroll 1
  for (int d = 0; d < n; d++) level();
  return n > 0 ? (w ^ (0x55555555u >> (32 - 2 * n))) << (32 - 2 * n) : 0u;
}

// Quadrant path of a point: digit = (north ? 0 : 2) + (east ? 1 : 0), i.e.
// NW=0 NE=1 SW=2 SE=3 (include/ds/gvizQuadtree.h:11-17), so sorted paths are
// the reference's depth-first NW,NE,SW,SE order. lo is the digits of levels
// 33 to 64 (FULL only).
template <bool FULL>
__device__ __forceinline__ uint64_t quadrant_path(double2 p, const GraphRoot &R, uint64_t &lo) {
  double cx = R.cx, cy = R.cy, h = R.h0;
  p.x = __dadd_rn(p.x, 0.0);  // -0.0 becomes 0.0, nothing else changes
  p.y = __dadd_rn(p.y, 0.0);
  const uint32_t w0 = path_digits(p, cx, cy, h, R.D);
  const uint32_t w1 = path_digits(p, cx, cy, h, R.D - 16);
  if (FULL) {
    const uint32_t w2 = path_digits(p, cx, cy, h, R.D - 32);
    const uint32_t w3 = path_digits(p, cx, cy, h, R.D - 48);
    lo = ((uint64_t)w2 << 32) | w3;
  }
  return ((uint64_t)w0 << 32) | w1;
}

// Composite sort key (graph, quadrant path) of every point, and the counts of
// the first sorted digit. Only the first 32 levels are descended here: the
// sort orders the top 48 bits, and the few points whose sorted bits meet
// another's take their whole path in k_runs. The descent replays the
// reference's FP64 steps, 9 instructions per level, four of them FP64. Eight
// blocks per SM stride over the points: a block's 256 counts go to the same
// few cache lines as every other's, and 4,096 blocks of one point per thread
// spend 16 us on them. 23 us at 1,048,576 points; all levels at 35
// instructions each, and the counts in a pass of their own, 60.
__global__ __launch_bounds__(kThreads) void k_keys(
    const double2 *__restrict__ pos, const uint32_t *__restrict__ gid,
    const unsigned long long *__restrict__ box, GraphRoot *roots, uint64_t *ck, uint32_t *idx,
    uint32_t *digits, uint32_t *status, uint32_t V, int gbits) {
  step_order();
  __shared__ uint32_t cnt[256];
  static_assert(kThreads == 256, "one thread per digit");
  cnt[threadIdx.x] = 0u;
  __syncthreads();
  for (uint32_t i = blockIdx.x * kThreads + threadIdx.x; i < V; i += gridDim.x * kThreads) {
    const uint32_t g = gid ? gid[i] : 0u;
    const double2 p = pos[i];
    const GraphRoot R = graph_root(box + 4 * (size_t)g);
    if (i == 0 || (gid && gid[i - 1] != g)) {  // the graph's first point
      roots[g] = R;
      if (R.capped) atomicOr(status, GVIZ_ST_DEPTH_CAP);
    }
    uint64_t lo;
    const uint64_t hi = quadrant_path<false>(p, R, lo);
    const uint64_t key = gbits ? (((uint64_t)g << (64 - gbits)) | (hi >> gbits)) : hi;
    ck[i] = key;
    idx[i] = i;
    atomicAdd(&cnt[(uint32_t)(key >> GVIZ_SORT_SKIP_BITS) & 255u], 1u);
  }
  __syncthreads();
  if (cnt[threadIdx.x]) atomicAdd(digits + threadIdx.x, cnt[threadIdx.x]);
}

// ---------------------------------------------------------------------------
// runs of equal composite keys
// ---------------------------------------------------------------------------

// The sorted points' paths, from the composite keys themselves. A point whose
// sorted bits (the top 48) differ from its neighbours' needs no more than
// the key holds. Runs of equal sorted bits of 2..k points lie in one leaf:
// their paths are cut to the common prefix (the leaf keeps them in vertex
// order, as the reference does). The points of longer runs take their whole
// path from the descent, and the run's first point lists the run, whose end
// it finds by a galloping search, for k_sort_runs. One pass over keys in
// order, 28 B per point, no gathers but those points'.
__global__ __launch_bounds__(kThreads) void k_runs(
    const uint64_t *__restrict__ ck, const uint32_t *__restrict__ idx,
    const double2 *__restrict__ pos, const GraphRoot *__restrict__ roots, uint32_t *counts,
    uint32_t *deep, uint64_t *sHi, uint64_t *sLo, uint32_t V, uint32_t k, int gbits) {
  step_order();
  const uint32_t s = blockIdx.x * kThreads + threadIdx.x;
  if (s >= V) return;
  const uint64_t full = ck[s];
  const uint64_t key = full >> GVIZ_SORT_SKIP_BITS;
  uint64_t hi = full << gbits, lo = 0;
  uint32_t back = 0, fwd = 0;  // equal keys before and after, counted to k
  while (back < k && back < s && (ck[s - back - 1u] >> GVIZ_SORT_SKIP_BITS) == key) back++;
  while (back + fwd < k && s + fwd + 1u < V && (ck[s + fwd + 1u] >> GVIZ_SORT_SKIP_BITS) == key)
    fwd++;
  if (back + fwd >= k) {  // more than k points
    const uint32_t g = gbits ? (uint32_t)(full >> (64 - gbits)) : 0u;
    hi = quadrant_path<true>(pos[idx[s]], roots[g], lo);
    if (back == 0) {
      uint32_t last = s + fwd, hiS = V;  // the run's end is in (last, hiS]
      for (uint32_t step = 1u;; step <<= 1) {
        const uint32_t probe = last + step;
        if (probe >= V || probe < last) break;
        if ((ck[probe] >> GVIZ_SORT_SKIP_BITS) != key) {
          hiS = probe;
          break;
        }
        last = probe;
      }
      while (hiS - last > 1u) {
        const uint32_t mid = last + (hiS - last) / 2u;
        if ((ck[mid] >> GVIZ_SORT_SKIP_BITS) == key)
          last = mid;
        else
          hiS = mid;
      }
      const uint32_t slot = atomicAdd(&counts[1], 1u);
      deep[2 * slot] = s;
      deep[2 * slot + 1] = hiS - s;
    }
  } else if (back + fwd > 0) {
    hi = (key << GVIZ_SORT_SKIP_BITS) << gbits;
  }
  sHi[s] = hi;
  sLo[s] = lo;
}

__device__ __forceinline__ bool key_less(uint64_t ah, uint64_t al, uint32_t av,
                                         uint64_t bh, uint64_t bl, uint32_t bv) {
  if (ah != bh) return ah < bh;
  if (al != bl) return al < bl;
  return av < bv;
}

// Bitonic sort of each deep run by (full path, vertex index) in shared memory.
__global__ __launch_bounds__(512) void k_sort_runs(
    uint64_t *sHi, uint64_t *sLo, uint32_t *idx, const uint32_t *__restrict__ deep,
    const uint32_t *__restrict__ counts, uint32_t *status) {
  step_order();
  extern __shared__ unsigned char smem[];
  uint64_t *kh = reinterpret_cast<uint64_t *>(smem);
  uint64_t *kl = kh + GVIZ_FIX_MAX;
  uint32_t *kv = reinterpret_cast<uint32_t *>(kl + GVIZ_FIX_MAX);
  const uint32_t nDeep = counts[1];
  for (uint32_t r = blockIdx.x; r < nDeep; r += gridDim.x) {
    const uint32_t start = deep[2 * r], len = deep[2 * r + 1];
    if (len > GVIZ_FIX_MAX) {
      int diff = 0;
      for (uint32_t j = threadIdx.x; j < len; j += blockDim.x) {
        if (sHi[start + j] != sHi[start] || sLo[start + j] != sLo[start]) diff = 1;
      }
      if (__syncthreads_or(diff) && threadIdx.x == 0)
        atomicOr(status, GVIZ_ST_DEEP_RUN);
      continue;
    }
    uint32_t P = 1;
    while (P < len) P <<= 1;
    for (uint32_t j = threadIdx.x; j < P; j += blockDim.x) {
      if (j < len) {
        kh[j] = sHi[start + j];
        kl[j] = sLo[start + j];
        kv[j] = idx[start + j];
      } else {
        kh[j] = ~0ull;
        kl[j] = ~0ull;
        kv[j] = ~0u;
      }
    }
    __syncthreads();
    for (uint32_t size = 2; size <= P; size <<= 1) {
      for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
        for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) {
          uint32_t j = i ^ stride;
          if (j > i) {
            bool asc = (i & size) == 0;
            bool gt = key_less(kh[j], kl[j], kv[j], kh[i], kl[i], kv[i]);
            if (gt == asc) {
              uint64_t t64 = kh[i];
              kh[i] = kh[j];
              kh[j] = t64;
              t64 = kl[i];
              kl[i] = kl[j];
              kl[j] = t64;
              uint32_t t32 = kv[i];
              kv[i] = kv[j];
              kv[j] = t32;
            }
          }
        }
        __syncthreads();
      }
    }
    for (uint32_t j = threadIdx.x; j < len; j += blockDim.x) {
      sHi[start + j] = kh[j];
      sLo[start + j] = kl[j];
      idx[start + j] = kv[j];
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// buckets (identical full paths) and the binary radix tree
// ---------------------------------------------------------------------------

// Buckets, the runs of identical full paths, numbered by a single-pass scan
// (sort.cu): a warp takes 256 consecutive sorted points in rounds of 32, the
// ballot of bucket starts gives each its number in the warp. Where k_sort_runs
// left a run too long for it unsorted (GVIZ_ST_DEEP_RUN, an error of the
// call), there are no buckets and so no tree: the kernels that follow need
// sorted keys, without them a node's children may lie outside its range.
__global__ __launch_bounds__(kThreads) void k_buckets(
    const uint64_t *__restrict__ sHi, const uint64_t *__restrict__ sLo,
    const uint64_t *__restrict__ ck, uint32_t *bStart, uint64_t *bHi, uint64_t *bLo,
    uint32_t *bGid, uint2 *upLeaf, uint64_t *state, uint32_t *total, uint32_t *status, uint32_t V,
    int gbits) {
  step_order();
  constexpr int kRounds = GVIZ_SCAN_TILE / kThreads;
  __shared__ uint32_t sTile;
  const uint32_t unsorted = *status & GVIZ_ST_DEEP_RUN;
  if (threadIdx.x == 0) sTile = scan_ticket(state);
  __syncthreads();
  if (unsorted) return;
  const uint32_t tile = sTile;
  const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
  const uint32_t s0 = tile * GVIZ_SCAN_TILE + w * (32u * kRounds) + lane;
  uint64_t hi[kRounds], lo[kRounds];
  uint32_t starts[kRounds], g[kRounds];
  uint32_t count = 0;
#pragma unroll
  for (int r = 0; r < kRounds; r++) {
    const uint32_t s = min(s0 + 32u * r, V - 1u);
    hi[r] = sHi[s];
    lo[r] = sLo[s];
    g[r] = gbits ? (uint32_t)(ck[s] >> (64 - gbits)) : 0u;
  }
#pragma unroll
  for (int r = 0; r < kRounds; r++) {
    const uint32_t s = s0 + 32u * r;
    uint64_t ph = __shfl_up_sync(0xffffffffu, hi[r], 1);
    uint64_t pl = __shfl_up_sync(0xffffffffu, lo[r], 1);
    uint32_t pg = __shfl_up_sync(0xffffffffu, g[r], 1);
    if (lane == 0 && s > 0 && s < V) {
      ph = sHi[s - 1u];
      pl = sLo[s - 1u];
      pg = gbits ? (uint32_t)(ck[s - 1u] >> (64 - gbits)) : 0u;
    }
    const bool start = s < V && (s == 0 || ph != hi[r] || pl != lo[r] || pg != g[r]);
    starts[r] = __ballot_sync(0xffffffffu, start);
    count += __popc(starts[r]);
  }
  const uint32_t nTiles = (V + GVIZ_SCAN_TILE - 1u) / GVIZ_SCAN_TILE;
  uint32_t b = scan_tile_prefix<kThreads>(state, tile, count, nTiles, total, status);
#pragma unroll
  for (int r = 0; r < kRounds; r++) {
    if ((starts[r] >> lane) & 1u) {
      const uint32_t at = b + __popc(starts[r] & ((1u << lane) - 1u));
      bStart[at] = s0 + 32u * r;
      bHi[at] = hi[r];
      bLo[at] = lo[r];
      bGid[at] = g[r];
      upLeaf[at] = make_uint2(GVIZ_NONE, 0u);
    }
    b += __popc(starts[r]);
  }
}

// Common-prefix length in bits of the composite keys (graph id:32,
// path:128) of buckets a and b; -1 outside [0, U). Keys of buckets
// [T0, T0 + kKarrasTile) come from the block's shared-memory copy; bGid is
// null for a single graph (every graph id is 0).
constexpr int kKarrasTile = 3 * kThreads;

struct KarrasKeys {
  const uint64_t *bHi, *bLo;
  const uint32_t *bGid;
  const uint64_t *sHi, *sLo;  // shared copies of [T0, T0 + kKarrasTile)
  int T0, U;
  __device__ __forceinline__ uint64_t hi(int b) const {
    return (unsigned)(b - T0) < (unsigned)kKarrasTile ? sHi[b - T0] : bHi[b];
  }
  __device__ __forceinline__ uint64_t lo(int b) const {
    return (unsigned)(b - T0) < (unsigned)kKarrasTile ? sLo[b - T0] : bLo[b];
  }
};

__device__ __forceinline__ int bdelta(int a, int b, const KarrasKeys &k) {
  if (b < 0 || b >= k.U) return -1;
  if (k.bGid) {
    uint32_t gx = k.bGid[a] ^ k.bGid[b];
    if (gx) return __clz(gx);
  }
  uint64_t x = k.hi(a) ^ k.hi(b);
  if (x) return 32 + __clzll(x);
  x = k.lo(a) ^ k.lo(b);
  if (x) return 96 + __clzll(x);
  return 160;
}

// A node's sums are made by the smallest unit that holds all its buckets:
// level 0, a block of k_bottom_up (256 buckets); level 1, a block of k_top
// over a super-range of 2^superBits buckets; level 2, k_top's single block for
// the rest. Nodes that join graphs (a common prefix inside the graph id) are
// of no level. A Karras node is one end of its own range, so its index places
// it.
__device__ __forceinline__ int node_level(uint32_t p, int delta, uint32_t first, uint32_t last,
                                          uint32_t U, int superBits) {
  if (delta < 32) return 0;
  const uint32_t B0 = p & ~(uint32_t)(kThreads - 1);
  if (first >= B0 && last < min(B0 + kThreads, U)) return 0;
  return (first >> superBits) == (last >> superBits) ? 1 : 2;
}

// The listed nodes: those of level 1 by super-range (its list starts at its
// first bucket's index), those of level 2; and per node {kPreLocal, -} or,
// until k_top replaces it by the node's preorder position, {kPreListed +
// level, its place in its list}.
struct TopLists {
  uint32_t *list1, *count1, *list2, *count2;
  uint2 *pre;
  int superBits;
};
constexpr uint32_t kPreLocal = 0xFFFFFFFEu;
constexpr uint32_t kPreListed = 0xFFFFFF00u;  // + level

// Node i of the binary radix tree (Karras 2012, algorithm of section 4);
// returns its level (node_level).
__device__ __forceinline__ int karras_node(int i, const KarrasKeys &k, uint32_t *nLeft,
                                           uint32_t *nRight, uint32_t *nFirst, uint32_t *nLast,
                                           int32_t *nDelta, uint2 *upInt, uint2 *upLeaf,
                                           int superBits) {
  const int dir = (bdelta(i, i + 1, k) - bdelta(i, i - 1, k)) >= 0 ? 1 : -1;
  const int dmin = bdelta(i, i - dir, k);
  int lmax = 2;
  while (bdelta(i, i + lmax * dir, k) > dmin) lmax <<= 1;
  int l = 0;
  for (int t = lmax >> 1; t >= 1; t >>= 1)
    if (bdelta(i, i + (l + t) * dir, k) > dmin) l += t;
  const int j = i + l * dir;
  const int dnode = bdelta(i, j, k);
  int s = 0;
  int div = 2;
  int t;
  do {
    t = (l + div - 1) / div;
    if (bdelta(i, i + (s + t) * dir, k) > dnode) s += t;
    div <<= 1;
  } while (t > 1);
  const int gamma = i + s * dir + min(dir, 0);
  const int first = min(i, j), last = max(i, j);
  uint32_t left, right;
  if (first == gamma) {
    left = (uint32_t)gamma | GVIZ_LEAF_BIT;
    upLeaf[gamma].x = (uint32_t)i;
  } else {
    left = (uint32_t)gamma;
    upInt[gamma].x = (uint32_t)i;
  }
  if (last == gamma + 1) {
    right = (uint32_t)(gamma + 1) | GVIZ_LEAF_BIT;
    upLeaf[gamma + 1].x = (uint32_t)i;
  } else {
    right = (uint32_t)(gamma + 1);
    upInt[gamma + 1].x = (uint32_t)i;
  }
  nLeft[i] = left;
  nRight[i] = right;
  nFirst[i] = (uint32_t)first;
  nLast[i] = (uint32_t)last;
  nDelta[i] = dnode;
  if (i == 0) upInt[0].x = GVIZ_NONE;
  return node_level((uint32_t)i, dnode, (uint32_t)first, (uint32_t)last, (uint32_t)k.U,
                    superBits);
}

// Karras, "Maximizing parallelism in the construction of BVHs, octrees and
// k-d trees" (HPG 2012), algorithm of section 4 over unique bucket keys.
// Block j finds nodes [256 j, 256 j + 256); the keys of the 256 buckets on
// either side are staged in shared memory first, where most of the
// searches stay.
__global__ __launch_bounds__(kThreads) void k_karras(
    const uint64_t *__restrict__ bHi, const uint64_t *__restrict__ bLo,
    const uint32_t *__restrict__ bGid, const uint32_t *__restrict__ counts,
    uint32_t *nLeft, uint32_t *nRight, uint32_t *nFirst, uint32_t *nLast,
    int32_t *nDelta, uint2 *upInt, uint2 *upLeaf, TopLists top) {
  step_order();
  __shared__ uint64_t sHi[kKarrasTile], sLo[kKarrasTile];
  __shared__ uint32_t sCount[2], sBase[2];
  const int U = (int)counts[2];
  const int B0 = (int)(blockIdx.x * kThreads);
  if (B0 >= U - 1) return;
  if (threadIdx.x < 2) sCount[threadIdx.x] = 0u;
  KarrasKeys k{bHi, bLo, bGid, sHi, sLo, B0 - kThreads, U};
  for (int j = threadIdx.x; j < kKarrasTile; j += kThreads) {
    const int b = k.T0 + j;
    if (b >= 0 && b < U) {
      sHi[j] = bHi[b];
      sLo[j] = bLo[b];
    }
  }
  __syncthreads();
  const int i = B0 + threadIdx.x;
  int level = 0;
  if (i < U - 1)
    level = karras_node(i, k, nLeft, nRight, nFirst, nLast, nDelta, upInt, upLeaf, top.superBits);
  // the block's nodes above blocks join their level's list
  uint32_t at = 0;
  if (level > 0) at = atomicAdd(&sCount[level - 1], 1u);
  __syncthreads();
  if (threadIdx.x < 2 && sCount[threadIdx.x])
    sBase[threadIdx.x] = atomicAdd(threadIdx.x ? top.count2 : top.count1 + (B0 >> top.superBits),
                                   sCount[threadIdx.x]);
  __syncthreads();
  if (level > 0) {
    at += sBase[level - 1];
    uint32_t *const list1 = top.list1 + ((B0 >> top.superBits) << top.superBits);
    (level == 1 ? list1 : top.list2)[at] = (uint32_t)i;
    top.pre[i] = make_uint2(kPreListed + (uint32_t)level, at);
  } else if (i < U - 1) {
    top.pre[i] = make_uint2(kPreLocal, 0u);
  }
}
struct BU {
  const uint32_t *idx, *bStart, *bGid, *counts, *nLeft, *nRight, *nFirst, *nLast;
  const int32_t *nDelta;
  const double *mass;
  const double2 *pos;
  uint2 *upInt, *upLeaf;
  uint32_t *nCounter;
  double *bM, *bSX, *bSY, *nM, *nSX, *nSY;
  uint32_t *bCnt, *bT, *nCnt, *nT, *nFlag, *rootNode, *rootT, *status;
  // second central moments {Qxx, Qxy, Qyy, -}, or null: summed and shifted
  // in FP64, stored in FP32 (they only feed FP32 features)
  float4 *bQ, *nQ;
  TopLists top;
  uint32_t *total;  // single graph: the number of records (else null)
  uint32_t V, k;
};

// x is its graph's root: T records
__device__ __forceinline__ void put_root(const BU &a, uint32_t g, uint32_t x, uint32_t T) {
  a.rootNode[g] = x;
  a.rootT[g] = T;
  if (a.total) *a.total = T;
}

// second central moments of a child about its own centre of mass
__device__ __forceinline__ float4 child_q(const BU &a, uint32_t c) {
  return (c & GVIZ_LEAF_BIT) ? a.bQ[c & ~GVIZ_LEAF_BIT] : a.nQ[c];
}

// parallel-axis shift of a child's moments to the parent's centre of mass
// (px, py): M_c (c_c - p)^2 = (S_c - M_c p)^2 / M_c, the difference in FP64,
// the rest in FP32 like the stored moments
__device__ __forceinline__ void add_shifted(float4 &q, const float4 qc, double M, double SX,
                                            double SY, double px, double py) {
  q.x += qc.x;
  q.y += qc.y;
  q.z += qc.z;
  if (M > 1e-9 || M < -1e-9) {
    const float tx = (float)(SX - M * px), ty = (float)(SY - M * py);
    const float im = 1.0f / (float)M;
    q.x += tx * tx * im;
    q.y += tx * ty * im;
    q.z += ty * ty * im;
  }
}

__device__ __forceinline__ void child_vals(const BU &a, uint32_t c, double &M,
                                           double &SX, double &SY,
                                           uint32_t &cnt, uint32_t &T) {
  // plain loads: the acquire on the arrival counter (block or device scope)
  // makes the sibling's stores visible
  if (c & GVIZ_LEAF_BIT) {
    uint32_t b = c & ~GVIZ_LEAF_BIT;
    M = a.bM[b];
    SX = a.bSX[b];
    SY = a.bSY[b];
    cnt = a.bCnt[b];
    T = a.bT[b];
  } else {
    M = a.nM[c];
    SX = a.nSX[c];
    SY = a.nSY[c];
    cnt = a.nCnt[c];
    T = a.nT[c];
  }
}

__device__ __forceinline__ uint2 *up_of(const BU &a, uint32_t c) {
  return (c & GVIZ_LEAF_BIT) ? a.upLeaf + (c & ~GVIZ_LEAF_BIT) : a.upInt + c;
}

// A node from its children's sums (left first: fixed order, deterministic
// sums): mass, mass-weighted position sums, point count, subtree size in
// emitted records, the absorbed and collapsed (a capacity leaf) flags and its
// children's preorder link weights wl, wr; with kQ the second moments about
// its centre of mass.
struct TopSums {
  double M, SX, SY;
  uint32_t cnt, T;
  float4 q;
};

struct Combined {
  TopSums s;
  uint32_t flag, wl, wr;
};

template <bool kQ>
__device__ __forceinline__ Combined combined(const BU &a, bool absorbed, const TopSums &L,
                                             const TopSums &R) {
  Combined c;
  c.s.M = L.M + R.M;
  c.s.SX = L.SX + R.SX;
  c.s.SY = L.SY + R.SY;
  c.s.cnt = L.cnt + R.cnt;
  const bool collapsed = !absorbed && c.s.cnt <= a.k;
  c.s.T = absorbed ? L.T + R.T : (collapsed ? 1u + c.s.cnt : 1u + L.T + R.T);
  c.s.q = make_float4(0.f, 0.f, 0.f, 0.f);
  if (kQ) {
    double px = 0.0, py = 0.0;
    if (c.s.M > 1e-9 || c.s.M < -1e-9) {
      const double im = __drcp_rn(c.s.M);  // one reciprocal on the serial climb
      px = c.s.SX * im;
      py = c.s.SY * im;
    }
    add_shifted(c.s.q, L.q, L.M, L.SX, L.SY, px, py);
    add_shifted(c.s.q, R.q, R.M, R.SX, R.SY, px, py);
  }
  c.flag = (absorbed ? 1u : 0u) | (collapsed ? 2u : 0u);
  const uint32_t base = absorbed ? 0u : 1u;
  const uint32_t dead = collapsed ? 0x80000000u : 0u;
  c.wl = base | dead;
  c.wr = (base + L.T) | dead;
  return c;
}

// c to global memory: node p's sums and flags and its children's link weights
template <bool kQ>
__device__ __forceinline__ void put_combined(const BU &a, uint32_t p, uint32_t l, uint32_t r,
                                             const Combined &c) {
  if (kQ) a.nQ[p] = c.s.q;
  a.nM[p] = c.s.M;
  a.nSX[p] = c.s.SX;
  a.nSY[p] = c.s.SY;
  a.nCnt[p] = c.s.cnt;
  a.nT[p] = c.s.T;
  a.nFlag[p] = c.flag;
  up_of(a, l)->y = c.wl;
  up_of(a, r)->y = c.wr;
}

// p, of delta dp, shares its quadtree level with its binary parent, of delta
// dpp (none: dpp < 32): two path bits per level
__device__ __forceinline__ bool is_absorbed(int dp, int dpp) {
  return dpp >= 32 && ((dp - 32) >> 1) == ((dpp - 32) >> 1);
}

// Per-block shared state of k_bottom_up: the sums of the block's buckets
// [B0, B1) (slot b - B0), the sums of its in-block internal nodes (slot
// p - B0; a Karras node is one end of its own range, so an internal node
// whose bucket range lies in [B0, B1) has its index there too) and the shape
// of the internal nodes [B0, B1), loaded once and coalesced.
template <bool kQ>
struct BUShared {
  uint32_t arrive[kThreads];
  double lM[kThreads], lSX[kThreads], lSY[kThreads];
  double iM[kThreads], iSX[kThreads], iSY[kThreads];
  uint32_t lCnt[kThreads], lT[kThreads], iCnt[kThreads], iT[kThreads];
  uint32_t left[kThreads], right[kThreads], first[kThreads], last[kThreads], up[kThreads];
  int32_t delta[kThreads];
  float4 lQ[kQ ? kThreads : 1], iQ[kQ ? kThreads : 1];
};

// Sums per bucket, then each thread climbs; the second child to arrive at a
// node combines both (left first: fixed order, deterministic sums). A node
// whose buckets all belong to this block has both children summed by
// threads of this block: its arrivals meet in shared memory with block-scope
// ordering and its children's sums are read from shared memory. A climb
// stops at the first node spanning blocks, which k_top sums. Every node's
// sums also go to global memory (k_emit reads them).
template <bool kQ>
__global__ __launch_bounds__(kThreads) void k_bottom_up(BU a) {
  step_order();
  __shared__ BUShared<kQ> s;
  const uint32_t U = a.counts[2];
  const uint32_t B0 = blockIdx.x * kThreads;
  const uint32_t B1 = min(B0 + kThreads, U);
  const uint32_t tid = threadIdx.x;
  s.arrive[tid] = 0u;
  if (B0 + tid + 1 < U) {  // internal nodes are [0, U - 1)
    const uint32_t p = B0 + tid;
    s.left[tid] = a.nLeft[p];
    s.right[tid] = a.nRight[p];
    s.first[tid] = a.nFirst[p];
    s.last[tid] = a.nLast[p];
    s.up[tid] = a.upInt[p].x;
    s.delta[tid] = a.nDelta[p];
  }
  __syncthreads();
  const uint32_t b = B0 + tid;
  if (b >= U) return;
  const uint32_t start = a.bStart[b];
  const uint32_t end = (b + 1 < U) ? a.bStart[b + 1] : a.V;
  double M = 0.0, SX = 0.0, SY = 0.0;
  for (uint32_t j = start; j < end; j++) {
    uint32_t i = a.idx[j];
    double m = a.mass[i];
    double2 p = a.pos[i];
    M += m;
    SX += m * p.x;
    SY += m * p.y;
  }
  uint32_t cnt = end - start;
  uint32_t T = cnt == 1 ? 1u : 1u + cnt;
  if (kQ) {
    double cx = 0.0, cy = 0.0;
    if (M > 1e-9 || M < -1e-9) {
      cx = SX / M;
      cy = SY / M;
    }
    // a single point has no second moments about itself: the bucket's own
    // pass over its points runs only for two or more
    double4 q = make_double4(0.0, 0.0, 0.0, 0.0);
    for (uint32_t j = start; cnt > 1u && j < end; j++) {
      const uint32_t i = a.idx[j];
      const double m = a.mass[i];
      const double2 p = a.pos[i];
      const double dx = p.x - cx, dy = p.y - cy;
      q.x += m * dx * dx;
      q.y += m * dx * dy;
      q.z += m * dy * dy;
    }
    const float4 fq = make_float4((float)q.x, (float)q.y, (float)q.z, 0.f);
    a.bQ[b] = fq;
    s.lQ[tid] = fq;
  }
  a.bM[b] = M;
  a.bSX[b] = SX;
  a.bSY[b] = SY;
  a.bCnt[b] = cnt;
  a.bT[b] = T;
  s.lM[tid] = M;
  s.lSX[tid] = SX;
  s.lSY[tid] = SY;
  s.lCnt[tid] = cnt;
  s.lT[tid] = T;
  const uint32_t g = a.bGid[b];
  uint32_t x = b | GVIZ_LEAF_BIT;
  uint32_t p = a.upLeaf[b].x;
  for (int guard = 0;; guard++) {
    if (guard > GVIZ_MAX_CLIMB) {
      atomicOr(a.status, GVIZ_ST_TREE);
      return;
    }
    const bool pin = p >= B0 && p < B1;  // false for GVIZ_NONE
    const int dp = p == GVIZ_NONE ? 0 : (pin ? s.delta[p - B0] : a.nDelta[p]);
    if (p == GVIZ_NONE || dp < 32) {
      put_root(a, g, x, T);
      *up_of(a, x) = make_uint2(GVIZ_NONE, 0u);
      return;
    }
    if (!pin || s.first[p - B0] < B0 || s.last[p - B0] >= B1) return;  // spans blocks
    const uint32_t l = s.left[p - B0], r = s.right[p - B0], pp = s.up[p - B0];
    const int dpp = pp == GVIZ_NONE ? 0
                    : ((pp >= B0 && pp < B1) ? s.delta[pp - B0] : a.nDelta[pp]);
    // release this child's sums / acquire the sibling's: the second thread
    // to arrive combines both, reading them from shared memory (both
    // children lie in [B0, B1) and were summed by this block)
    cuda::atomic_ref<uint32_t, cuda::thread_scope_block> arrivals(s.arrive[p - B0]);
    if (arrivals.fetch_add(1u, cuda::memory_order_acq_rel) == 0u) return;
    auto child = [&](uint32_t x) {
      TopSums t;
      const uint32_t c = (x & ~GVIZ_LEAF_BIT) - B0;
      t.q = make_float4(0.f, 0.f, 0.f, 0.f);
      if (x & GVIZ_LEAF_BIT) {
        t.M = s.lM[c], t.SX = s.lSX[c], t.SY = s.lSY[c], t.cnt = s.lCnt[c], t.T = s.lT[c];
        if (kQ) t.q = s.lQ[c];
      } else {
        t.M = s.iM[c], t.SX = s.iSX[c], t.SY = s.iSY[c], t.cnt = s.iCnt[c], t.T = s.iT[c];
        if (kQ) t.q = s.iQ[c];
      }
      return t;
    };
    const Combined z = combined<kQ>(a, is_absorbed(dp, dpp), child(l), child(r));
    put_combined<kQ>(a, p, l, r, z);
    const uint32_t c = p - B0;  // an in-block parent reads the sums from here
    s.iM[c] = z.s.M;
    s.iSX[c] = z.s.SX;
    s.iSY[c] = z.s.SY;
    s.iCnt[c] = z.s.cnt;
    s.iT[c] = T = z.s.T;
    if (kQ) s.iQ[c] = z.s.q;
    x = p;
    p = pp;
  }
}

// Sums and preorder positions of the nodes of one level's list, by one block:
// level 1, block s the list of super-range s; level 2, one block. A listed
// node's children are listed themselves or were summed by an earlier kernel.
// The block keeps the list's sums, links and arrivals in shared memory and
// climbs there: nodes without listed children are combined first, and the
// second listed child to be combined goes on with its parent. Then every
// node adds the link weights up to the last ancestor in the list: up to the
// graph's root that is its preorder position (without the graph base), below
// a node of level 2 it is relative to that last ancestor, which k_emit adds.
// A list above kTopCap nodes is worked off by the same block in global memory,
// slower at level 2 than the whole grid's climb was (33,554,432 uniform points,
// node phase 8.26 -> 8.80 ms; 256 clusters of 4,000 points over 40 nested
// octaves 0.53 -> 0.78), though no step measured is slower for it.
// Bound by latency: five dependent loads to fill a list, then one chain of
// shared-memory steps as deep as the tree above the blocks (15 to 26 levels
// here). One device-scope climb through those levels, a fence, an arrival and
// a reload of ~3 us each, took 59 us at 65,537 vertices and 71 at 1,048,576,
// and the positions 7 and 19 more; both kernels together take 23 and 47.
template <bool kQ, int CAP>
struct __align__(16) TopShared {
  double2 s0[CAP];        // M, SX
  double sy[CAP];
  uint2 ct[CAP];          // cnt, T
  uint4 node[CAP];        // children's places, absorbed, parent's place (kTop*)
  float4 q[kQ ? CAP : 1];
  uint32_t id[CAP], lc[CAP], rc[CAP];  // node ids: its own, its children's
  uint32_t w[CAP];            // weight (and dead bit) of the link to the parent
  uint32_t wl[CAP], wr[CAP];  // and of the links to the children
  uint32_t arrive[CAP];
  uint8_t listed[CAP];        // listed children: 0, 1, 2
};
constexpr uint32_t kTopRoot = 0xFFFFFFFFu;  // parent: none, the node is a graph's root
constexpr uint32_t kTopOut = 0xFFFFFFFEu;   // parent: of a higher level
constexpr uint32_t kTopTwo = 0x80000000u;   // parent's place: both its children are listed

template <bool kQ>
__device__ __forceinline__ TopSums summed_child(const BU &a, uint32_t c) {
  TopSums s;
  child_vals(a, c, s.M, s.SX, s.SY, s.cnt, s.T);
  s.q = kQ ? child_q(a, c) : make_float4(0.f, 0.f, 0.f, 0.f);
  return s;
}

__device__ __forceinline__ int level_of(const BU &a, uint32_t p, uint32_t U) {
  return node_level(p, a.nDelta[p], a.nFirst[p], a.nLast[p], U, a.top.superBits);
}

// A list too long for shared memory: the same climb and positions over the
// nodes' global sums, links and counters (block scope: no other block
// touches these nodes).
template <bool kQ>
__device__ void top_in_global(const BU &a, const uint32_t *list, uint32_t n, int level,
                              uint32_t U) {
  auto listed = [&](uint32_t c) {
    return !(c & GVIZ_LEAF_BIT) && level_of(a, c, U) == level;
  };
  for (uint32_t e = threadIdx.x; e < n; e += blockDim.x) {
    uint32_t p = list[e];
    if (listed(a.nLeft[p]) || listed(a.nRight[p])) continue;
    for (int guard = 0;; guard++) {
      if (guard > GVIZ_MAX_CLIMB) {
        atomicOr(a.status, GVIZ_ST_TREE);
        break;
      }
      const uint32_t l = a.nLeft[p], r = a.nRight[p], pp = a.upInt[p].x;
      const int dpp = pp == GVIZ_NONE ? 0 : a.nDelta[pp];
      const Combined z = combined<kQ>(a, is_absorbed(a.nDelta[p], dpp), summed_child<kQ>(a, l),
                                      summed_child<kQ>(a, r));
      put_combined<kQ>(a, p, l, r, z);
      if (dpp < 32) {
        put_root(a, a.bGid[a.nFirst[p]], p, z.s.T);
        *up_of(a, p) = make_uint2(GVIZ_NONE, 0u);
        break;
      }
      if (level_of(a, pp, U) != level) break;
      cuda::atomic_ref<uint32_t, cuda::thread_scope_block> arrivals(a.nCounter[pp]);
      const uint32_t need = (listed(a.nLeft[pp]) ? 1u : 0u) + (listed(a.nRight[pp]) ? 1u : 0u);
      if (arrivals.fetch_add(1u, cuda::memory_order_acq_rel) + 1u < need) break;
      a.nCounter[pp] = 0u;
      p = pp;
    }
  }
  __syncthreads();
  for (uint32_t e = threadIdx.x; e < n; e += blockDim.x) {
    uint32_t x = list[e], pre = 0, dead = 0;
    uint2 u = a.upInt[x];
    for (int guard = 0; u.x != GVIZ_NONE && level_of(a, u.x, U) == level; guard++) {
      if (guard > GVIZ_MAX_CLIMB) {
        dead = 1;
        break;
      }
      pre += u.y & 0x7fffffffu;
      dead |= u.y >> 31;
      x = u.x;
      u = a.upInt[x];
    }
    a.top.pre[list[e]] = make_uint2(dead ? GVIZ_NONE : pre, u.x == GVIZ_NONE ? GVIZ_NONE : x);
  }
}

template <bool kQ, int LEVEL, int CAP, int THREADS>
__global__ __launch_bounds__(THREADS) void k_top(BU a) {
  step_order();
  extern __shared__ __align__(16) unsigned char topDyn[];
  TopShared<kQ, CAP> &s = *reinterpret_cast<TopShared<kQ, CAP> *>(topDyn);
  const uint32_t n = LEVEL == 1 ? a.top.count1[blockIdx.x] : *a.top.count2;
  const uint32_t *list =
      LEVEL == 1 ? a.top.list1 + ((size_t)blockIdx.x << a.top.superBits) : a.top.list2;
  if (n > (uint32_t)CAP) {
    top_in_global<kQ>(a, list, n, LEVEL, a.counts[2]);
    return;
  }
  auto hold = [&](uint32_t e, const TopSums &c) {
    s.s0[e] = make_double2(c.M, c.SX);
    s.sy[e] = c.SY;
    s.ct[e] = make_uint2(c.cnt, c.T);
    if (kQ) s.q[e] = c.q;
  };
  auto held = [&](uint32_t e) {
    TopSums c;
    const double2 m = s.s0[e];
    const uint2 k = s.ct[e];
    c.M = m.x;
    c.SX = m.y;
    c.SY = s.sy[e];
    c.cnt = k.x;
    c.T = k.y;
    c.q = kQ ? s.q[e] : make_float4(0.f, 0.f, 0.f, 0.f);
    return c;
  };
  // every entry's shape, and the sums of the children summed before: of one
  // such child they are held in the entry's own place until it is combined,
  // an entry with two is combined right away
  for (uint32_t e = threadIdx.x; e < n; e += THREADS) {
    const uint32_t p = list[e];
    const uint32_t l = a.nLeft[p], r = a.nRight[p], pp = a.upInt[p].x;
    const int dp = a.nDelta[p], dpp = pp == GVIZ_NONE ? 0 : a.nDelta[pp];
    const uint2 none = make_uint2(kPreLocal, 0u);
    const uint2 tl = (l & GVIZ_LEAF_BIT) ? none : a.top.pre[l];
    const uint2 tr = (r & GVIZ_LEAF_BIT) ? none : a.top.pre[r];
    const uint2 tp = pp == GVIZ_NONE ? none : a.top.pre[pp];
    const bool inL = tl.x == kPreListed + LEVEL, inR = tr.x == kPreListed + LEVEL;
    const bool absorbed = is_absorbed(dp, dpp);
    const uint32_t par = dpp < 32 ? kTopRoot : (tp.x == kPreListed + LEVEL ? tp.y : kTopOut);
    s.node[e] = make_uint4(inL ? tl.y : e, inR ? tr.y : e, absorbed ? 1u : 0u, par);
    s.id[e] = p;
    s.lc[e] = l;
    s.rc[e] = r;
    s.arrive[e] = 0u;
    s.listed[e] = (inL ? 1 : 0) + (inR ? 1 : 0);
    if (!inL && !inR) {
      const Combined z =
          combined<kQ>(a, absorbed, summed_child<kQ>(a, l), summed_child<kQ>(a, r));
      hold(e, z.s);
      s.wl[e] = z.wl;
      s.wr[e] = z.wr;
    } else if (!inL || !inR) {
      hold(e, summed_child<kQ>(a, inL ? r : l));
    }
  }
  __syncthreads();
  for (uint32_t e = threadIdx.x; e < n; e += THREADS) {  // (places, or kTopOut and above)
    const uint32_t par = s.node[e].w;
    if (par < kTopOut && s.listed[par] == 2) s.node[e].w = par | kTopTwo;
  }
  __syncthreads();
  for (uint32_t e0 = threadIdx.x; e0 < n; e0 += THREADS) {
    if (s.listed[e0]) continue;
    uint32_t par = s.node[e0].w;
    for (int guard = 0; par < kTopOut; guard++) {
      if (guard > GVIZ_MAX_CLIMB) {
        atomicOr(a.status, GVIZ_ST_TREE);
        break;
      }
      const uint32_t e = par & ~kTopTwo;
      if (par & kTopTwo) {
        // release this child's sums, acquire the other's (both in shared memory)
        __threadfence_block();
        if (atomicAdd(&s.arrive[e], 1u) == 0u) break;
        __threadfence_block();
      }
      const uint4 nd = s.node[e];
      const Combined z = combined<kQ>(a, nd.z != 0u, held(nd.x), held(nd.y));
      hold(e, z.s);
      s.wl[e] = z.wl;
      s.wr[e] = z.wr;
      par = nd.w;
    }
  }
  __syncthreads();
  // each entry tells its listed children their links' weights
  for (uint32_t e = threadIdx.x; e < n; e += THREADS) {
    const uint4 nd = s.node[e];
    if (nd.x != e) s.w[nd.x] = s.wl[e];
    if (nd.y != e) s.w[nd.y] = s.wr[e];
  }
  __syncthreads();
  for (uint32_t e = threadIdx.x; e < n; e += THREADS) {
    const uint32_t p = s.id[e];
    const uint4 nd = s.node[e];
    Combined z;
    z.s = held(e);
    z.flag = nd.z | (nd.z == 0u && z.s.cnt <= a.k ? 2u : 0u);
    z.wl = s.wl[e];
    z.wr = s.wr[e];
    put_combined<kQ>(a, p, s.lc[e], s.rc[e], z);
    if (nd.w == kTopRoot) {
      put_root(a, a.bGid[a.nFirst[p]], p, z.s.T);
      *up_of(a, p) = make_uint2(GVIZ_NONE, 0u);
    }
    uint32_t x = e, par = nd.w, pre = 0, dead = 0;
    for (int guard = 0; par < kTopOut; guard++) {
      if (guard > GVIZ_MAX_CLIMB) {
        dead = 1;
        break;
      }
      pre += s.w[x] & 0x7fffffffu;
      dead |= s.w[x] >> 31;
      x = par & ~kTopTwo;
      par = s.node[x].w;
    }
    a.top.pre[p] = make_uint2(dead ? GVIZ_NONE : pre, par == kTopOut ? s.id[x] : GVIZ_NONE);
  }
}

constexpr int kTopCap = 2048;  // 156 KB of shared memory, 188 with second moments
// With 2^16 buckets to a super-range some lists are longer. All the shared memory
// there is leaves no L1: 30 us slower where 2,048 suffice (BA 1,500,000 401 against
// 371), but lists worked off in global memory take longer (R-MAT 4,194,304 with 16
// bits 1,393 against 1,601).
template <bool kQ>
constexpr int kTopCapLarge = kQ ? 2432 : 2944;
constexpr int kTop1Threads = 512, kTop2Threads = 1024;

template <bool kQ, int CAP>
void launch_top_cap(const BU &bu, uint32_t supers, cudaStream_t st) {
  constexpr size_t smem = sizeof(TopShared<kQ, CAP>);
  launch_after(st, k_top<kQ, 1, CAP, kTop1Threads>, supers, kTop1Threads, smem, bu);
  // a layout of one super-range has no nodes above it
  if (supers > 1) launch_after(st, k_top<kQ, 2, CAP, kTop2Threads>, 1, kTop2Threads, smem, bu);
}

template <bool kQ>
void launch_top(const BU &bu, uint32_t V, cudaStream_t st) {
  const uint32_t supers = (uint32_t)top_count_entries(V);
  if (super_bits(V) < 16) launch_top_cap<kQ, kTopCap>(bu, supers, st);
  else launch_top_cap<kQ, kTopCapLarge<kQ>>(bu, supers, st);
}

template <bool kQ, int CAP>
void top_smem_limits() {
  constexpr int smem = (int)sizeof(TopShared<kQ, CAP>);
  static_assert(smem <= 227 * 1024, "a block's shared memory");
  cudaFuncSetAttribute(k_top<kQ, 1, CAP, kTop1Threads>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  cudaFuncSetAttribute(k_top<kQ, 2, CAP, kTop2Threads>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}

// preorder position (without the graph base) and whether any ancestor is a
// collapsed (capacity) leaf
__device__ __forceinline__ void walk_up(uint2 u, const uint2 *__restrict__ upInt,
                                        uint32_t &pre, uint32_t &dead) {
  pre = 0;
  dead = 0;
  for (int guard = 0; u.x != GVIZ_NONE; guard++) {
    if (guard > GVIZ_MAX_CLIMB) {  // never expected: report as dead
      dead = 1;
      return;
    }
    pre += u.y & 0x7fffffffu;
    dead |= u.y >> 31;
    u = upInt[u.x];
  }
}

struct EM {
  const uint32_t *idx, *bStart, *bGid, *bCnt, *counts, *nFirst, *nLast, *nFlag,
      *nT, *nCnt, *graphBase, *nLeft, *nRight;
  const int32_t *nDelta;
  const uint2 *upInt, *upLeaf;
  const double *bM, *bSX, *bSY, *nM, *nSX, *nSY, *mass, *radius;
  const double2 *pos;
  const GraphRoot *roots;
  void *nodes;
  uint32_t *status;
  double theta;
  uint32_t V, k, maxNodes;
  int f64;
  // far-field side records (null unless requested)
  const float4 *bQ, *nQ;
  const uint64_t *bHi, *bLo;
  FarCell *cells;
  uint32_t *leafPre;
  uint32_t *cellCnt;  // per record: points below it, 1 for a point (null unless requested)
  uint4 *kids;        // per cell: its children's preorder slots (null unless requested)
  const uint2 *pre;  // per internal node: see k_top
};

__device__ __forceinline__ void put_count(const EM &a, uint32_t at, uint32_t c) {
  if (a.cellCnt && at < a.maxNodes) a.cellCnt[at] = c;
}

// the even bits of x (bit 2j -> bit j)
__device__ __forceinline__ uint64_t even_bits(uint64_t x) {
  x &= 0x5555555555555555ull;
  x = (x | (x >> 1)) & 0x3333333333333333ull;
  x = (x | (x >> 2)) & 0x0f0f0f0f0f0f0f0full;
  x = (x | (x >> 4)) & 0x00ff00ff00ff00ffull;
  x = (x | (x >> 8)) & 0x0000ffff0000ffffull;
  return (x | (x >> 16)) & 0x00000000ffffffffull;
}

// Geometric centre of the cell at `depth` on the path (hi, lo), in closed
// form: with E (S) the east (south) bits of the path's first `depth` levels
// read as an integer, the descent's steps of +-h0 / 2^d sum to
// cx = cx0 + h0 ((2E + 1) / 2^depth - 1), cy = cy0 - h0 ((2S + 1) / 2^depth - 1).
// (Only a model feature: FP64 rounding may differ from the step-by-step
// descent in the last bits.)
__device__ void cell_center(const GraphRoot &R, uint64_t hi, uint64_t lo,
                            int depth, double &cx, double &cy) {
  const uint64_t eh = even_bits(hi), sh = even_bits(hi >> 1);  // levels 1..32
  uint64_t E, S;
  if (depth <= 32) {
    E = depth > 0 ? eh >> (32 - depth) : 0ull;
    S = depth > 0 ? sh >> (32 - depth) : 0ull;
  } else {
    const uint64_t el = even_bits(lo), sl = even_bits(lo >> 1);  // levels 33..64
    E = (eh << (depth - 32)) | (el >> (64 - depth));
    S = (sh << (depth - 32)) | (sl >> (64 - depth));
  }
  const double ex = ldexp(2.0 * (double)E + 1.0, -depth) - 1.0;
  const double sy = ldexp(2.0 * (double)S + 1.0, -depth) - 1.0;
  cx = R.cx + R.h0 * ex;
  cy = R.cy - R.h0 * sy;
}

__device__ void put_far(const EM &a, uint32_t at, const GraphRoot &R,
                        uint32_t keyBucket, int depth, double h, float4 q,
                        double M, double SX, double SY, uint32_t s0,
                        uint32_t s1) {
  if (!a.cells || at >= a.maxNodes) return;
  const double im = (M > 1e-30 || M < -1e-30) ? 1.0 / M : 0.0;
  double comx = 0.0, comy = 0.0;
  if (M > 1e-9 || M < -1e-9) {
    comx = SX * im;
    comy = SY * im;
  }
  double gx, gy;
  cell_center(R, a.bHi[keyBucket], a.bLo[keyBucket], depth, gx, gy);
  const double ih = h > 0.0 ? 1.0 / h : 0.0;
  FarCell c;
  c.qa = (float)((q.x - q.z) * im);
  c.qb = (float)(2.0 * q.y * im);
  c.tr = (float)((q.x + q.z) * im);
  c.h = (float)h;
  c.ox = (float)((gx - comx) * ih);
  c.oy = (float)((gy - comy) * ih);
  c.s0 = s0;
  c.s1 = s1;
  a.cells[at] = c;
}

__device__ void put_cell(const EM &a, uint32_t at, double M, double SX,
                         double SY, double h, uint32_t next) {
  if (at >= a.maxNodes) {
    atomicOr(a.status, GVIZ_ST_TREE);
    return;
  }
  double cx = 0.0, cy = 0.0;
  if (M > 1e-9 || M < -1e-9) {
    cx = SX / M;
    cy = SY / M;
  }
  if (a.f64) {
    NodeD n;
    n.x = cx;
    n.y = cy;
    n.mass = M;
    n.size = h;
    n.next = (int32_t)next;
    n.info = -1;
    n.pad0 = n.pad1 = 0;
    reinterpret_cast<NodeD *>(a.nodes)[at] = n;
  } else {
    NodeF n;
    ds_split(cx, n.xh, n.xl);
    ds_split(cy, n.yh, n.yl);
    n.mass = (float)M;
    if (isinf(h)) {
      n.size = INFINITY;
    } else {
      double t = 2.0 * h / a.theta;
      n.size = (float)(t * t);
    }
    n.next = (int32_t)next;
    n.info = -1;
    reinterpret_cast<NodeF *>(a.nodes)[at] = n;
  }
}

// Point v's leaf record at preorder slot `at`, from its position, mass and
// radius.
__device__ void put_leaf_vals(const EM &a, uint32_t at, uint32_t v, double2 p, double m,
                              double r) {
  if (at >= a.maxNodes) {
    atomicOr(a.status, GVIZ_ST_TREE);
    return;
  }
  if (a.leafPre) a.leafPre[v] = at;
  put_count(a, at, 1u);  // every record has its point count: k_far_groups reads it first
  if (a.f64) {
    NodeD n;
    n.x = p.x;
    n.y = p.y;
    n.mass = m;
    n.size = r;
    n.next = (int32_t)(at + 1);
    n.info = (int32_t)v;
    n.pad0 = n.pad1 = 0;
    reinterpret_cast<NodeD *>(a.nodes)[at] = n;
  } else {
    NodeF n;
    ds_split(p.x, n.xh, n.xl);
    ds_split(p.y, n.yh, n.yl);
    n.mass = (float)m;
    n.size = (float)r;
    n.next = (int32_t)(at + 1);
    n.info = (int32_t)v;
    reinterpret_cast<NodeF *>(a.nodes)[at] = n;
  }
}

__device__ void put_leaf(const EM &a, uint32_t at, uint32_t v) {
  put_leaf_vals(a, at, v, a.pos[v], a.mass[v], a.radius[v]);
}

// Children of a cell for walks that expand several cells at once (a cell's
// first child is the next preorder slot, the others sit behind their elder
// siblings' subtrees): up to four preorder slots in quadrant order,
// GVIZ_NONE where a quadrant is empty; a cell whose children are a run of
// more than four points (a leaf bucket or a capacity leaf) stores
// {first slot, GVIZ_KIDS_RUN, count}.
__device__ __forceinline__ uint32_t link_weight(const EM &a, uint32_t c) {
  const uint2 u = (c & GVIZ_LEAF_BIT) ? a.upLeaf[c & ~GVIZ_LEAF_BIT] : a.upInt[c];
  return u.y & 0x7fffffffu;
}

__device__ void put_kids_run(const EM &a, uint32_t at, uint32_t c) {
  if (!a.kids || at >= a.maxNodes) return;
  a.kids[at] = c <= 4u ? make_uint4(at + 1u, c > 1u ? at + 2u : GVIZ_NONE,
                                    c > 2u ? at + 3u : GVIZ_NONE, c > 3u ? at + 4u : GVIZ_NONE)
                       : make_uint4(at + 1u, GVIZ_KIDS_RUN, c, 0u);
}

// A quadtree node p: its binary children, or their children where a child
// was absorbed into p's level (two path bits per quadtree level), each at p's
// slot plus the weights of the links down to it.
__device__ void put_kids_quad(const EM &a, uint32_t at, uint32_t p) {
  if (!a.kids || at >= a.maxNodes) return;
  uint32_t out[4] = {GVIZ_NONE, GVIZ_NONE, GVIZ_NONE, GVIZ_NONE};
  int n = 0;
  const uint32_t ch[2] = {a.nLeft[p], a.nRight[p]};
  for (int i = 0; i < 2; i++) {
    const uint32_t c = ch[i];
    const uint32_t wc = at + link_weight(a, c);
    if (!(c & GVIZ_LEAF_BIT) && (a.nFlag[c] & 1u)) {
      const uint32_t g0 = a.nLeft[c], g1 = a.nRight[c];
      if (n < 4) out[n++] = wc + link_weight(a, g0);
      if (n < 4) out[n++] = wc + link_weight(a, g1);
    } else if (n < 4) {
      out[n++] = wc;
    }
  }
  a.kids[at] = make_uint4(out[0], out[1], out[2], out[3]);
}

// depth of the nearest quadtree ancestor of a node whose binary parent is p
__device__ __forceinline__ int quad_parent_depth(const EM &a, uint32_t p) {
  if (p != GVIZ_NONE && (a.nFlag[p] & 1u)) p = a.upInt[p].x;
  return p == GVIZ_NONE ? -1 : ((a.nDelta[p] - 32) >> 1);
}

// The records of internal node p (a quadtree cell or a capacity leaf) at
// preorder position pre (without the graph base).
__device__ void emit_internal(const EM &a, uint32_t U, uint32_t p, uint32_t pre,
                              uint32_t fb, uint32_t g, double M, double SX, double SY,
                              uint32_t T) {
  const GraphRoot R = a.roots[g];
  if (a.nFlag[p] & 2u) {  // capacity leaf: wrapper + points in vertex order
    const uint32_t lb = a.nLast[p];
    const uint32_t s0 = a.bStart[fb];
    const uint32_t s1 = (lb + 1 < U) ? a.bStart[lb + 1] : a.V;
    put_cell(a, pre, M, SX, SY, INFINITY, pre + T);
    put_count(a, pre, s1 - s0);
    put_kids_run(a, pre, s1 - s0);
    uint32_t ids[GVIZ_MAX_NODES_PER_CELL];
    uint32_t c = s1 - s0;
    for (uint32_t j = 0; j < c; j++) {
      uint32_t v = a.idx[s0 + j];
      uint32_t q = j;
      while (q > 0 && ids[q - 1] > v) {
        ids[q] = ids[q - 1];
        q--;
      }
      ids[q] = v;
    }
    for (uint32_t j = 0; j < c; j++) put_leaf(a, pre + 1 + j, ids[j]);
    return;
  }
  const int q = (a.nDelta[p] - 32) >> 1;
  put_cell(a, pre, M, SX, SY, ldexp(R.h0, -q), pre + T);
  put_kids_quad(a, pre, p);
  if (a.cells) {
    const uint32_t lb = a.nLast[p];
    const uint32_t s0 = a.bStart[fb];
    const uint32_t s1 = (lb + 1 < U) ? a.bStart[lb + 1] : a.V;
    put_far(a, pre, R, fb, q, ldexp(R.h0, -q), a.nQ[p], M, SX, SY, s0, s1);
    put_count(a, pre, s1 - s0);
  }
}

// The records of bucket b (a point, or the points of one smallest cell
// behind a wrapper cell) at preorder position pre (without the graph base).
__device__ void emit_bucket(const EM &a, uint32_t U, uint32_t b, uint32_t pre, uint2 ub,
                            uint32_t g, uint32_t c, uint32_t s0) {
  const GraphRoot R = a.roots[g];
  const int qp = quad_parent_depth(a, ub.x);
  const bool testable = c > a.k && qp < R.D - 1;
  const double h = testable ? ldexp(R.h0, -(R.D - 1)) : (double)INFINITY;
  put_cell(a, pre, a.bM[b], a.bSX[b], a.bSY[b], h, pre + 1 + c);
  put_count(a, pre, c);
  put_kids_run(a, pre, c);
  if (a.cells && testable)
    put_far(a, pre, R, b, R.D - 1, h, a.bQ[b], a.bM[b], a.bSX[b], a.bSY[b], s0,
            s0 + c);
  for (uint32_t j = 0; j < c; j++) put_leaf(a, pre + 1 + j, a.idx[s0 + j]);
}

// A node's preorder position relative to its graph's base is the sum of the
// link weights up to the graph's root; k_top gives it for the nodes above
// blocks (kPreLocal: not one), so a walk up stops at the first of them.

// Shared by the threads of one k_emit block: parent links and k_top's entries
// of the internal nodes [C0, C0 + kEmitSpan).
constexpr uint32_t kEmitSpan = kThreads / 2;
struct EmitShared {
  uint2 up[kEmitSpan], pre[kEmitSpan];
};

// k_top's position of a node above blocks (t, its entry): below a node of
// level 2 it is relative to the last ancestor of level 1, t.y.
__device__ __forceinline__ uint32_t top_pre(const EM &a, uint2 t, bool &dead) {
  dead = t.x == GVIZ_NONE;
  if (t.y == GVIZ_NONE) return t.x;
  const uint2 u = a.upInt[t.y];
  const uint32_t above = a.pre[u.x].x;
  dead = dead || (u.y >> 31) || above == GVIZ_NONE;
  return t.x + u.y + above;
}

// Preorder position (without the graph base) of the node whose parent link
// is u. dead: an ancestor is a capacity leaf.
__device__ __forceinline__ uint32_t emit_pre(const EM &a, const EmitShared &s, uint32_t C0,
                                             uint2 u, bool &dead) {
  uint32_t pre = 0;
  dead = false;
  for (int guard = 0; u.x != GVIZ_NONE; guard++) {
    if (guard > GVIZ_MAX_CLIMB || (u.y >> 31)) {  // the guard is never expected
      dead = true;
      return 0;
    }
    pre += u.y;
    const uint32_t x = u.x;
    const bool cached = x - C0 < kEmitSpan;
    const uint2 t = cached ? s.pre[x - C0] : a.pre[x];
    if (t.x != kPreLocal) return pre + top_pre(a, t, dead);
    u = cached ? s.up[x - C0] : a.upInt[x];
  }
  return pre;
}

// Node and leaf records in preorder: block j emits internal nodes and
// buckets [C0, C0 + kEmitSpan), C0 = kEmitSpan j, one per thread. Bound by the
// latency of its gathers along the tree (15 of 17 cycles between a warp's
// instructions), so eight blocks share an SM at 32 registers, a few of them
// spilled: 1,048,576 vertices 100 -> 79 us (five blocks at 48 registers; six
// at 40: 91).
__global__ __launch_bounds__(kThreads, 8) void k_emit(EM a) {
  step_order();
  __shared__ EmitShared s;
  const uint32_t U = a.counts[2];
  const uint32_t nInt = U - 1;
  const uint32_t C0 = blockIdx.x * kEmitSpan;
  if (C0 >= U) return;
  const uint32_t i = threadIdx.x % kEmitSpan;
  const uint32_t t = C0 + i;
  if (threadIdx.x < kEmitSpan && t < nInt) {
    s.up[i] = a.upInt[t];
    s.pre[i] = a.pre[t];
  }
  __syncthreads();
  // each record's inputs are loaded before the walk up, whose end (the
  // preorder position) only the stores need
  if (threadIdx.x < kEmitSpan) {
    if (t < nInt && a.nDelta[t] >= 32 && !(a.nFlag[t] & 1u)) {
      const uint32_t fb = a.nFirst[t];
      const double M = a.nM[t], SX = a.nSX[t], SY = a.nSY[t];
      const uint32_t T = a.nT[t];
      const uint32_t g = a.bGid[fb];
      const uint32_t base = a.graphBase[g];
      bool dead;
      const uint32_t pre = s.pre[i].x == kPreLocal ? emit_pre(a, s, C0, s.up[i], dead)
                                                   : top_pre(a, s.pre[i], dead);
      if (!dead) emit_internal(a, U, t, pre + base, fb, g, M, SX, SY, T);
    }
  } else if (t < U) {
    const uint2 ub = a.upLeaf[t];
    const uint32_t g = a.bGid[t], c = a.bCnt[t], s0 = a.bStart[t];
    const uint32_t base = a.graphBase[g];
    const uint32_t v = a.idx[s0];  // the point of a single-point bucket
    double2 pv = make_double2(0.0, 0.0);
    double mv = 0.0, rv = 0.0;
    if (c == 1) {
      pv = a.pos[v];
      mv = a.mass[v];
      rv = a.radius[v];
    }
    bool dead;
    const uint32_t pre = emit_pre(a, s, C0, ub, dead);
    if (dead) return;
    if (c == 1)
      put_leaf_vals(a, pre + base, v, pv, mv, rv);
    else
      emit_bucket(a, U, t, pre + base, ub, g, c, s0);
  }
}

// Target groups of the learned cell-group walk: every cell of at most
// kGroupMax points whose parent holds more (or a root of at most kGroupMax
// points) is one group. Consecutive such children of one parent are packed
// into one group while the sum stays <= kGroupMax and the rectangle of
// their quadrants holds no other child of the parent (NW+NE, SW+SE, NW+SW
// with NE empty, ...), so a group's bounding box never covers points that
// are not its own; a group is a preorder range [x, y). A cell of more than
// four children is a leaf bucket (all its points in one smallest cell): its
// points are cut into runs of kGroupMax. Thread t < total handles the
// children of node t; thread maxNodes + g the root of graph g. The order of
// the groups in the list does not matter: a group's forces depend only on
// the group.
constexpr uint32_t kGroupMax = 32;

struct GroupArgs {
  const NodeF *nodes;
  const uint4 *kids;
  const FarCell *cells;
  const uint32_t *cellCnt, *counts, *graphBase, *rootT;
  uint4 *groups;
  uint32_t *nGroups;
  uint32_t maxNodes, G, cap;
};

__device__ __forceinline__ int4 node_link(const NodeF *nodes, uint32_t j) {
  return __ldg(reinterpret_cast<const int4 *>(nodes + j) + 1);  // mass, size, next, info
}

// quadrant (NW 0, NE 1, SW 2, SE 3) of the point set of node j inside a
// cell centred at (cx, cy), from its centre of mass
__device__ __forceinline__ uint32_t child_quadrant(const NodeF *nodes, uint32_t j, double cx,
                                                   double cy) {
  const NodeF n = nodes[j];
  const double x = (double)n.xh + (double)n.xl, y = (double)n.yh + (double)n.yl;
  return (x >= cx ? 1u : 0u) | (y < cy ? 2u : 0u);
}

// Each thread finds its groups (at most four packs of a branching cell, a
// root, or the runs of a leaf bucket); one atomic per warp reserves the
// warp's slots.
__global__ __launch_bounds__(kThreads) void k_far_groups(GroupArgs a) {
  step_order();
  const uint32_t t = blockIdx.x * kThreads + threadIdx.x;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t total = min(a.counts[3], a.maxNodes);
  uint32_t px[4], py[4], pc[4];
  uint32_t np = 0;                 // packs held in px/py/pc
  uint32_t runX = 0, runEnd = 0;   // a leaf bucket's runs [runX, runEnd)
  if (t >= a.maxNodes) {
    const uint32_t g = t - a.maxNodes;
    if (g < a.G) {
      const uint32_t r = a.graphBase[g], T = a.rootT[g];
      if (T != 0 && r < total) {
        const uint32_t c = a.cellCnt[r];
        if (c <= kGroupMax) {
          px[0] = r;
          py[0] = min(r + T, total);
          pc[0] = c;
          np = 1;
        }
      }
    }
  } else if (t < total && a.cellCnt[t] > kGroupMax) {  // (a point's count is 1)
    const int4 l = node_link(a.nodes, t);
    {
      const uint32_t end = min(max((uint32_t)l.z, t + 1u), total);
      uint32_t chX[4], chY[4], chC[4], chQ[4];
      int nc = 0;
      // the children from the cell's child record (independent loads): a
      // run of more than four points is a leaf bucket
      const uint4 kd = a.kids[t];
      const bool bucket = kd.y == GVIZ_KIDS_RUN;
      if (!bucket) {
        const uint32_t kk[4] = {kd.x, kd.y, kd.z, kd.w};
#pragma unroll
        for (int i = 0; i < 4; i++)
          if (kk[i] > t && kk[i] < end) chX[nc++] = kk[i];
        for (int i = 0; i < nc; i++) {
          chY[i] = i + 1 < nc ? chX[i + 1] : end;
          chC[i] = a.cellCnt[chX[i]];
        }
      }
      if (bucket) {  // points of one smallest cell: runs of kGroupMax leaves
        runX = t + 1u;
        runEnd = end;
      } else {
        const NodeF pn = a.nodes[t];
        const FarCell pcell = a.cells[t];
        const double cx = (double)pn.xh + (double)pn.xl + (double)pcell.ox * (double)pcell.h;
        const double cy = (double)pn.yh + (double)pn.yl + (double)pcell.oy * (double)pcell.h;
        for (int i = 0; i < nc; i++) chQ[i] = child_quadrant(a.nodes, chX[i], cx, cy);
        int first = -1;
        uint32_t pcnt = 0, r0 = 0, r1 = 0, c0 = 0, c1 = 0;  // pack, its quadrant rectangle
        for (int i = 0; i <= nc; i++) {
          if (i < nc && chC[i] <= kGroupMax && first >= 0 && pcnt + chC[i] <= kGroupMax) {
            const uint32_t R0 = min(r0, chQ[i] >> 1), R1 = max(r1, chQ[i] >> 1);
            const uint32_t C0 = min(c0, chQ[i] & 1u), C1 = max(c1, chQ[i] & 1u);
            bool fits = true;
            for (int k = 0; k < nc; k++) {
              if (k >= first && k <= i) continue;
              const uint32_t r = chQ[k] >> 1, c = chQ[k] & 1u;
              if (r >= R0 && r <= R1 && c >= C0 && c <= C1) fits = false;
            }
            if (fits) {
              r0 = R0, r1 = R1, c0 = C0, c1 = C1;
              pcnt += chC[i];
              continue;
            }
          }
          if (first >= 0) {
            px[np] = chX[first];
            py[np] = chY[i - 1];
            pc[np] = pcnt;
            np++;
          }
          first = -1;
          if (i < nc && chC[i] <= kGroupMax) {  // a larger child is cut by its own thread
            first = i;
            pcnt = chC[i];
            r0 = r1 = chQ[i] >> 1;
            c0 = c1 = chQ[i] & 1u;
          }
        }
      }
    }
  }
  const uint32_t nRuns = (runEnd - runX + kGroupMax - 1u) / kGroupMax;
  const uint32_t mine = np + nRuns;
  uint32_t incl = mine;  // inclusive warp scan of the group counts
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (uint32_t)o) incl += y;
  }
  const uint32_t warpTotal = __shfl_sync(0xffffffffu, incl, 31);
  uint32_t base = 0;
  if (lane == 0 && warpTotal) base = atomicAdd(a.nGroups, warpTotal);
  base = __shfl_sync(0xffffffffu, base, 0) + incl - mine;
  for (uint32_t k = 0; k < np; k++)
    if (base + k < a.cap) a.groups[base + k] = make_uint4(px[k], py[k], pc[k], 0u);
  for (uint32_t k = 0; k < nRuns; k++) {
    const uint32_t x = runX + k * kGroupMax, y = min(x + kGroupMax, runEnd);
    if (base + np + k < a.cap) a.groups[base + np + k] = make_uint4(x, y, y - x, 0u);
  }
}

// Inspection: per vertex, the index of its target group.
__global__ __launch_bounds__(kThreads) void k_group_members(const NodeF *nodes,
                                                            const uint4 *groups,
                                                            const uint32_t *nGroups,
                                                            uint32_t cap, uint32_t *groupOf) {
  const uint32_t gi = blockIdx.x * kThreads + threadIdx.x;
  if (gi >= min(*nGroups, cap)) return;
  const uint4 G = groups[gi];
  for (uint32_t j = G.x; j < G.y; j++) {
    const int4 l = node_link(nodes, j);
    if (l.w >= 0) groupOf[l.w] = gi;
  }
}

// Inspection: per point, the depth of the reference leaf holding it.
__global__ __launch_bounds__(kThreads) void k_leaf_depth(EM a, int32_t *depthOut) {
  const uint32_t U = a.counts[2];
  if (U == 0) return;  // no tree
  const uint32_t t = blockIdx.x * kThreads + threadIdx.x;
  const uint32_t nInt = U - 1;
  if (t < nInt) {
    const uint32_t p = t;
    if (a.nDelta[p] < 32 || !(a.nFlag[p] & 2u) || (a.nFlag[p] & 1u)) return;
    uint32_t pre, dead;
    walk_up(a.upInt[p], a.upInt, pre, dead);
    if (dead) return;
    const int d = quad_parent_depth(a, a.upInt[p].x) + 1;
    const uint32_t fb = a.nFirst[p], lb = a.nLast[p];
    const uint32_t s0 = a.bStart[fb];
    const uint32_t s1 = (lb + 1 < U) ? a.bStart[lb + 1] : a.V;
    for (uint32_t s = s0; s < s1; s++) depthOut[a.idx[s]] = d;
    return;
  }
  const uint32_t b = t - nInt;
  if (t < nInt || b >= U) return;
  uint32_t pre, dead;
  walk_up(a.upLeaf[b], a.upInt, pre, dead);
  if (dead) return;
  const uint32_t c = a.bCnt[b];
  const GraphRoot R = a.roots[a.bGid[b]];
  const int d = c > a.k ? R.D : quad_parent_depth(a, a.upLeaf[b].x) + 1;
  const uint32_t s0 = a.bStart[b];
  for (uint32_t j = 0; j < c; j++) depthOut[a.idx[s0 + j]] = d;
}

EM make_em(gvizCudaForce *h) {
  EM a;
  a.idx = h->d_idx;
  a.bStart = h->d_bStart;
  a.bGid = h->d_bGid;
  a.bCnt = h->d_bCnt;
  a.counts = h->d_counts;
  a.nFirst = h->d_nFirst;
  a.nLast = h->d_nLast;
  a.nFlag = h->d_nFlag;
  a.nT = h->d_nT;
  a.nCnt = h->d_nCnt;
  a.graphBase = h->d_graphBase;
  a.nDelta = h->d_nDelta;
  a.upInt = h->d_upInt;
  a.upLeaf = h->d_upLeaf;
  a.bM = h->d_bM;
  a.bSX = h->d_bSX;
  a.bSY = h->d_bSY;
  a.nM = h->d_nM;
  a.nSX = h->d_nSX;
  a.nSY = h->d_nSY;
  a.mass = h->d_mass;
  a.radius = h->d_radius;
  a.pos = h->d_pos;
  a.roots = h->d_roots;
  a.nodes = h->d_nodes;
  a.status = h->d_status;
  a.maxNodes = (uint32_t)h->maxNodes;
  a.theta = h->params.theta;
  a.V = (uint32_t)h->V;
  a.k = h->params.nodesPerCell;
  a.f64 = h->params.precision == GVIZ_CUDA_FP64;
  a.bQ = h->farSide ? h->d_bQ : nullptr;
  a.nQ = h->farSide ? h->d_nQ : nullptr;
  a.bHi = h->d_bHi;
  a.bLo = h->d_bLo;
  a.cells = h->farSide ? h->d_cells : nullptr;
  a.leafPre = h->farSide ? h->d_leafPre : nullptr;
  a.cellCnt = (h->farSide && h->params.farCellGroups) ? h->d_cellCnt : nullptr;
  a.nLeft = h->d_nLeft;
  a.nRight = h->d_nRight;
  a.kids = a.f64 ? nullptr : h->d_kids;  // the FP32 walks expand cells by them
  a.pre = h->d_pre;
  return a;
}

inline uint32_t blocks_for(size_t n) {
  return (uint32_t)((n + kThreads - 1) / kThreads);
}

}  // namespace

void enqueue_tree_build(gvizCudaForce *h) {
  const uint32_t V = (uint32_t)h->V;
  cudaStream_t st = h->stream;
  // status, counters, boxes, subtree sizes (a graph without vertices gets no
  // root: its size must read 0), the scan's and the sort's state
  cudaMemsetAsync(h->d_zero, 0, h->zeroBytes, st);
  k_bbox_chunks<<<h->nChunks, kThreads, 0, st>>>(h->d_pos, h->d_chunkBegin, h->d_chunkEnd,
                                                  h->d_chunkGraph, h->d_box, h->d_status);
  launch_after(st, k_keys, std::min(blocks_for(V), 148u * 8u), kThreads, 0, h->d_pos, h->d_gid,
               h->d_box, h->d_roots, h->d_ck, h->d_idx, sort_digit_counts(h), h->d_status, V,
               h->gbits);
  prof_mark(h, "tree_keys");
  radix_sort_pairs(h, h->d_ck, h->d_idx, h->d_ckAlt, h->d_idxAlt, V);
  launch_after(st, k_runs, blocks_for(V), kThreads, 0, h->d_ck, h->d_idx, h->d_pos, h->d_roots,
               h->d_counts, h->d_deepRuns, h->d_sHi, h->d_sLo, V, h->params.nodesPerCell,
               h->gbits);
  const size_t fixSmem = (size_t)GVIZ_FIX_MAX * 20;
  launch_after(st, k_sort_runs, 148, 512, fixSmem, h->d_sHi, h->d_sLo, h->d_idx, h->d_deepRuns,
               h->d_counts, h->d_status);
  launch_after(st, k_buckets, (V + GVIZ_SCAN_TILE - 1) / GVIZ_SCAN_TILE, kThreads, 0, h->d_sHi,
               h->d_sLo, h->d_ck, h->d_bStart, h->d_bHi, h->d_bLo, h->d_bGid, h->d_upLeaf,
               h->d_scanState, h->d_counts + 2, h->d_status, V, h->gbits);
  prof_mark(h, "tree_buckets");
  TopLists top;
  top.list1 = h->d_flag;  // V entries, free after the sort
  top.list2 = h->d_deepRuns;
  top.count1 = h->d_topCount;
  top.count2 = h->d_counts + 4;
  top.pre = h->d_pre;
  top.superBits = super_bits(V);
  launch_after(st, k_karras, blocks_for(V), kThreads, 0, h->d_bHi, h->d_bLo,
               h->G > 1 ? h->d_bGid : nullptr, h->d_counts, h->d_nLeft, h->d_nRight, h->d_nFirst,
               h->d_nLast, h->d_nDelta, h->d_upInt, h->d_upLeaf, top);
  BU bu;
  bu.idx = h->d_idx;
  bu.bStart = h->d_bStart;
  bu.bGid = h->d_bGid;
  bu.counts = h->d_counts;
  bu.nLeft = h->d_nLeft;
  bu.nRight = h->d_nRight;
  bu.nFirst = h->d_nFirst;
  bu.nLast = h->d_nLast;
  bu.nDelta = h->d_nDelta;
  bu.mass = h->d_mass;
  bu.pos = h->d_pos;
  bu.upInt = h->d_upInt;
  bu.upLeaf = h->d_upLeaf;
  bu.nCounter = h->d_nCounter;
  bu.bM = h->d_bM;
  bu.bSX = h->d_bSX;
  bu.bSY = h->d_bSY;
  bu.nM = h->d_nM;
  bu.nSX = h->d_nSX;
  bu.nSY = h->d_nSY;
  bu.bCnt = h->d_bCnt;
  bu.bT = h->d_bT;
  bu.nCnt = h->d_nCnt;
  bu.nT = h->d_nT;
  bu.nFlag = h->d_nFlag;
  bu.rootNode = h->d_rootNode;
  bu.rootT = h->d_rootT;
  bu.status = h->d_status;
  bu.V = V;
  bu.k = h->params.nodesPerCell;
  bu.bQ = h->farSide ? h->d_bQ : nullptr;
  bu.nQ = h->farSide ? h->d_nQ : nullptr;
  bu.top = top;
  bu.total = h->G == 1 ? h->d_counts + 3 : nullptr;
  if (bu.bQ) {
    launch_after(st, k_bottom_up<true>, blocks_for(V), kThreads, 0, bu);
    launch_top<true>(bu, V, st);
  } else {
    launch_after(st, k_bottom_up<false>, blocks_for(V), kThreads, 0, bu);
    launch_top<false>(bu, V, st);
  }
  // (a single graph starts at slot 0, and its root told the total)
  if (h->G > 1) scan_exclusive(h, h->d_rootT, h->d_graphBase, h->G, h->d_counts + 3);
  EM em = make_em(h);
  launch_after(st, k_emit, (uint32_t)((V + kEmitSpan - 1) / kEmitSpan), kThreads, 0, em);
  if (em.cellCnt && !em.f64) {
    GroupArgs ga;
    ga.nodes = reinterpret_cast<const NodeF *>(h->d_nodes);
    ga.kids = h->d_kids;
    ga.cells = h->d_cells;
    ga.cellCnt = h->d_cellCnt;
    ga.counts = h->d_counts;
    ga.graphBase = h->d_graphBase;
    ga.rootT = h->d_rootT;
    ga.groups = h->d_groups;
    ga.nGroups = h->d_groupCount;
    ga.maxNodes = (uint32_t)h->maxNodes;
    ga.G = (uint32_t)h->G;
    ga.cap = (uint32_t)(V ? V : 1);
    cudaMemsetAsync(h->d_groupCount, 0, sizeof(uint32_t), st);
    k_far_groups<<<blocks_for((size_t)h->maxNodes + h->G), kThreads, 0, st>>>(ga);
  }
  prof_mark(h, "tree_nodes");
}

void enqueue_tree_export(gvizCudaForce *h, int32_t *leafDepth) {
  EM em = make_em(h);
  k_leaf_depth<<<blocks_for(2 * h->V), kThreads, 0, h->stream>>>(em,
                                                                 leafDepth);
}

void enqueue_group_export(gvizCudaForce *h, uint32_t *groupOf) {
  const uint32_t cap = (uint32_t)(h->V ? h->V : 1);
  k_group_members<<<blocks_for(cap), kThreads, 0, h->stream>>>(
      reinterpret_cast<const NodeF *>(h->d_nodes), h->d_groups, h->d_groupCount, cap, groupOf);
}

void tree_set_smem_limits() {
  cudaFuncSetAttribute(k_sort_runs, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       GVIZ_FIX_MAX * 20);
  top_smem_limits<false, kTopCap>();
  top_smem_limits<true, kTopCap>();
  top_smem_limits<false, kTopCapLarge<false>>();
  top_smem_limits<true, kTopCapLarge<true>>();
}

// Inspection: every cell of the compressed tree (branching nodes and
// multi-point leaves) at its preorder slot, with the reference node it
// stands for: depth, quadrant path, mass, centre of mass, point count.
namespace {

__device__ __forceinline__ uint64_t dmask_hi(int d) {
  return d <= 0 ? 0ull : (d >= 32 ? ~0ull : (~0ull << (64 - 2 * d)));
}
__device__ __forceinline__ uint64_t dmask_lo(int d) {
  return d <= 32 ? 0ull : (d >= 64 ? ~0ull : (~0ull << (128 - 2 * d)));
}

struct CellOut {
  int32_t *depth;
  uint64_t *hi, *lo, *cnt;
  double *mass, *cx, *cy;
  const uint64_t *bHi, *bLo;
};

__device__ void cell_out(const CellOut &o, uint32_t at, int d, uint32_t b,
                         double M, double SX, double SY, uint64_t c) {
  o.depth[at] = d;
  o.hi[at] = o.bHi[b] & dmask_hi(d);
  o.lo[at] = o.bLo[b] & dmask_lo(d);
  o.mass[at] = M;
  const bool ok = M > 1e-9 || M < -1e-9;
  o.cx[at] = ok ? SX / M : 0.0;
  o.cy[at] = ok ? SY / M : 0.0;
  o.cnt[at] = c;
}

__global__ __launch_bounds__(kThreads) void k_cell_dump(EM a, CellOut o) {
  const uint32_t U = a.counts[2];
  if (U == 0) return;  // no tree
  const uint32_t t = blockIdx.x * kThreads + threadIdx.x;
  const uint32_t nInt = U - 1;
  if (t < nInt) {
    const uint32_t p = t;
    if (a.nDelta[p] < 32 || (a.nFlag[p] & 1u)) return;
    uint32_t pre, dead;
    walk_up(a.upInt[p], a.upInt, pre, dead);
    if (dead) return;
    const uint32_t fb = a.nFirst[p];
    pre += a.graphBase[a.bGid[fb]];
    const int d = (a.nFlag[p] & 2u) ? quad_parent_depth(a, a.upInt[p].x) + 1
                                    : ((a.nDelta[p] - 32) >> 1);
    cell_out(o, pre, d, fb, a.nM[p], a.nSX[p], a.nSY[p], a.nCnt[p]);
    return;
  }
  const uint32_t b = t - nInt;
  if (t < nInt || b >= U) return;
  const uint32_t c = a.bCnt[b];
  if (c < 2) return;
  uint32_t pre, dead;
  walk_up(a.upLeaf[b], a.upInt, pre, dead);
  if (dead) return;
  const GraphRoot R = a.roots[a.bGid[b]];
  pre += a.graphBase[a.bGid[b]];
  const int d = c > a.k ? R.D : quad_parent_depth(a, a.upLeaf[b].x) + 1;
  cell_out(o, pre, d, b, a.bM[b], a.bSX[b], a.bSY[b], c);
}

}  // namespace

void enqueue_cell_dump(gvizCudaForce *h, int32_t *depth, uint64_t *hi,
                       uint64_t *lo, double *mass, double *cx, double *cy,
                       uint64_t *cnt) {
  EM em = make_em(h);
  CellOut o;
  o.depth = depth;
  o.hi = hi;
  o.lo = lo;
  o.cnt = cnt;
  o.mass = mass;
  o.cx = cx;
  o.cy = cy;
  o.bHi = h->d_bHi;
  o.bLo = h->d_bLo;
  k_cell_dump<<<blocks_for(2 * h->V), kThreads, 0, h->stream>>>(em, o);
}
