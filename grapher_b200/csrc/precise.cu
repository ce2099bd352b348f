// precise.cu -- FP64 force kernels and the ForceAtlas2 speed / update
// kernels. This translation unit is compiled with --fmad=false so every
// a*b+c rounds twice, exactly like the reference's C (x86-64, no FMA):
// with the same inputs and the same order of terms the FP64 walk, the FP64
// exact kernel and the FA2 arithmetic reproduce the reference's rounding.
//
//  * k_attr_f64  : src/embedders/gvizForceEmbedder.c:93-100 in CSR order
//  * k_walk_f64  : bhAccumulateRepulsion (:35-74), a warp steps through the
//                  union of its targets' nodes, terms summed in the
//                  reference's DFS order
//  * k_exact_f64 : the BH-off loop (:104-115), j ascending, j != i
//  * k_fa2_*     : swing/traction sums, updateGlobalSpeed (:140-185),
//                  applySpeedRange (:187-197), step tail (:467-492)
#include <math.h>

#include <algorithm>

#include <cuda/atomic>

#include "epilogue.cuh"
#include "internal.cuh"

int dir_table_upload_precise(const double *t) {
  return cudaMemcpyToSymbol(c_dirTable, t, sizeof(double) * 2 * GVIZ_DIR_TABLE) ==
                 cudaSuccess ? 0 : -1;
}

EpiArgs make_epi(gvizCudaForce *h) {
  EpiArgs e;
  e.pos = h->d_pos;
  e.degree = h->d_degree;
  e.mass = h->d_mass;
  e.sf = h->forceOnly ? h->d_applied : h->d_sf;
  e.sfOld = h->d_sfOld;
  e.disp = h->d_disp;
  e.att = h->d_att;
  e.rep = h->d_rep;
  e.swing = h->d_swing;
  e.trac = h->d_trac;
  e.repVec = h->repVecOut;
  e.gravityK = h->params.gravityK;
  return e;
}

namespace {

constexpr int kThreads = 256;
constexpr int kWalkThreads = 128;
constexpr uint32_t kWalkList = 1024;  // listed nodes per warp of the walk
constexpr int kExactTile = 256;
constexpr uint32_t kInf = 0xffffffffu;

struct Attr64Args {
  const uint32_t *rowOff, *cols, *gid, *active, *list;
  const double2 *pos;
  double2 *out;
  double k;
  uint32_t n;  // entries of list
};

// one attraction term of the vertex at p towards q; false: no term
template <int MODEL>
__device__ __forceinline__ bool attr_term64(double2 p, double2 q, double k, double &tx,
                                            double &ty) {
  const double dx = q.x - p.x;
  const double dy = q.y - p.y;
  const double dist = sqrt(dx * dx + dy * dy);
  if (dist < 1e-9) return false;
  double s;
  if (MODEL == GVIZ_CUDA_MODEL_FR)
    s = dist / k;
  else
    s = log(1.0 + dist) / dist;
  tx = s * dx;
  ty = s * dy;
  return true;
}

// Vertices with at most GVIZ_HEAVY_DEGREE neighbours: one thread each.
template <int MODEL>
__global__ __launch_bounds__(kThreads) void k_attr_f64(Attr64Args a) {
  const uint32_t i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= a.n) return;
  const uint32_t v = a.list[i];
  if (a.active && !a.active[a.gid ? a.gid[v] : 0u]) return;
  const double2 p = a.pos[v];
  double ax = 0.0, ay = 0.0;
  const uint32_t e1 = a.rowOff[v + 1];
  for (uint32_t e = a.rowOff[v]; e < e1; e++) {
    double tx, ty;
    if (attr_term64<MODEL>(p, a.pos[a.cols[e]], a.k, tx, ty)) {
      ax += tx;
      ay += ty;
    }
  }
  a.out[v] = make_double2(ax, ay);
}

// The others: one warp each. The lanes compute 32 terms of the row side by
// side (the gather, square root, logarithm and division of a term take a
// thousand cycles one after the other) and lanes 0 and 1 add their x and y in
// row order, so the sums are the serial loop's bit for bit. The next terms'
// positions are on their way meanwhile. A row of 1,000 entries set the
// kernel's time: 281 us at 20,000 vertices (LinLog, highest degree ~800),
// now 36.
constexpr int kHeavyThreads = 128;

template <int MODEL>
__global__ __launch_bounds__(kHeavyThreads) void k_attr_f64_heavy(Attr64Args a) {
  __shared__ double term[kHeavyThreads / 32][2][32];
  const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t i = blockIdx.x * (kHeavyThreads / 32) + w;
  if (i >= a.n) return;  // the whole warp
  const uint32_t v = a.list[i];
  if (a.active && !a.active[a.gid ? a.gid[v] : 0u]) return;
  const double2 p = a.pos[v];
  const uint32_t e0 = a.rowOff[v], e1 = a.rowOff[v + 1];
  double sum = 0.0;  // lane 0: x, lane 1: y
  double2 q = p;
  if (e0 + lane < e1) q = a.pos[a.cols[e0 + lane]];
  for (uint32_t e = e0; e < e1; e += 32u) {
    double2 next = p;
    if (e + 32u + lane < e1) next = a.pos[a.cols[e + 32u + lane]];
    double tx = 0.0, ty = 0.0;
    const bool has = e + lane < e1 && attr_term64<MODEL>(p, q, a.k, tx, ty);
    const uint32_t mask = __ballot_sync(0xffffffffu, has);
    term[w][0][lane] = tx;
    term[w][1][lane] = ty;
    __syncwarp();
    if (lane < 2u) {
#pragma unroll 8
      for (int j = 0; j < 32; j++) {
        const double t = term[w][lane][j];
        if ((mask >> j) & 1u) sum += t;
      }
    }
    __syncwarp();
    q = next;
  }
  const double sy = __shfl_sync(0xffffffffu, sum, 1);
  if (lane == 0u) a.out[v] = make_double2(sum, sy);
}

// FR / LinLog repulsion term added to (ax, ay) with the reference's
// operation order (include/core/gvizVec.h:404-428, 552-578;
// src/embedders/gvizForceDirected.c:141-149 for FR's mass * force).
template <int MODEL>
__device__ __forceinline__ void rep_term64(double vx, double vy, double ux,
                                           double uy, double vMass,
                                           double oMass, double radiusSum,
                                           double kk, double C, uint32_t self,
                                           uint32_t other, double &ax,
                                           double &ay) {
  const double dx = ux - vx;
  const double dy = uy - vy;
  const double distSq = dx * dx + dy * dy;
  const double dist = sqrt(distSq);
  const double gap = dist - radiusSum;
  const double num = (MODEL == GVIZ_CUDA_MODEL_FR) ? kk : vMass * oMass;
  const double mag = gap > 0.0 ? num / gap : num * C;
  double dirx, diry;
  if (dist > 0.0) {
    dirx = dx / dist;
    diry = dy / dist;
  } else {
    coincident_dir(self, other, dirx, diry);
  }
  if (MODEL == GVIZ_CUDA_MODEL_FR) {
    const double sx = 0.0 - mag * dirx;
    const double sy = 0.0 - mag * diry;
    const double m = (double)(unsigned long long)oMass;
    ax += m * sx;
    ay += m * sy;
  } else {
    ax -= mag * dirx;
    ay -= mag * diry;
  }
}

struct Walk64Args {
  const NodeD *nodes;
  const uint32_t *idx, *gid, *active, *graphBase, *rootT;
  const double2 *pos;
  const double *mass, *radius;
  const double2 *attD;
  EpiArgs epi;
  double kk, overlapC, theta, theta2;
  uint32_t V, maxNodes;
  uint32_t targets;  // per warp
};

struct NodeRec {
  double2 n0, n1;
  int4 n2;
};

__device__ __forceinline__ NodeRec load_node(const Walk64Args &a, uint32_t i) {
  NodeRec r;
  r.n0 = __ldg(reinterpret_cast<const double2 *>(a.nodes + i));
  r.n1 = __ldg(reinterpret_cast<const double2 *>(a.nodes + i) + 1);
  r.n2 = __ldg(reinterpret_cast<const int4 *>(a.nodes + i) + 2);
  return r;
}

// Each warp walks `targets` path-sorted targets together, a lane for each.
// LISTS: a target's lane only lists the nodes whose terms it takes; when a
// list is full and at the end all lanes compute listed terms side by side, 32 /
// targets of them per target, added in list order by shuffles. Without, a
// target's own lane computes each term as the walk meets it, while the others
// wait: a term (a square root, three divisions) is longer than a step of the
// walk. The sums are the same to the bit.
template <int MODEL, bool LISTS>
__global__ __launch_bounds__(kWalkThreads) void k_walk_f64(Walk64Args a) {
  step_order();
  const unsigned lane = threadIdx.x & 31u;
  const uint32_t s = ((blockIdx.x * kWalkThreads + threadIdx.x) >> 5) * a.targets + lane;
  const bool valid = lane < a.targets && s < a.V;
  const uint32_t v = valid ? a.idx[s] : 0u;
  const uint32_t g = (valid && a.gid) ? a.gid[v] : 0u;
  const bool act = valid && (a.active == nullptr || a.active[g] != 0u);
  uint32_t resume = 0, myEnd = 0;
  double vx = 0.0, vy = 0.0, mv = 0.0, rv = 0.0;
  if (act) {
    resume = a.graphBase[g];
    myEnd = min(resume + a.rootT[g], a.maxNodes);
    const double2 p = a.pos[v];
    vx = p.x;
    vy = p.y;
    mv = a.mass[v];
    rv = a.radius[v];
  }
  // lane = target * helpers + helper while terms are computed
  const uint32_t helpers = LISTS ? 32u / a.targets : 1u, mine = lane / helpers;
  const double tx = __shfl_sync(0xffffffffu, vx, mine), ty = __shfl_sync(0xffffffffu, vy, mine);
  const double tm = __shfl_sync(0xffffffffu, mv, mine), tr = __shfl_sync(0xffffffffu, rv, mine);
  const uint32_t tv = __shfl_sync(0xffffffffu, v, mine);
  __shared__ uint32_t lists[kWalkThreads / 32][LISTS ? kWalkList : 1u];
  uint32_t *const warpList = lists[threadIdx.x >> 5];
  const uint32_t room = kWalkList / a.targets;
  uint32_t cnt = 0;  // listed for the lane's target
  double ax = 0.0, ay = 0.0;
  const auto take_lists = [&]() {
    __syncwarp();
    const uint32_t n = __shfl_sync(0xffffffffu, cnt, mine);
    const uint32_t most = __reduce_max_sync(0xffffffffu, cnt);
    const uint32_t *const list = warpList + mine * room;
    for (uint32_t k = 0; k < most; k += helpers) {
      const uint32_t e = k + lane % helpers;
      double fx = 0.0, fy = 0.0;
      if (e < n) {
        const NodeRec r = load_node(a, list[e]);
        const bool isLeaf = r.n2.y >= 0;
        rep_term64<MODEL>(tx, ty, r.n0.x, r.n0.y, tm, r.n1.x, isLeaf ? tr + r.n1.y : tr, a.kk,
                          a.overlapC, tv, isLeaf ? (uint32_t)r.n2.y : tv, fx, fy);
      }
      for (uint32_t j = 0; j < helpers; j++) {
        const double ux = __shfl_sync(0xffffffffu, fx, mine * helpers + j);
        const double uy = __shfl_sync(0xffffffffu, fy, mine * helpers + j);
        if (k + j < n) {
          ax += ux;
          ay += uy;
        }
      }
    }
    cnt = 0;
    __syncwarp();
  };
  uint32_t nxt = resume < myEnd ? resume : kInf;
  uint32_t cur = __reduce_min_sync(0xffffffffu, nxt);
  // The walk is a chain of node records. The one after `cur` is cur + 1 where
  // a lane opens it, else (every other lane waits at the end of a subtree
  // around it) the one behind its subtree: both are on their way while this
  // one is worked on.
  NodeRec n = cur != kInf ? load_node(a, cur) : NodeRec();
  while (cur != kInf) {
    const NodeRec in = load_node(a, min(cur + 1u, a.maxNodes - 1u));
    const uint32_t behind = max((uint32_t)n.n2.x, cur + 1u);
    const NodeRec out = load_node(a, min(behind, a.maxNodes - 1u));
    const double2 n0 = n.n0, n1 = n.n1;
    const int4 n2 = n.n2;
    const bool active = cur >= resume && cur < myEnd;
    const bool isLeaf = n2.y >= 0;
    const bool massOk = n1.x != 0.0;
    bool open = false, term = false;
    if (active && massOk) {
      if (isLeaf) {
        if (LISTS)
          term = (uint32_t)n2.y != v;
        else if ((uint32_t)n2.y != v)
          rep_term64<MODEL>(vx, vy, n0.x, n0.y, mv, n1.x, rv + n1.y, a.kk,
                            a.overlapC, v, (uint32_t)n2.y, ax, ay);
      } else {
        // the reference's test, 2h / dist < theta, settled by its squares
        // wherever those are further apart than any rounding of either
        const double dx = n0.x - vx;
        const double dy = n0.y - vy;
        const double d2 = dx * dx + dy * dy;
        const double lhs = 4.0 * n1.y * n1.y, rhs = a.theta2 * d2;
        bool accept = lhs < rhs * (1.0 - 1e-12);
        if (!accept && !(lhs > rhs * (1.0 + 1e-12))) accept = (2.0 * n1.y) / sqrt(d2) < a.theta;
        if (!accept)
          open = true;
        else if (LISTS)
          term = true;
        else
          rep_term64<MODEL>(vx, vy, n0.x, n0.y, mv, n1.x, rv, a.kk,
                            a.overlapC, v, v, ax, ay);
      }
    }
    if (LISTS) {
      if (term) warpList[lane * room + cnt++] = cur;
      if (__any_sync(0xffffffffu, cnt == room)) take_lists();
    }
    if (active) resume = open ? cur + 1u : behind;
    nxt = resume < myEnd ? resume : kInf;
    const uint32_t last = cur;
    cur = __reduce_min_sync(0xffffffffu, nxt);
    if (cur == last + 1u)
      n = in;
    else if (cur == behind)
      n = out;
    else if (cur != kInf)  // the next graph's tree
      n = load_node(a, cur);
  }
  if constexpr (LISTS) {
    take_lists();
    if (!__shfl_sync(0xffffffffu, act ? 1 : 0, mine) || lane % helpers != 0u) return;
    const double2 at = a.attD[tv];
    force_epilogue(a.epi, tv, at.x, at.y, ax, ay);
  } else {
    if (!act) return;
    const double2 at = a.attD[v];
    force_epilogue(a.epi, v, at.x, at.y, ax, ay);
  }
}

struct Exact64Args {
  const double2 *pos;
  const double *mass, *radius;
  const uint32_t *gid, *active, *targets;
  const uint64_t *graphOff;
  const double2 *attD;
  EpiArgs epi;
  double2 *judgeOut;  // k_judge_f64: the targets' repulsion vectors
  double kk, overlapC;
  uint32_t n;         // number of targets (V, or the list length)
};

template <int MODEL>
__global__ __launch_bounds__(kThreads) void k_exact_f64(Exact64Args a) {
  step_order();
  __shared__ double2 sp[kExactTile];
  __shared__ double2 smr[kExactTile];
  __shared__ uint32_t sRange[2];
  const uint32_t t = blockIdx.x * kThreads + threadIdx.x;
  const bool valid = t < a.n;
  const uint32_t v = valid ? t : 0u;
  const uint32_t g = (valid && a.gid) ? a.gid[v] : 0u;
  const bool act = valid && (a.active == nullptr || a.active[g] != 0u);
  uint32_t gb = 0, ge = 0;
  if (act) {
    gb = (uint32_t)a.graphOff[g];
    ge = (uint32_t)a.graphOff[g + 1];
  }
  if (threadIdx.x == 0) {
    sRange[0] = kInf;
    sRange[1] = 0;
  }
  __syncthreads();
  if (act) {
    atomicMin(&sRange[0], gb);
    atomicMax(&sRange[1], ge);
  }
  __syncthreads();
  const uint32_t lo = sRange[0], hi = sRange[1];
  double vx = 0.0, vy = 0.0, mv = 0.0, rv = 0.0;
  if (act) {
    const double2 p = a.pos[v];
    vx = p.x;
    vy = p.y;
    mv = a.mass[v];
    rv = a.radius[v];
  }
  double ax = 0.0, ay = 0.0;
  for (uint32_t t0 = lo; t0 < hi; t0 += kExactTile) {
    __syncthreads();
    const uint32_t j = t0 + threadIdx.x;
    if (threadIdx.x < kExactTile && j < hi) {
      sp[threadIdx.x] = a.pos[j];
      smr[threadIdx.x] = make_double2(a.mass[j], a.radius[j]);
    }
    __syncthreads();
    const uint32_t cnt = min((uint32_t)kExactTile, hi - t0);
    if (act) {
      for (uint32_t q = 0; q < cnt; q++) {
        const uint32_t jj = t0 + q;
        if (jj == v || jj < gb || jj >= ge) continue;
        const double2 u = sp[q];
        const double2 mr = smr[q];
        rep_term64<MODEL>(vx, vy, u.x, u.y, mv, mr.x, rv + mr.y, a.kk,
                          a.overlapC, v, jj, ax, ay);
      }
    }
  }
  if (!act) return;
  const double2 at = a.attD[v];
  force_epilogue(a.epi, v, at.x, at.y, ax, ay);
}

// Exact repulsion of listed targets, for error measurements. The sources of
// a block's graphs are split into gridDim.y ranges of whole tiles, so that a
// few thousand targets fill the GPU (4,096 targets are 32 blocks per range);
// every range's sums go to `partial` and k_judge_combine adds them in range
// order. FP64 issue bounds the loop. Without overlap prevention a term is
// num / d^2 along d: ten FP64 instructions on a straight-line path with a
// reciprocal of its own, chunks of 32 sources that meet the target, a
// coincident point or an extreme distance taken again with the division (or,
// beyond the range, the root and divisions of rep_term64); with overlap
// prevention it is the term of rep_term64. 4,096 targets among 131,072
// vertices: 48 ms in 16 blocks of one serial sum, 0.90 split over blocks with
// a division and three branches per term, 0.55 now (0.30 at the FP64 pipe's
// rate). 8 / 16 / 24 / 32 / 48 blocks per SM of the 8 that fit take 0.77 / 0.62
// / 0.58 / 0.55 / 0.51, the sum of the partials 10 / 14 / 20 / 25 / 36 us.
struct JudgeArgs {
  Exact64Args e;
  double2 *partial;  // [gridDim.y][n]
};

constexpr int kJudgeThreads = 128;
constexpr int kJudgeTile = 128;
constexpr uint32_t kJudgeChunk = 32;
constexpr int kJudgeBlocksPerSM = 8;
constexpr int kCombineThreads = 64;  // a chain of loads per target: over many SMs
// high words of the squared distances the straight-line terms take:
// [2^-900, 2^1022), where neither the reciprocal nor its product overflows
constexpr uint32_t kJudgeLow = (1023u - 900u) << 20, kJudgeSpan = (1022u + 900u) << 20;

// 1 / d for d in [2^-900, 2^1022): the hardware's approximation and one step
// of the third-order (Chebyshev) iteration r + r (e + e^2), e = 1 - d r, which
// leaves 2^-52: no branch, three FP64 instructions.
__device__ __forceinline__ double reciprocal64(double d) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  const double e = __fma_rn(-d, r, 1.0);
  return __fma_rn(r, __fma_rn(e, e, e), r);
}

template <int MODEL, bool OVERLAP>
__global__ __launch_bounds__(kJudgeThreads, kJudgeBlocksPerSM) void k_judge_f64(JudgeArgs ja) {
  const Exact64Args &a = ja.e;
  __shared__ double2 sp[kJudgeTile];
  __shared__ double sm[kJudgeTile], sr[kJudgeTile];
  __shared__ uint32_t sRange[2];
  const uint32_t t = blockIdx.x * kJudgeThreads + threadIdx.x;
  const bool act = t < a.n;
  const uint32_t v = act ? a.targets[t] : 0u;
  const uint32_t g = (act && a.gid) ? a.gid[v] : 0u;
  if (threadIdx.x == 0) {
    sRange[0] = kInf;
    sRange[1] = 0;
  }
  __syncthreads();
  uint32_t gb = 0, ge = 0;
  double2 p = make_double2(0.0, 0.0);
  double mv = 0.0, rv = 0.0;
  if (act) {
    gb = (uint32_t)a.graphOff[g];
    ge = (uint32_t)a.graphOff[g + 1];
    atomicMin(&sRange[0], gb);
    atomicMax(&sRange[1], ge);
    p = a.pos[v];
    mv = a.mass[v];
    rv = a.radius[v];
  }
  __syncthreads();
  const uint32_t lo = sRange[0], hi = sRange[1];
  const uint32_t nTile = hi > lo ? (hi - lo + kJudgeTile - 1) / kJudgeTile : 0u;
  const uint32_t per = (nTile + gridDim.y - 1) / gridDim.y;
  const uint32_t s0 = lo + min(blockIdx.y * per, nTile) * kJudgeTile;
  const uint32_t s1 = min(hi, lo + min((blockIdx.y + 1) * per, nTile) * kJudgeTile);
  double ax = 0.0, ay = 0.0;
  for (uint32_t t0 = s0; t0 < s1; t0 += kJudgeTile) {
    __syncthreads();
    const uint32_t j = t0 + threadIdx.x;
    if (j < hi) {
      sp[threadIdx.x] = a.pos[j];
      const double m = a.mass[j];
      // FR: the truncated mass times k^2 (src/embedders/gvizForceModel.c:20)
      sm[threadIdx.x] =
          !OVERLAP && MODEL == GVIZ_CUDA_MODEL_FR ? a.kk * (double)(unsigned long long)m : m;
      if (OVERLAP) sr[threadIdx.x] = a.radius[j];
    }
    __syncthreads();
    const uint32_t cnt = min((uint32_t)kJudgeTile, hi - t0);
    if (!act) continue;
    for (uint32_t c0 = 0; c0 < cnt; c0 += kJudgeChunk) {
      double bx = 0.0, by = 0.0;
      // a whole chunk of the target's graph, straight-line: taken again below
      // when it meets the target, a coincident point or an extreme distance
      const bool whole = !OVERLAP && c0 + kJudgeChunk <= cnt && t0 + c0 >= gb &&
                         t0 + c0 + kJudgeChunk <= ge;
      uint32_t odd = whole ? 0u : kJudgeSpan;
      if (whole) {
#pragma unroll 4
        for (uint32_t q = c0; q < c0 + kJudgeChunk; q++) {
          const double2 u = sp[q];
          const double dx = u.x - p.x, dy = u.y - p.y;
          const double d2 = __fma_rn(dx, dx, dy * dy);
          odd = max(odd, (uint32_t)__double2hiint(d2) - kJudgeLow);
          const double s = -sm[q] * reciprocal64(d2);
          bx = __fma_rn(s, dx, bx);
          by = __fma_rn(s, dy, by);
        }
      }
      if (odd >= kJudgeSpan) {
        bx = by = 0.0;
        const uint32_t c1 = min(c0 + kJudgeChunk, cnt);
#pragma unroll 1
        for (uint32_t q = c0; q < c1; q++) {
          const uint32_t jj = t0 + q;
          if (jj == v || jj < gb || jj >= ge) continue;
          const double2 u = sp[q];
          if (OVERLAP) {
            rep_term64<MODEL>(p.x, p.y, u.x, u.y, mv, sm[q], rv + sr[q], a.kk, a.overlapC, v, jj,
                              bx, by);
          } else {
            const double dx = u.x - p.x, dy = u.y - p.y;
            const double d2 = __fma_rn(dx, dx, dy * dy);
            if ((uint32_t)__double2hiint(d2) - kJudgeLow < kJudgeSpan) {
              const double s = -sm[q] / d2;
              bx = __fma_rn(s, dx, bx);
              by = __fma_rn(s, dy, by);
            } else {
              // coincident, or so close or far that the quotient by the square
              // leaves the range: the terms of rep_term64
              const double dist = sqrt(dx * dx + dy * dy);
              const double mag = dist > 0.0 ? sm[q] / dist : sm[q] * a.overlapC;
              double ux, uy;
              if (dist > 0.0) {
                ux = dx / dist;
                uy = dy / dist;
              } else {
                coincident_dir(v, jj, ux, uy);
              }
              bx -= mag * ux;
              by -= mag * uy;
            }
          }
        }
      }
      ax += bx;
      ay += by;
    }
  }
  if (!act) return;
  if (!OVERLAP && MODEL != GVIZ_CUDA_MODEL_FR) {
    ax *= mv;
    ay *= mv;
  }
  ja.partial[(size_t)blockIdx.y * a.n + t] = make_double2(ax, ay);
}

__global__ __launch_bounds__(kCombineThreads) void k_judge_combine(JudgeArgs ja, uint32_t splits) {
  const uint32_t t = blockIdx.x * kCombineThreads + threadIdx.x;
  if (t >= ja.e.n) return;
  double sx = 0.0, sy = 0.0;
#pragma unroll 16
  for (uint32_t s = 0; s < splits; s++) {
    const double2 q = ja.partial[(size_t)s * ja.e.n + t];
    sx += q.x;
    sy += q.y;
  }
  ja.e.judgeOut[t] = make_double2(sx, sy);
}

// ---------------------------------------------------------------------------
// ForceAtlas2 speed regulation and the position update
// ---------------------------------------------------------------------------

struct Fa2Args {
  const uint32_t *chunkBegin, *chunkEnd, *chunkGraph, *gChunkBegin,
      *gChunkEnd;
  const uint64_t *graphOff;
  const double *swing, *trac, *att, *rep, *meanDegPlusOne;
  const double2 *disp;
  double2 *pos, *applied;
  ChunkStat *chunkStat;
  uint32_t *chunksDone;  // per graph, zero between kernels
  double *speed, *eff, *stats, *lastStats;
  uint32_t *active, *anyActive;
  uint64_t *iter, *runLeft;
  const double *runEps;
  double jitterTolerance, gravityK;
  uint32_t G;
  int strict;
};

// Fixed-shape block sum: strided per-thread partials, xor-shuffle tree,
// warp partials added in warp order. Same inputs -> same bits.
__device__ __forceinline__ double block_sum(double v, double *sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31u) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kThreads / 32; w++) r += sh[w];
  __syncthreads();
  return r;
}

__device__ __forceinline__ double block_max(double v, double *sh) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31u) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kThreads / 32; w++) r = fmax(r, sh[w]);
  __syncthreads();
  return r;
}

// Whether this block is the last of its graph's chunks to get here: its
// chunk's sums are visible to that block, and the counter is zero again for
// the next kernel. For the whole block, after thread 0 wrote the sums.
__device__ __forceinline__ bool last_chunk(const Fa2Args &a, uint32_t g) {
  __shared__ uint32_t sLast;
  if (threadIdx.x == 0) {
    cuda::atomic_ref<uint32_t, cuda::thread_scope_device> done(a.chunksDone[g]);
    const uint32_t n = a.gChunkEnd[g] - a.gChunkBegin[g];
    sLast = done.fetch_add(1u, cuda::memory_order_acq_rel) == n - 1u;
    if (sLast) done.store(0u, cuda::memory_order_relaxed);
  }
  __syncthreads();
  return sLast != 0u;
}

// updateGlobalSpeed, src/embedders/gvizForceEmbedder.c:140-185, per graph:
// thread 0 applies the rule to the block's sums of the graph's chunks (or,
// strict, to the vertices in order).
__device__ void fa2_speed(const Fa2Args &a, uint32_t g, double *sh) {
  double totalSwing = 0.0, totalTraction = 0.0;
  if (a.strict) {
    if (threadIdx.x == 0)
      for (uint64_t v = a.graphOff[g]; v < a.graphOff[g + 1]; v++) {
        totalSwing += a.swing[v];
        totalTraction += a.trac[v];
      }
  } else {
    for (uint32_t c = a.gChunkBegin[g] + threadIdx.x; c < a.gChunkEnd[g]; c += kThreads) {
      totalSwing += __ldcg(&a.chunkStat[c].a);
      totalTraction += __ldcg(&a.chunkStat[c].b);
    }
    totalSwing = block_sum(totalSwing, sh);
    totalTraction = block_sum(totalTraction, sh);
  }
  if (threadIdx.x != 0) return;
  if (totalTraction < 1e-7) return;
  double speed = a.speed[g], eff = a.eff[g];
  const double n = (double)(a.graphOff[g + 1] - a.graphOff[g]);
  const double estimatedOptimalJT = 0.05 * sqrt(n);
  const double minJT = sqrt(estimatedOptimalJT);
  const double maxJT = 10.0;
  double jt = a.jitterTolerance *
              fmax(minJT, fmin(maxJT, estimatedOptimalJT * totalTraction / (n * n)));
  if (totalSwing / totalTraction > 2.0) {
    if (eff > 0.05) eff *= 0.5;
    jt = fmax(jt, a.jitterTolerance);
  }
  const double targetSpeed =
      totalSwing > 1e-7 ? jt * eff * totalTraction / totalSwing : speed;
  if (totalSwing > jt * totalTraction) {
    if (eff > 0.05) eff *= 0.7;
  } else if (speed < 1000.0) {
    eff *= 1.3;
  }
  if (eff < 0.05)
    eff = 0.05;
  else if (eff > 1.0)
    eff = 1.0;
  speed += fmin(targetSpeed - speed, 0.5 * speed);
  a.speed[g] = speed;
  a.eff[g] = eff;
}

// Swing and traction sums of every chunk; the last chunk of a graph to finish
// adds them up and applies the speed rule. A chunk's loads are all in flight
// at once (a serial chain of them is what a block would otherwise take its
// time with); every sum keeps its fixed order: strided per-thread partials,
// the block's tree, the chunks in order.
__global__ __launch_bounds__(kThreads) void k_fa2_speed(Fa2Args a) {
  step_order();
  __shared__ double sh[kThreads / 32];
  const uint32_t c = blockIdx.x;
  const uint32_t g = a.chunkGraph[c];
  if (!a.active[g]) return;
  constexpr int kItems = GVIZ_CHUNK / kThreads;
  const uint32_t v0 = a.chunkBegin[c] + threadIdx.x, v1 = a.chunkEnd[c];
  double swing[kItems], trac[kItems];
#pragma unroll
  for (int r = 0; r < kItems; r++) {
    const uint32_t v = v0 + r * kThreads;
    swing[r] = v < v1 ? a.swing[v] : 0.0;
    trac[r] = v < v1 ? a.trac[v] : 0.0;
  }
  double sw = 0.0, tr = 0.0;
#pragma unroll
  for (int r = 0; r < kItems; r++) {
    sw += swing[r];  // (adding zeros past the end changes nothing)
    tr += trac[r];
  }
  sw = block_sum(sw, sh);
  tr = block_sum(tr, sh);
  if (threadIdx.x == 0) {
    a.chunkStat[c].a = sw;
    a.chunkStat[c].b = tr;
  }
  if (last_chunk(a, g)) fa2_speed(a, g, sh);
}

// The step tail's statistics of graph g (:478-492) and its Run bookkeeping.
__device__ void fa2_stats(const Fa2Args &a, uint32_t g, double *sh) {
  double mx = 0.0, sAtt = 0.0, sRep = 0.0;
  if (a.strict) {
    if (threadIdx.x == 0)
      for (uint64_t v = a.graphOff[g]; v < a.graphOff[g + 1]; v++) {
        const double2 o = a.applied[v];
        const double nrm = sqrt(o.x * o.x + o.y * o.y);
        if (nrm > mx) mx = nrm;
        sAtt += a.att[v];
        sRep += a.rep[v];
      }
  } else {
    for (uint32_t c = a.gChunkBegin[g] + threadIdx.x; c < a.gChunkEnd[g]; c += kThreads) {
      mx = fmax(mx, __ldcg(&a.chunkStat[c].a));
      sAtt += __ldcg(&a.chunkStat[c].b);
      sRep += __ldcg(&a.chunkStat[c].c);
    }
    mx = block_max(mx, sh);
    sAtt = block_sum(sAtt, sh);
    sRep = block_sum(sRep, sh);
  }
  if (threadIdx.x != 0) return;
  const uint64_t n = a.graphOff[g + 1] - a.graphOff[g];
  const uint64_t it = a.iter[g];
  double *row = a.stats + ((it % GVIZ_STATS_CAP) * a.G + g) * 5;
  row[0] = mx;
  row[1] = a.speed[g];
  row[2] = n ? sAtt / (double)n : 0.0;
  row[3] = n ? sRep / (double)n : 0.0;
  row[4] = a.gravityK * a.meanDegPlusOne[g];
  for (int q = 0; q < 5; q++) a.lastStats[5 * g + q] = row[q];
  a.iter[g] = it + 1;
  const uint64_t left = a.runLeft[g] - 1;
  a.runLeft[g] = left;
  if (mx < a.runEps[g] || left == 0) {
    a.active[g] = 0;
    atomicSub(a.anyActive, 1u);
  }
}

// applySpeedRange (:187-197), position update and the statistics' chunk sums
// (:467-477); the last chunk of a graph to finish adds those up.
__global__ __launch_bounds__(kThreads) void k_fa2_apply(Fa2Args a) {
  step_order();
  __shared__ double sh[kThreads / 32];
  const uint32_t c = blockIdx.x;
  const uint32_t g = a.chunkGraph[c];
  if (!a.active[g]) return;
  const double speed = a.speed[g];
  const uint32_t v0 = a.chunkBegin[c] + threadIdx.x, v1 = a.chunkEnd[c];
  double mx = 0.0, sAtt = 0.0, sRep = 0.0;
  constexpr int kItems = 4;  // a thread's loads in flight at once
#pragma unroll
  for (int b = 0; b < GVIZ_CHUNK / kThreads; b += kItems) {
    double swing[kItems], att[kItems], rep[kItems];
    double2 f[kItems], p[kItems];
#pragma unroll
    for (int r = 0; r < kItems; r++) {
      const uint32_t v = v0 + (b + r) * kThreads;
      if (v < v1) {
        swing[r] = a.swing[v];
        f[r] = a.disp[v];
        att[r] = a.att[v];
        rep[r] = a.rep[v];
        p[r] = a.pos[v];
      }
    }
#pragma unroll
    for (int r = 0; r < kItems; r++) {
      const uint32_t v = v0 + (b + r) * kThreads;
      if (v < v1) {
        const double factor = speed / (1.0 + sqrt(speed * swing[r]));
        const double2 o = make_double2(f[r].x * factor, f[r].y * factor);
        a.applied[v] = o;
        const double nrm = sqrt(o.x * o.x + o.y * o.y);
        mx = fmax(mx, nrm);
        sAtt += att[r];
        sRep += rep[r];
        a.pos[v] = make_double2(p[r].x + o.x, p[r].y + o.y);
      }
    }
  }
  mx = block_max(mx, sh);
  sAtt = block_sum(sAtt, sh);
  sRep = block_sum(sRep, sh);
  if (threadIdx.x == 0) {
    a.chunkStat[c].a = mx;
    a.chunkStat[c].b = sAtt;
    a.chunkStat[c].c = sRep;
  }
  if (last_chunk(a, g) && !a.strict) fa2_stats(a, g, sh);
}

// Strict reductions: one block per graph, thread 0 sums the vertices in order.
__global__ __launch_bounds__(kThreads) void k_fa2_speed_strict(Fa2Args a) {
  step_order();
  __shared__ double sh[kThreads / 32];
  if (a.active[blockIdx.x]) fa2_speed(a, blockIdx.x, sh);
}
__global__ __launch_bounds__(kThreads) void k_fa2_stats_strict(Fa2Args a) {
  step_order();
  __shared__ double sh[kThreads / 32];
  if (a.active[blockIdx.x]) fa2_stats(a, blockIdx.x, sh);
}

// The step tail of the graphs without vertices, which have no chunk whose last
// block would do it: their rounds count and stop like any other's. Launched
// only where there are any.
__global__ __launch_bounds__(kThreads) void k_fa2_stats_empty(Fa2Args a, const uint32_t *graphs) {
  step_order();
  __shared__ double sh[kThreads / 32];
  const uint32_t g = graphs[blockIdx.x];
  if (a.active[g]) fa2_stats(a, g, sh);
}

inline uint32_t blocks(size_t n, int t) { return (uint32_t)((n + t - 1) / t); }

Fa2Args make_fa2(gvizCudaForce *h) {
  Fa2Args a;
  a.chunkBegin = h->d_chunkBegin;
  a.chunkEnd = h->d_chunkEnd;
  a.chunkGraph = h->d_chunkGraph;
  a.gChunkBegin = h->d_gChunkBegin;
  a.gChunkEnd = h->d_gChunkEnd;
  a.graphOff = h->d_graphOff;
  a.swing = h->d_swing;
  a.trac = h->d_trac;
  a.att = h->d_att;
  a.rep = h->d_rep;
  a.meanDegPlusOne = h->d_meanDegPlusOne;
  a.disp = h->d_disp;
  a.pos = h->d_pos;
  a.applied = h->d_applied;
  a.chunkStat = h->d_chunkStat;
  a.chunksDone = h->d_chunksDone;
  a.speed = h->d_speed;
  a.eff = h->d_eff;
  a.stats = h->d_stats;
  a.lastStats = h->d_lastStats;
  a.active = h->d_active;
  a.anyActive = h->d_anyActive;
  a.iter = h->d_iter;
  a.runLeft = h->d_runLeft;
  a.runEps = h->d_runEps;
  a.jitterTolerance = h->params.jitterTolerance;
  a.gravityK = h->params.gravityK;
  a.G = (uint32_t)h->G;
  a.strict = h->params.strictReductions;
  return a;
}

Exact64Args make_exact64(gvizCudaForce *h) {
  Exact64Args a;
  a.pos = h->d_pos;
  a.mass = h->d_mass;
  a.radius = h->d_radius;
  a.gid = h->d_gid;
  a.active = h->d_active;
  a.targets = nullptr;
  a.graphOff = h->d_graphOff;
  a.attD = h->d_attD;
  a.epi = make_epi(h);
  a.judgeOut = nullptr;
  a.kk = h->params.edgeLength * h->params.edgeLength;
  a.overlapC = h->params.overlapConstant;
  a.n = (uint32_t)h->V;
  return a;
}

}  // namespace

template <int MODEL>
static void launch_attraction_f64(gvizCudaForce *h, Attr64Args a) {
  const uint32_t *const lists[3] = {h->d_attrLight, h->d_attrHeavy, h->d_hubV};
  const uint32_t counts[3] = {h->nAttrLight, h->nAttrHeavy, h->nHubs};
  for (int l = 2; l >= 0; l--) {  // the longest rows first
    if (!counts[l]) continue;
    a.list = lists[l];
    a.n = counts[l];
    if (l == 0)
      k_attr_f64<MODEL><<<blocks(a.n, kThreads), kThreads, 0, h->stream>>>(a);
    else
      k_attr_f64_heavy<MODEL><<<blocks(a.n, kHeavyThreads / 32), kHeavyThreads, 0, h->stream>>>(a);
  }
}

void enqueue_attraction_f64(gvizCudaForce *h) {
  Attr64Args a;
  a.rowOff = h->d_rowOff;
  a.cols = h->d_cols;
  a.gid = h->d_gid;
  a.active = h->d_active;
  a.pos = h->d_pos;
  a.out = h->d_attD;
  a.k = h->params.edgeLength;
  if (h->model == GVIZ_CUDA_MODEL_FR)
    launch_attraction_f64<GVIZ_CUDA_MODEL_FR>(h, a);
  else
    launch_attraction_f64<GVIZ_CUDA_MODEL_LINLOG>(h, a);
  prof_mark(h, "attraction_f64");
}

// Targets per warp of the FP64 walk: 32 path-sorted targets share a walk, but
// below 148 SMs x 20 warps the walk's latency counts, not the work, and
// fewer targets per warp make more and shorter walks. A target's sum does not
// depend on it. Walk in us (LinLog BA, theta 0.8) with 2 / 4 / 8 / 16 / 32
// targets and lists: 700 vertices 41 / 48 / 57 / 74 / 113, 3,000 55 / 61 / 70 /
// 96 / 150, 9,000 118 / 83 / 88 / 115 / 178, 20,000 225 / 150 / 113 / 135 / 200,
// 40,000 436 / 287 / 205 / 168 / 228; without lists 65, 92, 118, 152 and 192 at
// its best of 4 to 32. With a warp full of targets there are no idle lanes to
// compute terms and the walk without lists is the faster: 80,000 258 against
// 272, 200,000 509 against 680.
static uint32_t walk64_targets(size_t V) {
  uint32_t t = 2;
  while (t < 32 && V > (size_t)t * 148 * 20) t *= 2;
  return t;
}

template <int MODEL>
static void launch_walk64(const Walk64Args &a, cudaStream_t st) {
  const uint32_t grid = blocks(((a.V + a.targets - 1) / a.targets) * (size_t)32, kWalkThreads);
  if (a.targets < 32) k_walk_f64<MODEL, true><<<grid, kWalkThreads, 0, st>>>(a);
  else k_walk_f64<MODEL, false><<<grid, kWalkThreads, 0, st>>>(a);
}

void enqueue_walk_f64(gvizCudaForce *h) {
  Walk64Args a;
  a.nodes = reinterpret_cast<const NodeD *>(h->d_nodes);
  a.idx = h->d_idx;
  a.gid = h->d_gid;
  a.active = h->d_active;
  a.graphBase = h->d_graphBase;
  a.rootT = h->d_rootT;
  a.pos = h->d_pos;
  a.mass = h->d_mass;
  a.radius = h->d_radius;
  a.attD = h->d_attD;
  a.epi = make_epi(h);
  a.kk = h->params.edgeLength * h->params.edgeLength;
  a.overlapC = h->params.overlapConstant;
  a.theta = h->params.theta;
  a.theta2 = a.theta * a.theta;
  a.targets = walk64_targets(h->V);
  a.V = (uint32_t)h->V;
  a.maxNodes = (uint32_t)h->maxNodes;
  if (h->model == GVIZ_CUDA_MODEL_FR) launch_walk64<GVIZ_CUDA_MODEL_FR>(a, h->stream);
  else launch_walk64<GVIZ_CUDA_MODEL_LINLOG>(a, h->stream);
  prof_mark(h, "bh_walk_f64");
}

void enqueue_exact_f64(gvizCudaForce *h) {
  Exact64Args a = make_exact64(h);
  if (h->model == GVIZ_CUDA_MODEL_FR)
    k_exact_f64<GVIZ_CUDA_MODEL_FR><<<blocks(h->V, kThreads), kThreads, 0, h->stream>>>(a);
  else
    k_exact_f64<GVIZ_CUDA_MODEL_LINLOG><<<blocks(h->V, kThreads), kThreads, 0, h->stream>>>(a);
  prof_mark(h, "exact_f64");
}

// Source ranges of the judge's kernel for n targets among V vertices: 32
// blocks per SM where the tiles allow.
uint32_t exact_judge_splits(size_t V, size_t n) {
  const size_t tb = (n + kJudgeThreads - 1) / kJudgeThreads;
  const size_t s = tb ? 148 * 32 / tb : 1;
  return (uint32_t)std::max<size_t>(1, std::min(s, (V + kJudgeTile - 1) / kJudgeTile));
}

// partial: exact_judge_splits(V, n) * n entries
void enqueue_exact_judge(gvizCudaForce *h, const uint32_t *d_targets, size_t n,
                         double2 *d_out, double2 *partial) {
  JudgeArgs ja;
  ja.e = make_exact64(h);
  ja.e.targets = d_targets;
  ja.e.judgeOut = d_out;
  ja.e.n = (uint32_t)n;
  ja.partial = partial;
  const uint32_t splits = exact_judge_splits(h->V, n);
  const dim3 grid(blocks(n, kJudgeThreads), splits);
  const bool ov = h->params.preventOverlap != 0;
  if (h->model == GVIZ_CUDA_MODEL_FR) {
    if (ov) k_judge_f64<GVIZ_CUDA_MODEL_FR, true><<<grid, kJudgeThreads, 0, h->stream>>>(ja);
    else k_judge_f64<GVIZ_CUDA_MODEL_FR, false><<<grid, kJudgeThreads, 0, h->stream>>>(ja);
  } else {
    if (ov) k_judge_f64<GVIZ_CUDA_MODEL_LINLOG, true><<<grid, kJudgeThreads, 0, h->stream>>>(ja);
    else k_judge_f64<GVIZ_CUDA_MODEL_LINLOG, false><<<grid, kJudgeThreads, 0, h->stream>>>(ja);
  }
  k_judge_combine<<<blocks(n, kCombineThreads), kCombineThreads, 0, h->stream>>>(ja, splits);
}

void enqueue_fa2(gvizCudaForce *h) {
  Fa2Args a = make_fa2(h);
  const uint32_t G = (uint32_t)h->G;
  if (a.strict) {
    launch_after(h->stream, k_fa2_speed_strict, G, kThreads, 0, a);
    launch_after(h->stream, k_fa2_apply, h->nChunks, kThreads, 0, a);
    launch_after(h->stream, k_fa2_stats_strict, G, kThreads, 0, a);
  } else {
    launch_after(h->stream, k_fa2_speed, h->nChunks, kThreads, 0, a);
    launch_after(h->stream, k_fa2_apply, h->nChunks, kThreads, 0, a);
    if (h->nEmptyGraphs)
      launch_after(h->stream, k_fa2_stats_empty, h->nEmptyGraphs, kThreads, 0, a,
                   h->d_emptyGraphs);
  }
  prof_mark(h, "fa2_update");
}
