// Visibility edges: for each vertex pair (i < j), trace the segment p_i -> p_j
// against the part itself and against its cage; the pair is an edge iff the
// segment leaves the cage and does not cross the part.
//
// Reference: lib/ptx/ray_segments.cu:49-125 (one OptiX ray per pair, origin
// p_i, tmin 0.001, tmax |p_j - p_i|, any-hit), lib/src/intersections.cpp:327-385
// (edge iff hits cage && !hits self; pairs whose endpoints are both old are
// skipped when is_new is given; edges in row-major (i, j) order).
//
// GB300 design:
//  * Vertices are Morton-sorted; a persistent warp takes an 8 x 4 tile of
//    (origin, target) positions from a global counter, so the 32 segments of a
//    warp start and end close together (coherent traversal, dynamic balance).
//  * Warp-packet any-hit traversal of a 64-byte-node LBVH (both child boxes per
//    node): the warp follows one path (ballot of per-lane box tests), node
//    records are broadcast loads, the stack lives in registers; the
//    cage test runs first and the self test only for lanes whose segment
//    leaves the cage (few: most vertex pairs of a part are interior chords,
//    which cross neither surface).
//  * Segment-triangle test: edge functions W = D.(B x C), ... relative to the
//    origin in FP32 with an a-priori rounding bound (8 roundings per term,
//    bounded by 17u |D|_1 L^2). Only tests whose signs fall inside the bound
//    are re-decided: in double-float, and in FP64 (the oracle's formula) where
//    that is open too. FP64 runs at about two operations per clock and SM, and
//    segments inside a cut plane put many tests inside the bound: the two
//    halves of a torus (4.5M pairs, 6.9M such tests) went from 6.45 to 4.32
//    ms, a cut blob (0.15M of them) from 2.43 to 2.24 ms.
//  * Box test: centre and half extents, three FMAs per axis and box, with the
//    leaf boxes' widening covering its rounding (traverse.cuh).
//  * Self-test end-vertex policy: triangles incident to i or j are skipped.
//  * Results land in a bitset over the reference's linear pair index; a
//    popcount / scan / emit pass compacts it into the row-major edge list.
#include <math.h>

#include "order.cuh"
#include "traverse.cuh"

namespace vgpu {

// Pairs from which a call (or a part of a batched call) builds and uses the
// cage's free-space grid: below this the grid costs about what the walk saves.
constexpr int64_t kFreeGridMinPairs = 1 << 22;

// Tiles a warp of the walk takes at a time (one at a time, its row and column
// found anew, took 1.14 ms against 0.56 for 1.64 M tiles: the counter's atomics; 4, 8, 16 and 32 at a time with
// the table below 0.70, 0.67, 0.70 and 0.79), and its resident CTAs per SM
// (8, 10, 12 and 16: 0.68, 0.67, 0.70 and 0.71).
constexpr int kWalkRun = 8, kWalkBlocks = 10;

// Warps a tile is split over at most (tile_split): with 1, 2, 4, 8 and 16 the
// traversal of a 162-vertex blob takes 69, 61, 56, 51 and 53 us, of a 128-vertex
// torus 126, 112, 84, 69 and 67; from some 600 vertices on there are no free warps.
constexpr int kMaxSplit = 8;

// Cells per side of the cube's faces in a reach table (reach_side): more of them
// clear more pairs (10,242 points, all pairs: 33.0 of 52.4 M with 4, 46.1 with 8,
// 50.3 with 16) but take longer to fill; table and walk 0.69 ms with 6, 0.70 with
// 8, 0.76 with 10, and 1.75 without a table and one tile at a time.
constexpr int kReachSide = 6;

// Pairs up to which a call emits and sends its edges without waiting for
// their number (128 KB of room; the wait it saves is about 15 us).
constexpr int64_t kFewPairs = 1 << 14;

struct VisParams {
  const float* pts;
  int32_t n;
  const uint32_t* rows;    // sorted positions -> original ids (rows of the tile space)
  const uint32_t* cols;    // same for columns
  int32_t nr, nc;
  int triangular;          // 1: rows == cols and pairs with row < col
  const uint8_t* is_new;   // masked mode
  const int32_t* newrank;  // masked mode: position of a new vertex in rows, else INT_MAX
  TileMesh mesh;           // the cage and the part
  uint32_t* bitset;
  VisCounters* cnt;
  unsigned* status;
  unsigned long long total_tiles;
  int64_t ntc;                          // tile columns
  int64_t ntr;                          // tile rows
  const unsigned long long* row_start;  // triangular mode: first tile of each tile row
  FreeGridView cage_free;               // the cage's free-space grid (lb null: none)
  FreeReach cage_reach;                 // and the points' reaches in it (reach null: none)
  // After a walk: the tiles with lanes left for the traversal, and per such
  // tile the lanes that are done (no pair, degenerate, or cleared).
  unsigned long long* pend_tiles;       // null: no walk, every tile is traversed
  uint32_t* pend_done;
};

// Work item w -> tile (tr, tc). Rectangle mode: row-major. Triangular mode:
// tile row tr holds tile columns [floor(TR tr / TC), ntc); row_start is the
// exclusive prefix of those counts (binary search).
__device__ __forceinline__ void tile_of(const VisParams& P, unsigned long long w, int64_t& tr,
                                        int64_t& tc, int TR, int TC) {
  if (!P.triangular) {
    if ((w >> 32) == 0 && P.ntc <= 0xffffffffLL) {  // 64-bit division is a long routine
      const uint32_t q = (uint32_t)w / (uint32_t)P.ntc;
      tr = q;
      tc = (uint32_t)w - q * (uint32_t)P.ntc;
      return;
    }
    tr = (int64_t)(w / (unsigned long long)P.ntc);
    tc = (int64_t)(w % (unsigned long long)P.ntc);
    return;
  }
  if (TR >= TC) {
    // r = TR / TC is an integer and row t holds ntc - r t tiles (never
    // negative: r (ntr - 1) <= ntc), so row t starts at
    // S(t) = t ntc - r t (t - 1) / 2. S(t) = w at
    // t = (B - sqrt(B^2 - 8 r w)) / 2r with B = 2 ntc + r, all but the root in
    // integers; the root in FP32 (off by less than a row for n <= 2^24) and its
    // rounding settled exactly. In FP64, whose units are few, this bound the
    // whole walk: 1.5 ms for 1.64 M tiles with hardly a grid read left.
    const int64_t r = TR / TC, ntc = P.ntc, B = 2 * ntc + r;
    auto S = [&](int64_t t) { return t * ntc - r * t * (t - 1) / 2; };
    const int64_t D = B * B - 8 * r * (int64_t)w;
    int64_t t = (B - (int64_t)sqrtf(D > 0 ? (float)D : 0.f)) / (2 * r);
    t = t < 0 ? 0 : (t > P.ntr - 1 ? P.ntr - 1 : t);
    while (t > 0 && (unsigned long long)S(t) > w) --t;
    while (t < P.ntr - 1 && (unsigned long long)S(t + 1) <= w) ++t;
    tr = t;
    tc = t * r + (int64_t)(w - (unsigned long long)S(t));
    return;
  }
  int64_t lo = 0, hi = P.ntr - 1;
  while (lo < hi) {
    int64_t mid = (lo + hi + 1) >> 1;
    if (P.row_start[mid] <= w) lo = mid; else hi = mid - 1;
  }
  tr = lo;
  tc = (tr * TR) / TC + (int64_t)(w - P.row_start[tr]);
}

__global__ void tile_row_counts_kernel(int64_t ntr, int64_t ntc, int TR, int TC,
                                       uint32_t* __restrict__ counts) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < ntr;
       r += (int64_t)gridDim.x * blockDim.x) {
    int64_t c = ntc - (r * TR) / TC;
    counts[r] = (uint32_t)(c > 0 ? c : 0);
  }
}

// The pair of `lane` in tile w of P's tile space (original vertex ids i < j),
// or valid = false.
template <int TR>
__device__ __forceinline__ bool lane_pair(const VisParams& P, unsigned long long w, int lane, uint32_t& i,
                                          uint32_t& j) {
  constexpr int TC = 32 / TR;
  int64_t tr, tc;
  tile_of(P, w, tr, tc, TR, TC);
  const int64_t a = tr * TR + lane / TC;
  const int64_t b = tc * TC + lane % TC;
  bool valid;
  uint32_t oi = 0, oj = 0;
  if (P.triangular) {
    valid = a < b && b < P.nc;
    if (valid) {
      oi = P.rows[a];
      oj = P.cols[b];
    }
  } else {
    valid = a < P.nr && b < P.nc;
    if (valid) {
      oi = P.rows[a];
      oj = P.cols[b];
      valid = oi != oj && (!P.is_new[oj] || P.newrank[oj] > a);
    }
  }
  i = min(oi, oj);
  j = max(oi, oj);
  return valid;
}

// What a walk kernel counts per lane.
struct WalkSums {
  unsigned pairs, deg, cleared;
  unsigned long long steps;
};

// Walks `count` tiles of P's tile space from tile w on. Lane l's pair of a tile
// is lane_pair's; the row's point stays in registers along a tile row, and the
// next tile is the next of the row or the first of the next row. Tiles with
// lanes left are listed as base + their number, a run's together with one atomic
// (18 M pairs in an open soup, nearly all left: 0.20 ms, 0.44 with one a tile). Their
// done lanes wait in `run` (kWalkRun words of the warp's in shared memory): in a
// register more visibility_multi_walk_kernel spills in its loop (1.82 ms for a bowl's
// parts, 1.50 so). Few tiles are left where the walk pays, so a tile's done lanes are
// stored only then (a store and a warp barrier for each: 52 M pairs 0.50 ms, 0.48 so).
template <int TR>
__device__ __forceinline__ void walk_tiles(const VisParams& P, unsigned long long w, int count,
                                           unsigned long long base, int lane, WalkSums& sum,
                                           uint32_t* __restrict__ run, unsigned long long* __restrict__ pending,
                                           unsigned long long* __restrict__ pend_tiles,
                                           uint32_t* __restrict__ pend_done) {
  constexpr int TC = 32 / TR;
  int64_t tr64, tc64;
  tile_of(P, w, tr64, tc64, TR, TC);
  static_assert(kWalkRun <= 32, "a lane per tile of a run");
  int tr = (int)tr64, tc = (int)tc64, row = -1;
  uint32_t oi = 0;
  unsigned left = 0;  // the tiles with lanes left
  float px = 0.f, py = 0.f, pz = 0.f;
  for (int k = 0; k < count; ++k) {
    const int a = tr * TR + lane / TC, b = tc * TC + lane % TC;
    if (tr != row) {
      row = tr;
      if (a < P.nr) {
        oi = P.rows[a];
        px = P.pts[3 * (int64_t)oi];
        py = P.pts[3 * (int64_t)oi + 1];
        pz = P.pts[3 * (int64_t)oi + 2];
      }
    }
    bool valid = P.triangular ? a < b && b < P.nc : a < P.nr && b < P.nc;
    uint32_t oj = 0;
    if (valid) {
      oj = P.cols[b];
      if (!P.triangular) valid = oi != oj && (!P.is_new[oj] || P.newrank[oj] > a);
    }
    bool done = true;
    if (valid) {
      ++sum.pairs;
      const float dx = __fsub_rn(P.pts[3 * (int64_t)oj], px), dy = __fsub_rn(P.pts[3 * (int64_t)oj + 1], py),
                  dz = __fsub_rn(P.pts[3 * (int64_t)oj + 2], pz);
      // The square of seg_length, which is positive when its root is.
      const float sq = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
      if (!(sq > 0.f)) {  // coincident endpoints (or NaN): never an edge (as in vis_tile)
        ++sum.deg;
      } else {
        float t0 = 0.f, s0 = 1.f;
        if (P.cage_reach.reach != nullptr) {
          const bool pos = P.cage_reach.by_pos != 0;
          cone_start(P.cage_reach, pos ? (uint32_t)a : oi, pos ? (uint32_t)b : oj, dx, dy, dz, t0, s0);
        }
        done = t0 >= s0 || (P.cage_free.lb != nullptr &&
                            trace_free(P.cage_free, px, py, pz, dx, dy, dz, __fsqrt_rn(sq), t0, s0, sum.steps));
        sum.cleared += done;
      }
    }
    const unsigned m = __ballot_sync(0xffffffffu, done);
    if (m != 0xffffffffu) {
      left |= 1u << k;
      if (lane == 0) run[k] = m;
    }
    if (++tc >= P.ntc) {
      ++tr;
      tc = P.triangular ? tr * TR / TC : 0;
    }
  }
  if (left) {
    unsigned long long at = 0;
    if (lane == 0) at = atomicAdd(pending, (unsigned long long)__popc(left));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(left & ((1u << lane) - 1u));
    __syncwarp();
    if (left >> lane & 1u) {
      pend_tiles[at] = base + w + lane;
      pend_done[at] = run[lane];
    }
    __syncwarp();
  }
}

__device__ __forceinline__ void walk_flush(VisCounters* __restrict__ cnt, int lane, const WalkSums& sum) {
  unsigned long long pairs = sum.pairs, deg = sum.deg, cleared = sum.cleared, steps = sum.steps;
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
    deg += __shfl_xor_sync(0xffffffffu, deg, o);
    cleared += __shfl_xor_sync(0xffffffffu, cleared, o);
    steps += __shfl_xor_sync(0xffffffffu, steps, o);
  }
  if (lane == 0) {
    if (pairs) atomicAdd(&cnt->pairs, pairs);
    if (deg) atomicAdd(&cnt->degenerate, deg);
    if (cleared) atomicAdd(&cnt->certified, cleared);
    if (steps) atomicAdd(&cnt->trace_steps, steps);
  }
}

// The reach table: entry k is point k % n (rows) in cell k / n, so a warp's
// walks start at neighbouring points in one direction and stay together.
__global__ void __launch_bounds__(256) visibility_reach_kernel(VisParams P, float* __restrict__ reach) {
  const FreeReach T = P.cage_reach;
  const int64_t count = (int64_t)T.n * 6 * T.m * T.m;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < count;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int row = (int)(k % T.n);
    const int64_t v = T.by_pos ? (int64_t)P.rows[row] : row;
    reach[k] = cell_reach(P.cage_free, P.pts[3 * v], P.pts[3 * v + 1], P.pts[3 * v + 2], T.m, (int)(k / T.n));
  }
}


// One tile (work item w of P's tile space) for the calling warp: the cage
// test, then the self test for lanes whose segment leaves the cage, and the
// edge bits. After a free-space walk (walked) the walk has taken the tile's
// pair and degenerate counts, and `done` marks the lanes it settled: they
// take no part.
template <int TR>
__device__ __forceinline__ void vis_tile(const VisParams& P, unsigned long long w, int lane, SegLeaf* leaf,
                                         unsigned long long* sum, unsigned& status_bits, bool walked,
                                         uint32_t done) {
  uint32_t i, j;
  const bool mine = !((done >> lane) & 1u);
  const bool valid = lane_pair<TR>(P, w, lane, i, j) && mine;
  float3 p = make_float3(0.f, 0.f, 0.f), q = make_float3(0.f, 0.f, 0.f);
  bool active = false;
  if (valid) {
    p = make_float3(P.pts[3 * (int64_t)i], P.pts[3 * (int64_t)i + 1], P.pts[3 * (int64_t)i + 2]);
    q = make_float3(P.pts[3 * (int64_t)j], P.pts[3 * (int64_t)j + 1], P.pts[3 * (int64_t)j + 2]);
    // coincident endpoints (or NaN): never an edge
    active = seg_length(__fsub_rn(q.x, p.x), __fsub_rn(q.y, p.y), __fsub_rn(q.z, p.z)) > 0.f;
  }
  const unsigned nv = __popc(__ballot_sync(0xffffffffu, valid)), na = __popc(__ballot_sync(0xffffffffu, active));
  if (lane == 0) {
    if (!walked) sum[kSumPairs] += nv;
    sum[kSumDegenerate] += nv - na;
  }
  if (!na) return;
  if (trace_tile(P.mesh, P.pts, i, j, p, q, active, leaf, sum, status_bits) == 1u) {
    const int64_t k = row_start(i, P.n) + (int64_t)(j - i - 1);
    atomicOr(&P.bitset[k >> 5], 1u << (k & 31));
  }
}

__device__ __forceinline__ void vis_flush_counters(VisCounters* cnt, unsigned* status, int lane,
                                                   const unsigned long long* sum, unsigned status_bits) {
  status_bits = __reduce_or_sync(0xffffffffu, status_bits);
  if (lane == 0) {
    unsigned long long* const to[kSums] = {&cnt->pairs,      &cnt->edges,    &cnt->self_hits,   &cnt->cage_hits,
                                           &cnt->degenerate, &cnt->rechecks, &cnt->node_visits, &cnt->tri_tests};
#pragma unroll
    for (int k = 0; k < kSums; ++k)
      if (sum[k]) atomicAdd(to[k], sum[k]);
    if (status_bits) atomicOr(status, status_bits);
  }
}

// Warps a tile is split over: as many (up to 8, four lanes each) as leave all of
// them resident. A warp runs its lanes' node and leaf tests one after another, so
// with few tiles the call is one such chain; each warp then takes 32 / split
// neighbouring pairs of the tile.
__device__ __forceinline__ int tile_split(unsigned long long tiles) {
  const unsigned long long warps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
  int split = 1;
  while (split < kMaxSplit && tiles * (2 * split) <= warps) split *= 2;
  return split;
}
// The lanes that are not part k's of a tile split in `split`.
__device__ __forceinline__ uint32_t split_others(int split, int k) {
  const int lanes = 32 / split;
  return split == 1 ? 0u : ~(((1u << lanes) - 1u) << (k * lanes));
}

template <int TR, int MINB>
__global__ void __launch_bounds__(kVisThreads, MINB) visibility_kernel(VisParams P) {
  const int lane = threadIdx.x & 31;
  __shared__ unsigned long long sums[kVisThreads / 32][kSums];
  __shared__ SegLeaf leaves[kVisThreads / 32];
  unsigned long long* sum = sums[threadIdx.x >> 5];
  SegLeaf* leaf = &leaves[threadIdx.x >> 5];
  if (lane < kSums) sum[lane] = 0;
  __syncwarp();
  unsigned status_bits = 0;
  // After a walk only the tiles it left are traversed (their count is on the
  // device, written by the walk kernel before this launch).
  const unsigned long long items = P.pend_tiles ? P.cnt->pending : P.total_tiles;
  const int split = tile_split(items);
  for (int guard = 0; guard < (1 << 30); ++guard) {
    unsigned long long w = 0;
    if (lane == 0) w = atomicAdd(&P.cnt->work, 1ull);
    w = __shfl_sync(0xffffffffu, w, 0);
    if (w >= items * split) break;
    uint32_t done = split_others(split, (int)(w % split));
    w /= split;
    if (P.pend_tiles) {
      done |= P.pend_done[w];
      w = P.pend_tiles[w];
    }
    // (one call: of two copies of the traversal one spilled in its loop, 10 %)
    vis_tile<TR>(P, w, lane, leaf, sum, status_bits, P.pend_tiles != nullptr, done);
  }
  vis_flush_counters(P.cnt, P.status, lane, sum, status_bits);
}

// The free-space walk over P's tile space, before the traversal kernel. It
// takes the pair and degenerate counts of every tile, and lists the tiles
// that keep a lane for the traversal (P.pend_tiles) with the lanes that are
// done (no pair, degenerate, or cleared: the segment cannot hit the cage;
// traverse.cuh, trace_free). Few registers, so many warps per SM hide the
// latency of the walk's dependent grid reads.
template <int TR>
__global__ void __launch_bounds__(kVisThreads, kWalkBlocks) visibility_walk_kernel(VisParams P) {
  const int lane = threadIdx.x & 31;
  __shared__ uint32_t runs[kVisThreads / 32][kWalkRun];
  uint32_t* run = runs[threadIdx.x >> 5];
  WalkSums sum = {};
  for (int guard = 0; guard < (1 << 30); ++guard) {
    unsigned long long w = 0;
    if (lane == 0) w = atomicAdd(&P.cnt->walk_work, (unsigned long long)kWalkRun);
    w = __shfl_sync(0xffffffffu, w, 0);
    if (w >= P.total_tiles) break;
    const int count = (int)min((unsigned long long)kWalkRun, P.total_tiles - w);
    walk_tiles<TR>(P, w, count, 0ull, lane, sum, run, &P.cnt->pending, P.pend_tiles, P.pend_done);
  }
  walk_flush(P.cnt, lane, sum);
}

// Many parts in one persistent launch: the work items of all parts are
// numbered consecutively (part p owns [tile_start[p], tile_start[p + 1])),
// and each warp finds the part of its item by binary search. Every part keeps
// its own tile space, mask and bitset region; the counters are shared.
__device__ __forceinline__ int part_of(const unsigned long long* __restrict__ tile_start, int n_parts,
                                       unsigned long long w) {
  int lo = 0, hi = n_parts - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tile_start[mid] <= w) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// With pend_tiles (after visibility_multi_walk_kernel) only the listed tiles
// are traversed, with the lanes the walk settled left out.
template <int TR, int MINB>
__global__ void __launch_bounds__(kVisThreads, MINB)
    visibility_multi_kernel(const VisParams* __restrict__ parts, int n_parts,
                            const unsigned long long* __restrict__ tile_start,
                            unsigned long long total_tiles, VisCounters* __restrict__ cnt,
                            unsigned* __restrict__ status, const unsigned long long* __restrict__ pend_tiles,
                            const uint32_t* __restrict__ pend_done) {
  const int lane = threadIdx.x & 31;
  __shared__ unsigned long long sums[kVisThreads / 32][kSums];
  __shared__ SegLeaf leaves[kVisThreads / 32];
  unsigned long long* sum = sums[threadIdx.x >> 5];
  SegLeaf* leaf = &leaves[threadIdx.x >> 5];
  if (lane < kSums) sum[lane] = 0;
  __syncwarp();
  unsigned status_bits = 0;
  const unsigned long long items = pend_tiles ? cnt->pending : total_tiles;
  const int split = tile_split(items);
  for (int guard = 0; guard < (1 << 30); ++guard) {
    unsigned long long w = 0;
    if (lane == 0) w = atomicAdd(&cnt->work, 1ull);
    w = __shfl_sync(0xffffffffu, w, 0);
    if (w >= items * split) break;
    uint32_t done = split_others(split, (int)(w % split));
    w /= split;
    if (pend_tiles) {
      done |= pend_done[w];
      w = pend_tiles[w];
    }
    const int p = part_of(tile_start, n_parts, w);
    vis_tile<TR>(parts[p], w - tile_start[p], lane, leaf, sum, status_bits, pend_tiles != nullptr, done);
  }
  vis_flush_counters(cnt, status, lane, sum, status_bits);
}

// The free-space walk over all parts' tiles (as visibility_walk_kernel; parts
// without a grid leave every pair to the traversal). Pending tiles are listed
// by their global number.
template <int TR>
__global__ void __launch_bounds__(kVisThreads, kWalkBlocks)
    visibility_multi_walk_kernel(const VisParams* __restrict__ parts, int n_parts,
                                 const unsigned long long* __restrict__ tile_start,
                                 unsigned long long total_tiles, VisCounters* __restrict__ cnt,
                                 unsigned long long* __restrict__ pend_tiles, uint32_t* __restrict__ pend_done) {
  const int lane = threadIdx.x & 31;
  __shared__ uint32_t runs[kVisThreads / 32][kWalkRun];
  uint32_t* run = runs[threadIdx.x >> 5];
  WalkSums sum = {};
  for (int guard = 0; guard < (1 << 30); ++guard) {
    unsigned long long w = 0;
    if (lane == 0) w = atomicAdd(&cnt->walk_work, (unsigned long long)kWalkRun);
    w = __shfl_sync(0xffffffffu, w, 0);
    if (w >= total_tiles) break;
    const unsigned long long end = min(w + kWalkRun, total_tiles);
    for (int pi = part_of(tile_start, n_parts, w); w < end; ++pi) {  // the run's parts
      const unsigned long long part_end = min(end, tile_start[pi + 1]);
      if (part_end <= w) continue;
      walk_tiles<TR>(parts[pi], w - tile_start[pi], (int)(part_end - w), tile_start[pi], lane, sum, run,
                     &cnt->pending, pend_tiles, pend_done);
      w = part_end;
    }
  }
  walk_flush(cnt, lane, sum);
}

// ---- vertex ordering ------------------------------------------------------
__global__ void point_bounds_kernel(const float* __restrict__ pts, int32_t n,
                                    VisCounters* __restrict__ c) {
  float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      float x = pts[3 * i + a];
      if (fabsf(x) < INFINITY) {
        lo[a] = fminf(lo[a], x);
        hi[a] = fmaxf(hi[a], x);
      }
    }
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
      hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
    }
  }
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      if (lo[a] <= hi[a]) {
        atomicMin(&c->pmin[a], f2o_v(lo[a]));
        atomicMax(&c->pmax[a], f2o_v(hi[a]));
      }
    }
  }
}

__device__ __forceinline__ uint64_t spread21_v(uint64_t x) {
  x &= 0x1fffffull;
  x = (x | (x << 32)) & 0x1f00000000ffffull;
  x = (x | (x << 16)) & 0x1f0000ff0000ffull;
  x = (x | (x << 8)) & 0x100f00f00f00f00full;
  x = (x | (x << 4)) & 0x10c30c30c30c30c3ull;
  x = (x | (x << 2)) & 0x1249249249249249ull;
  return x;
}

__global__ void point_morton_kernel(const float* __restrict__ pts, int32_t n,
                                    const VisCounters* __restrict__ c, int bits, uint64_t* __restrict__ keys,
                                    uint32_t* __restrict__ vals) {
  float lo[3], sc[3];
  const float top = (float)((1u << bits) - 1u);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    lo[a] = o2f_v(c->pmin[a]);
    float ext = o2f_v(c->pmax[a]) - lo[a];
    sc[a] = ext > 0.f ? top / ext : 0.f;
  }
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    uint64_t q[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      float x = (pts[3 * i + a] - lo[a]) * sc[a];
      x = fminf(fmaxf(x, 0.f), top);
      q[a] = (uint64_t)x;
    }
    keys[i] = (spread21_v(q[0]) << 2) | (spread21_v(q[1]) << 1) | spread21_v(q[2]);
    vals[i] = (uint32_t)i;
  }
}

__global__ void new_flags_kernel(const uint32_t* __restrict__ perm, const uint8_t* __restrict__ is_new,
                                 int32_t n, uint32_t* __restrict__ flags) {
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < n;
       s += (int64_t)gridDim.x * blockDim.x)
    flags[s] = is_new[perm[s]] ? 1u : 0u;
}

__global__ void new_rows_kernel(const uint32_t* __restrict__ perm, const uint32_t* __restrict__ flags,
                                const uint64_t* __restrict__ off, int32_t n,
                                uint32_t* __restrict__ rows, int32_t* __restrict__ newrank) {
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < n;
       s += (int64_t)gridDim.x * blockDim.x) {
    uint32_t v = perm[s];
    if (flags[s]) {
      rows[off[s]] = v;
      newrank[v] = (int32_t)off[s];
    } else {
      newrank[v] = 0x7fffffff;
    }
  }
}

// New points of a mask in device memory, added to *count. What a masked call does
// follows from it (the pairs, so the grid, the reach table and the tiles).
__global__ void mask_count_kernel(const uint8_t* __restrict__ is_new, int32_t n,
                                  unsigned long long* __restrict__ count) {
  unsigned c = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    c += is_new[i] != 0;
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, (unsigned long long)c);
}

// ---- bitset compaction ----------------------------------------------------
__global__ void bit_emit_kernel(const uint32_t* __restrict__ bits, int64_t nw,
                                const uint64_t* __restrict__ off, int64_t n,
                                uint32_t* __restrict__ edges) {
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < nw;
       w += (int64_t)gridDim.x * blockDim.x) {
    uint32_t m = bits[w];
    if (!m) continue;
    uint64_t o = off[w];
    const int64_t k0 = w * 32;
    // Row of k0: largest i with row_start(i) <= k0.
    double b2 = (double)(2 * n - 1);
    double disc = b2 * b2 - 8.0 * (double)k0;
    int64_t i = (int64_t)((b2 - sqrt(disc > 0 ? disc : 0.0)) * 0.5);
    if (i < 0) i = 0;
    if (i > n - 2) i = n - 2;
    while (i > 0 && row_start(i, n) > k0) --i;
    while (i + 1 <= n - 2 && row_start(i + 1, n) <= k0) ++i;
    while (m) {
      int bpos = __ffs(m) - 1;
      m &= m - 1;
      int64_t k = k0 + bpos;
      while (i + 1 <= n - 2 && row_start(i + 1, n) <= k) ++i;
      int64_t j = k - row_start(i, n) + i + 1;
      edges[2 * o] = (uint32_t)i;
      edges[2 * o + 1] = (uint32_t)j;
      ++o;
    }
  }
}

// Launch shapes the autotuner chooses from: tile rows (tile = TR x 32/TR pairs
// per warp) and the minimum resident CTAs per SM (register budget).
struct VisVariant {
  int tr;
  int minb;
};
static const VisVariant kVisVariants[] = {{8, 6}, {8, 8}, {4, 6}, {16, 6}, {2, 6}, {1, 6}, {32, 6}};
constexpr int kNumVisVariants = sizeof(kVisVariants) / sizeof(kVisVariants[0]);
// Untuned calls: 8 x 4 tiles at 8 resident CTAs per SM, the autotuner's pick
// on the s5 blob and the fastest on clipped parts (masked) by 3-6 %.
constexpr int kDefaultVisVariant = 1;

static int launch_vis_variant(visacd_ctx* ctx, int v, const VisParams& P) {
  const unsigned grid = (unsigned)(ctx->sm_count * kVisVariants[v].minb);
  if (P.pend_tiles != nullptr) {
    const unsigned wg = (unsigned)(ctx->sm_count * kWalkBlocks);
    switch (kVisVariants[v].tr) {
      case 8: VLAUNCH(ctx, kKVisWalk, wg, kVisThreads, 0, visibility_walk_kernel<8>, P); break;
      case 4: VLAUNCH(ctx, kKVisWalk, wg, kVisThreads, 0, visibility_walk_kernel<4>, P); break;
      case 16: VLAUNCH(ctx, kKVisWalk, wg, kVisThreads, 0, visibility_walk_kernel<16>, P); break;
      case 2: VLAUNCH(ctx, kKVisWalk, wg, kVisThreads, 0, visibility_walk_kernel<2>, P); break;
      case 1: VLAUNCH(ctx, kKVisWalk, wg, kVisThreads, 0, visibility_walk_kernel<1>, P); break;
      default: VLAUNCH(ctx, kKVisWalk, wg, kVisThreads, 0, visibility_walk_kernel<32>, P); break;
    }
  }
  switch (v) {
    case 0: VLAUNCH(ctx, kKVisibility, grid, kVisThreads, 0, (visibility_kernel<8, 6>), P); break;
    case 1: VLAUNCH(ctx, kKVisibility, grid, kVisThreads, 0, (visibility_kernel<8, 8>), P); break;
    case 2: VLAUNCH(ctx, kKVisibility, grid, kVisThreads, 0, (visibility_kernel<4, 6>), P); break;
    case 3: VLAUNCH(ctx, kKVisibility, grid, kVisThreads, 0, (visibility_kernel<16, 6>), P); break;
    case 4: VLAUNCH(ctx, kKVisibility, grid, kVisThreads, 0, (visibility_kernel<2, 6>), P); break;
    case 5: VLAUNCH(ctx, kKVisibility, grid, kVisThreads, 0, (visibility_kernel<1, 6>), P); break;
    default: VLAUNCH(ctx, kKVisibility, grid, kVisThreads, 0, (visibility_kernel<32, 6>), P); break;
  }
  return VISACD_OK;
}

// Shape class of a visibility call: log2 buckets of n and triangle counts, and
// the masked flag. The autotuner caches its pick per class in the context.
static uint32_t vis_shape_class(int32_t n, bool masked, const visacd_bvh* a, const visacd_bvh* b) {
  auto lg = [](int64_t x) { int r = 0; while (x > 1) { x >>= 1; ++r; } return r; };
  return (uint32_t)lg(n) | ((uint32_t)lg(a->nt + 1) << 6) | ((uint32_t)lg(b->nt + 1) << 12) |
         ((uint32_t)masked << 18);
}

static int choose_vis_variant(visacd_ctx* ctx, int32_t n, bool masked, const visacd_bvh* a,
                              const visacd_bvh* b) {
  if (ctx->vis_variant_override >= 0 && ctx->vis_variant_override < kNumVisVariants)
    return ctx->vis_variant_override;
  auto it = ctx->vis_tuned.find(vis_shape_class(n, masked, a, b));
  if (it != ctx->vis_tuned.end()) return it->second;
  return kDefaultVisVariant;
}

// Morton orders of points above kOrderMax: the general sort. perm: sorted
// position -> vertex.
static int points_order_large(visacd_ctx* ctx, const float* d_pts, int32_t n, VisCounters* cnt, uint32_t* perm) {
  VTRY(ensure_slot(ctx, kSlotVisKeys, (size_t)n * 8));
  VTRY(ensure_slot(ctx, kSlotVisKeysAlt, (size_t)n * 8));
  VTRY(ensure_slot(ctx, kSlotVisPermAlt, (size_t)n * 4));
  uint64_t* keys = slot<uint64_t>(ctx, kSlotVisKeys);
  const unsigned gp = grid_for(n, 256, 4LL * ctx->sm_count);
  // The ordered bounds start at (max, 0); the rest of the counters is zero.
  VCUDA(cudaMemsetAsync(cnt->pmin, 0xff, sizeof(cnt->pmin), ctx->stream));
  VCUDA(cudaMemsetAsync(cnt->pmax, 0, sizeof(cnt->pmax), ctx->stream));
  VLAUNCH(ctx, kKVisPrep, gp, 256, 0, point_bounds_kernel, d_pts, n, cnt);
  VLAUNCH(ctx, kKVisPrep, gp, 256, 0, point_morton_kernel, d_pts, n, cnt, morton_bits(n), keys, perm);
  return radix_sort_u64(ctx, keys, perm, slot<uint64_t>(ctx, kSlotVisKeysAlt),
                        slot<uint32_t>(ctx, kSlotVisPermAlt), n, 3 * morton_bits(n));
}

// The Morton orders of several point sets (the parts of a call), and for the
// masked ones their new points in order and every point's rank among them
// (rows and rank sized n each). Sets up to kOrderMax share one launch; its
// scratch is `scratch` (points_scratch bytes).
struct PointOrder {
  const float* pts;
  int32_t n;
  uint32_t* perm;
  const uint8_t* is_new;  // null: no mask
  uint32_t* rows;
  int32_t* rank;
};
static size_t points_scratch(const PointOrder* o, int count) {
  size_t b = 256;
  for (int k = 0; k < count; ++k)
    if (o[k].n > 1 && o[k].n <= kOrderMax) b += order_scratch(o[k].n, false);
  return b;
}
static OrderJob points_job(const PointOrder& q, char* scratch) {
  OrderJob j = {};
  j.verts = q.pts;
  j.nv = j.n = q.n;
  j.bits = morton_bits(q.n);
  order_carve(j, scratch);
  j.v0 = q.perm;
  j.is_new = q.is_new;
  j.rows = q.rows;
  j.rank = q.rank;
  return j;
}
static int points_order(visacd_ctx* ctx, const PointOrder* o, int count, char* scratch, VisCounters* cnt) {
  std::vector<OrderJob> jobs;
  for (int k = 0; k < count; ++k) {
    const PointOrder& q = o[k];
    if (q.n < 2) continue;
    if (q.n <= kOrderMax) {
      jobs.push_back(points_job(q, scratch));
      scratch += order_scratch(q.n, false);
      continue;
    }
    VTRY(points_order_large(ctx, q.pts, q.n, cnt, q.perm));
    if (q.is_new) {
      const unsigned gp = grid_for(q.n, 256, 4LL * ctx->sm_count);
      VTRY(ensure_slot(ctx, kSlotWordCounts, (size_t)q.n * 4));
      VTRY(ensure_slot(ctx, kSlotWordOffsets, (size_t)(q.n + 1) * 8));
      uint32_t* flags = slot<uint32_t>(ctx, kSlotWordCounts);
      uint64_t* off = slot<uint64_t>(ctx, kSlotWordOffsets);
      VLAUNCH(ctx, kKVisPrep, gp, 256, 0, new_flags_kernel, q.perm, q.is_new, q.n, flags);
      VTRY(exclusive_scan_u32_to_u64(ctx, flags, off, q.n));
      VLAUNCH(ctx, kKVisPrep, gp, 256, 0, new_rows_kernel, q.perm, flags, off, q.n, q.rows, q.rank);
    }
  }
  return jobs.empty() ? VISACD_OK : order_run(ctx, jobs.data(), (int)jobs.size());
}

// Where a single-part call keeps its orders.
static int order_slots(visacd_ctx* ctx, const float* d_pts, int32_t n, const uint8_t* d_new, PointOrder& o) {
  VTRY(ensure_slot(ctx, kSlotVisPerm, (size_t)n * 4));
  o = {d_pts, n, slot<uint32_t>(ctx, kSlotVisPerm), d_new, nullptr, nullptr};
  if (d_new) {
    VTRY(ensure_slot(ctx, kSlotVisRank, (size_t)n * 4 + (size_t)n * 4 + 256));
    o.rows = slot<uint32_t>(ctx, kSlotVisRank);
    o.rank = reinterpret_cast<int32_t*>(o.rows + ((n + 63) & ~63));
  }
  return VISACD_OK;
}

// Morton order of n device points into perm; synchronizes.
int vis_morton_order(visacd_ctx* ctx, const float* d_pts, int32_t n, uint32_t* perm) {
  if (n <= 0) return VISACD_OK;
  const PointOrder o = {d_pts, n, perm, nullptr, nullptr, nullptr};
  VTRY(ensure_slot(ctx, kSlotCounters, sizeof(VisCounters)));
  VTRY(ensure_slot(ctx, kSlotVisOrder, points_scratch(&o, 1)));
  if (n == 1) {
    VCUDA(cudaMemsetAsync(perm, 0, 4, ctx->stream));
  } else {
    VTRY(points_order(ctx, &o, 1, slot<char>(ctx, kSlotVisOrder), slot<VisCounters>(ctx, kSlotCounters)));
  }
  VCUDA(stream_wait(ctx));
  return VISACD_OK;
}

// Cells per side of a reach table for n points and a number of pairs: kReachSide,
// or fewer where the table would have more than a third as many entries as
// there are pairs (an entry costs about as many reads as a pair's walk without
// it), or more than 2^28 (1 GiB); below 3 none.
static int reach_side(int64_t n, int64_t pairs) {
  const double cells = std::min((double)pairs / 3.0, 268435456.0) / std::max((double)n, 1.0) / 6.0;
  const int m = (int)std::min((double)kReachSide, std::sqrt(cells));
  return m < 3 ? 0 : m;
}
static size_t reach_entries(int64_t n, int m) { return (size_t)n * 6 * m * m; }

static int launch_reach(visacd_ctx* ctx, const VisParams& P) {
  VLAUNCH(ctx, kKVisReach, grid_for((int64_t)reach_entries(P.cage_reach.n, P.cage_reach.m), 256, 16LL * ctx->sm_count),
          256, 0, visibility_reach_kernel, P, const_cast<float*>(P.cage_reach.reach));
  return VISACD_OK;
}

static int vis_device(visacd_ctx* ctx, const float* d_pts, int32_t n, const uint8_t* d_new,
                      const visacd_bvh* self_bvh, const visacd_bvh* cage_bvh, int64_t* n_edges,
                      visacd_vis_stats* stats, int64_t pairs, int32_t n_new, const PointOrder* ordered,
                      const uint32_t** few_edges) {
  // The cage's free-space grid, for calls with many pairs (`pairs`: the
  // call's pair count): built once per cage BVH, before this call's counters take
  // the shared scratch and staging buffers.
  const bool use_grid = ctx->vis_trace && n >= 2 && pairs >= kFreeGridMinPairs && cage_bvh->nt > 0;
  if (use_grid) VTRY(free_grid_build(ctx, const_cast<visacd_bvh*>(cage_bvh), pairs));
  VTRY(ensure_slot(ctx, kSlotCounters, sizeof(VisCounters)));
  VisCounters* cnt = slot<VisCounters>(ctx, kSlotCounters);
  VCUDA(cudaMemsetAsync(cnt, 0, sizeof(VisCounters), ctx->stream));
  ctx->last_n_edges = 0;

  const int64_t np = (int64_t)n * (n - 1) / 2;
  const int64_t nw = (np + 31) / 32;
  if (n < 2) {
    if (n_edges) *n_edges = 0;
    if (stats) memset(stats, 0, sizeof(*stats));
    return VISACD_OK;
  }
  // Morton order of the points; rows: the new ones in order.
  PointOrder order;
  if (ordered) {
    order = *ordered;
  } else {
    VTRY(order_slots(ctx, d_pts, n, d_new, order));
    VTRY(ensure_slot(ctx, kSlotVisOrder, points_scratch(&order, 1)));
    VTRY(points_order(ctx, &order, 1, slot<char>(ctx, kSlotVisOrder), cnt));
  }
  const uint32_t* perm = order.perm;

  const int variant = choose_vis_variant(ctx, n, d_new != nullptr, self_bvh, cage_bvh);
  const int TR = kVisVariants[variant].tr, TC = 32 / TR;
  VisParams P;
  memset(&P, 0, sizeof(P));
  P.pts = d_pts;
  P.n = n;
  P.cols = perm;
  P.nc = n;
  P.ntc = (n + TC - 1) / TC;
  if (d_new) {
    P.rows = order.rows;
    P.nr = n_new;
    P.triangular = 0;
    P.is_new = d_new;
    P.newrank = order.rank;
    P.ntr = (P.nr + TR - 1) / TR;
    P.total_tiles = (unsigned long long)P.ntr * (unsigned long long)P.ntc;
  } else {
    P.rows = perm;
    P.nr = n;
    P.triangular = 1;
    P.ntr = (n + TR - 1) / TR;
    if (TR < TC) {  // shapes whose tile rows have no closed form (tile_of)
      VTRY(ensure_slot(ctx, kSlotVisRowTiles, (size_t)P.ntr * 4 + (size_t)(P.ntr + 1) * 8 + 256));
      uint32_t* rc = slot<uint32_t>(ctx, kSlotVisRowTiles);
      uint64_t* rs = reinterpret_cast<uint64_t*>(rc + ((P.ntr + 63) & ~63LL));
      VLAUNCH(ctx, kKVisPrep, grid_for(P.ntr, 256, 4LL * ctx->sm_count), 256, 0,
              tile_row_counts_kernel, P.ntr, P.ntc, TR, TC, rc);
      VTRY(exclusive_scan_u32_to_u64(ctx, rc, rs, P.ntr));
      P.row_start = reinterpret_cast<const unsigned long long*>(rs);
    }
    // The same total as the device scan, counted here (no read-back).
    unsigned long long total = 0;
    for (int64_t r = 0; r < P.ntr; ++r) {
      const int64_t c = P.ntc - (r * TR) / TC;
      total += (unsigned long long)(c > 0 ? c : 0);
    }
    P.total_tiles = total;
  }
  P.mesh = tile_mesh(ctx, self_bvh, cage_bvh);
  // Large calls first clear what they can with the cage's free-space grid
  // (built at the top of this call): a walk kernel, then the traversal.
  if (use_grid && cage_bvh->free_lb && P.total_tiles > 0) {
    VTRY(ensure_slot(ctx, kSlotVisCleared, (size_t)P.total_tiles * 12 + 256));
    P.pend_tiles = slot<unsigned long long>(ctx, kSlotVisCleared);
    P.pend_done = reinterpret_cast<uint32_t*>(P.pend_tiles + P.total_tiles);
  }
  if (P.pend_tiles != nullptr) {
    const visacd_bvh* cb = cage_bvh;
    {
      P.cage_free.lb = cb->free_lb;
      P.cage_free.tex = cb->free_tex;
      P.cage_free.ox = cb->fg_ox;
      P.cage_free.oy = cb->fg_oy;
      P.cage_free.oz = cb->fg_oz;
      P.cage_free.h_up = cb->fg_h * 1.000001f;
      P.cage_free.inv_h = cb->fg_inv_h;
      P.cage_free.margin = cb->fg_margin;
      P.cage_free.nx = cb->fg_nx;
      P.cage_free.ny = cb->fg_ny;
      P.cage_free.nz = cb->fg_nz;
    }
    // Without room for the table the walk starts at the points.
    const int m = reach_side(n, pairs);
    if (m > 0 && ensure_slot(ctx, kSlotVisReach, reach_entries(n, m) * 4) == VISACD_OK) {
      P.cage_reach = FreeReach{slot<float>(ctx, kSlotVisReach), m, n, P.triangular};
      VTRY(launch_reach(ctx, P));
    }
  }
  VTRY(ensure_slot(ctx, kSlotBitset, (size_t)nw * 4));
  P.bitset = slot<uint32_t>(ctx, kSlotBitset);
  VCUDA(cudaMemsetAsync(P.bitset, 0, (size_t)nw * 4, ctx->stream));
  P.cnt = cnt;
  P.status = ctx->d_status;
  if (P.total_tiles > 0) VTRY(launch_vis_variant(ctx, variant, P));
  // Compaction: scan of the words' set bits, emit in linear-pair order.
  VTRY(ensure_slot(ctx, kSlotWordOffsets, (size_t)(nw + 1) * 8));
  uint64_t* wo = slot<uint64_t>(ctx, kSlotWordOffsets);
  const unsigned gw = grid_for(nw, 256, 16LL * ctx->sm_count);
  VTRY(exclusive_scan_bits(ctx, P.bitset, wo, nw));
  // A call with few pairs has room for all of them as edges: they are emitted,
  // and sent along with the counters, before their number is known here.
  const bool few = np <= kFewPairs;
  if (few) {
    VTRY(ensure_slot(ctx, kSlotEdgesOut, (size_t)np * 8));
    VLAUNCH(ctx, kKBitEmit, gw, 256, 0, bit_emit_kernel, P.bitset, nw, wo, (int64_t)n,
            slot<uint32_t>(ctx, kSlotEdgesOut));
  }
  // Counters and the status word (and those edges) in one wait.
  VisCounters* h = nullptr;
  uint32_t* hs = nullptr;
  constexpr size_t o_hs = (sizeof(VisCounters) + 15) & ~size_t(15);
  const bool send = few && few_edges;
  VTRY(pinned(ctx, o_hs + 64 + (send ? (size_t)np * 8 : 0), (void**)&h));
  hs = reinterpret_cast<uint32_t*>(reinterpret_cast<char*>(h) + o_hs);
  if (send) {
    *few_edges = hs + 16;
    VCUDA(cudaMemcpyAsync(hs + 16, ctx->buf[kSlotEdgesOut].p, (size_t)np * 8, cudaMemcpyDeviceToHost, ctx->stream));
  }
  VCUDA(cudaMemcpyAsync(h, cnt, sizeof(VisCounters), cudaMemcpyDeviceToHost, ctx->stream));
  VCUDA(cudaMemcpyAsync(hs, ctx->d_status, sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx->stream));
  VCUDA(stream_wait(ctx));
  const VisCounters hc = *h;
  VTRY(status_result(ctx, *hs, "visibility"));
  const int64_t ne = (int64_t)hc.edges;
  if (ne > 0 && !few) {
    VTRY(ensure_slot(ctx, kSlotEdgesOut, (size_t)ne * 8));
    VLAUNCH(ctx, kKBitEmit, gw, 256, 0, bit_emit_kernel, P.bitset, nw, wo, (int64_t)n,
            slot<uint32_t>(ctx, kSlotEdgesOut));
  }
  ctx->last_n_edges = ne;
  if (n_edges) *n_edges = ne;
  if (stats) {
    stats->pairs_tested = (int64_t)hc.pairs;
    stats->n_edges = ne;
    stats->self_hits = (int64_t)hc.self_hits;
    stats->cage_hits = (int64_t)hc.cage_hits;
    stats->fp64_rechecks = (int64_t)hc.rechecks;
    stats->degenerate = (int64_t)hc.degenerate;
    stats->node_visits = (int64_t)hc.node_visits;
    stats->tri_tests = (int64_t)hc.tri_tests;
  }
  ctx->last_vis_certified = (int64_t)hc.certified;
  ctx->last_vis_trace_steps = (int64_t)hc.trace_steps;
  return VISACD_OK;
}

// ---- several parts in one launch ------------------------------------------
// The edge list of all parts: word w of the concatenated bitset belongs to the
// part found by binary search over the parts' first words; its edges go to
// the global offset of the word (parts stay in order, each row-major).
__global__ void multi_emit_kernel(const VisParams* __restrict__ parts, int n_parts,
                                  const unsigned long long* __restrict__ word_start,
                                  const uint32_t* __restrict__ bits, int64_t nw,
                                  const uint64_t* __restrict__ off, uint32_t* __restrict__ edges) {
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < nw;
       w += (int64_t)gridDim.x * blockDim.x) {
    uint32_t m = bits[w];
    if (!m) continue;
    int lo = 0, hi = n_parts - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (word_start[mid] <= (unsigned long long)w) lo = mid; else hi = mid - 1;
    }
    const int64_t n = parts[lo].n;
    const int64_t k0 = (w - (int64_t)word_start[lo]) * 32;
    uint64_t o = off[w];
    double b2 = (double)(2 * n - 1);
    double disc = b2 * b2 - 8.0 * (double)k0;
    int64_t i = (int64_t)((b2 - sqrt(disc > 0 ? disc : 0.0)) * 0.5);
    if (i < 0) i = 0;
    if (i > n - 2) i = n - 2;
    while (i > 0 && row_start(i, n) > k0) --i;
    while (i + 1 <= n - 2 && row_start(i + 1, n) <= k0) ++i;
    while (m) {
      const int bpos = __ffs(m) - 1;
      m &= m - 1;
      const int64_t k = k0 + bpos;
      while (i + 1 <= n - 2 && row_start(i + 1, n) <= k) ++i;
      const int64_t j = k - row_start(i, n) + i + 1;
      edges[2 * o] = (uint32_t)i;
      edges[2 * o + 1] = (uint32_t)j;
      ++o;
    }
  }
}

// Edge offsets of the parts' first words (and the total) for the read-back.
__global__ void multi_part_offsets_kernel(const unsigned long long* __restrict__ word_start, int n_parts,
                                          const uint64_t* __restrict__ off, uint64_t* __restrict__ out) {
  for (int p = threadIdx.x; p <= n_parts; p += blockDim.x) out[p] = off[word_start[p]];
}

int visibility_multi_impl(visacd_ctx* ctx, int32_t n_parts, const float* const* pts, const int32_t* n_pts,
                          const uint8_t* const* is_new, const visacd_bvh* const* self_bvhs,
                          const visacd_bvh* const* cage_bvhs, int64_t* n_edges, visacd_vis_stats* stats) {
  VCHECK(ctx && n_parts > 0 && pts && n_pts && self_bvhs && cage_bvhs && n_edges, VISACD_ERR_INVALID_ARG,
         "visibility_batch: null argument");
  VCUDA(cudaSetDevice(ctx->device));
  constexpr int TR = 8, TC = 4;
  // Every part's checks, and the end of its BVHs' builds, come before anything
  // reads a BVH: a grid is kept for the BVH's life, so one laid from a build that
  // another context's stream had not finished would lose edges in every later call.
  for (int p = 0; p < n_parts; ++p) {
    const int32_t n = n_pts[p];
    const visacd_bvh* sb = self_bvhs[p];
    const visacd_bvh* cb = cage_bvhs[p];
    VCHECK(n >= 0 && (n == 0 || pts[p]) && sb && cb, VISACD_ERR_INVALID_ARG, "visibility_batch: bad part %d", p);
    VCHECK(n <= (1 << 24), VISACD_ERR_INVALID_ARG, "visibility_batch: part %d has n = %d above 2^24", p, n);
    VCHECK(sb->ctx && cb->ctx && sb->device == ctx->device && cb->device == ctx->device,
           VISACD_ERR_INVALID_ARG, "visibility_batch: part %d BVH is not on this context's device", p);
    VTRY(bvh_settle(ctx, sb));
    VTRY(bvh_settle(ctx, cb));
    VCHECK(sb->depth <= kStack && cb->depth <= kStack, VISACD_ERR_INVALID_ARG,
           "visibility_batch: part %d BVH depth %d/%d exceeds the traversal stack (%d)", p, sb->depth,
           cb->depth, kStack);
    VCHECK(sb->nt == 0 || sb->nv == n, VISACD_ERR_INVALID_ARG,
           "visibility_batch: part %d self BVH has %d vertices, points have %d", p, sb->nv, n);
  }
  // Free-space grids of the large parts' cages (built once per cage BVH),
  // before this call takes the shared scratch and staging buffers.
  // A part's pairs: all of them, or (masked) those with a new endpoint.
  std::vector<int64_t> part_pairs(n_parts, 0);
  std::vector<int32_t> nr(n_parts, 0);  // new points of the masked parts
  for (int p = 0; p < n_parts; ++p) {
    const int64_t n = n_pts[p];
    int64_t pairs = n * (n > 0 ? n - 1 : 0) / 2;
    if (is_new && is_new[p]) {
      int64_t k = 0;
      for (int64_t v = 0; v < n; ++v) k += is_new[p][v] != 0;
      nr[p] = (int32_t)k;
      pairs -= (n - k) * (n - k - 1) / 2;
    }
    part_pairs[p] = pairs;
  }
  bool any_grid = false;
  if (ctx->vis_trace) {
    for (int p = 0; p < n_parts; ++p) {
      if (part_pairs[p] >= kFreeGridMinPairs && cage_bvhs[p]->nt > 0) {
        VTRY(free_grid_build(ctx, const_cast<visacd_bvh*>(cage_bvhs[p]), part_pairs[p]));
        any_grid = any_grid || cage_bvhs[p]->free_lb != nullptr;
      }
    }
  }
  // Layout of the per-part arrays in one buffer (256-byte aligned pieces).
  auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
  std::vector<size_t> o_pts(n_parts), o_mask(n_parts), o_perm(n_parts), o_rows(n_parts),
      o_rank(n_parts);
  std::vector<int64_t> ntr_tri(n_parts, 0);
  size_t total = 0;
  unsigned long long words = 0;
  std::vector<unsigned long long> word_start(n_parts + 1);
  for (int p = 0; p < n_parts; ++p) {
    const int32_t n = n_pts[p];
    o_pts[p] = total;  total += al((size_t)std::max(n, 1) * 12);
    o_mask[p] = total; total += al((size_t)std::max(n, 1));
    o_perm[p] = total; total += al((size_t)std::max(n, 1) * 4);
    o_rows[p] = total; total += al((size_t)std::max(n, 1) * 4);
    o_rank[p] = total; total += al((size_t)std::max(n, 1) * 4);
    ntr_tri[p] = (n + TR - 1) / TR;
    word_start[p] = words;
    const unsigned long long np = (unsigned long long)n * (unsigned long long)(n > 0 ? n - 1 : 0) / 2;
    words += (np + 31) / 32;
  }
  word_start[n_parts] = words;
  const size_t o_desc = total;
  total += al(sizeof(VisParams) * (size_t)n_parts);
  const size_t o_tiles = total;
  total += al(8 * (size_t)(n_parts + 1));
  const size_t o_words = total;
  total += al(8 * (size_t)(n_parts + 1));
  const size_t o_poff = total;
  total += al(8 * (size_t)(n_parts + 1));
  VTRY(ensure_slot(ctx, kSlotVisMulti, total));
  char* base = slot<char>(ctx, kSlotVisMulti);
  // Upload points and masks.
  {
    size_t up_bytes = 0;
    for (int p = 0; p < n_parts; ++p) up_bytes += (size_t)n_pts[p] * 13;
    Stager up(ctx);
    VTRY(up.reserve(up_bytes + 8 * (size_t)(n_parts + 1), 2 * n_parts + 1));
    for (int p = 0; p < n_parts; ++p) {
      const int32_t n = n_pts[p];
      if (n) VTRY(up.put(base + o_pts[p], pts[p], (size_t)n * 12));
      if (n && is_new && is_new[p]) VTRY(up.put(base + o_mask[p], is_new[p], (size_t)n));
    }
    VTRY(up.put(base + o_words, word_start.data(), 8 * (size_t)(n_parts + 1)));
  }
  // Morton orders of the parts; rows and ranks of the masked ones.
  {
    std::vector<PointOrder> order(n_parts);
    for (int p = 0; p < n_parts; ++p) {
      const bool masked = is_new && is_new[p];
      order[p] = {reinterpret_cast<const float*>(base + o_pts[p]), n_pts[p],
                  reinterpret_cast<uint32_t*>(base + o_perm[p]),
                  masked ? reinterpret_cast<const uint8_t*>(base + o_mask[p]) : nullptr,
                  reinterpret_cast<uint32_t*>(base + o_rows[p]), reinterpret_cast<int32_t*>(base + o_rank[p])};
    }
    VTRY(ensure_slot(ctx, kSlotCounters, sizeof(VisCounters)));
    VTRY(ensure_slot(ctx, kSlotVisOrder, points_scratch(order.data(), n_parts)));
    VTRY(points_order(ctx, order.data(), n_parts, slot<char>(ctx, kSlotVisOrder),
                      slot<VisCounters>(ctx, kSlotCounters)));
  }
  // Part descriptors and the global work numbering.
  VTRY(ensure_slot(ctx, kSlotBitset, (size_t)std::max<unsigned long long>(words, 1) * 4));
  uint32_t* bits = slot<uint32_t>(ctx, kSlotBitset);
  VTRY(ensure_slot(ctx, kSlotCounters, sizeof(VisCounters)));
  VisCounters* cnt = slot<VisCounters>(ctx, kSlotCounters);
  std::vector<VisParams> desc(n_parts);
  std::vector<size_t> reach_at(n_parts, 0);  // of the parts with a reach table
  size_t reach_total = 0;
  std::vector<unsigned long long> tile_start(n_parts + 1, 0);
  unsigned long long tiles = 0;
  for (int p = 0; p < n_parts; ++p) {
    const int32_t n = n_pts[p];
    VisParams& P = desc[p];
    memset(&P, 0, sizeof(P));
    P.pts = reinterpret_cast<const float*>(base + o_pts[p]);
    P.n = n;
    P.cols = reinterpret_cast<const uint32_t*>(base + o_perm[p]);
    P.nc = n;
    P.ntc = (n + TC - 1) / TC;
    const bool masked = is_new && is_new[p];
    if (masked) {
      P.rows = reinterpret_cast<const uint32_t*>(base + o_rows[p]);
      P.nr = nr[p];
      P.triangular = 0;
      P.is_new = reinterpret_cast<const uint8_t*>(base + o_mask[p]);
      P.newrank = reinterpret_cast<const int32_t*>(base + o_rank[p]);
      P.ntr = (P.nr + TR - 1) / TR;
      P.total_tiles = n >= 2 ? (unsigned long long)P.ntr * (unsigned long long)P.ntc : 0ull;
    } else {
      P.rows = P.cols;
      P.nr = n;
      P.triangular = 1;
      P.ntr = ntr_tri[p];
      unsigned long long t = 0;
      for (int64_t r = 0; r < P.ntr; ++r) {
        const int64_t c = P.ntc - (r * TR) / TC;
        t += (unsigned long long)(c > 0 ? c : 0);
      }
      P.total_tiles = n >= 2 ? t : 0ull;
    }
    P.mesh = tile_mesh(ctx, self_bvhs[p], cage_bvhs[p]);
    const visacd_bvh* cb = cage_bvhs[p];
    if (any_grid && cb->free_lb && part_pairs[p] >= kFreeGridMinPairs) {
      P.cage_free.lb = cb->free_lb;
      P.cage_free.tex = cb->free_tex;
      P.cage_free.ox = cb->fg_ox;
      P.cage_free.oy = cb->fg_oy;
      P.cage_free.oz = cb->fg_oz;
      P.cage_free.h_up = cb->fg_h * 1.000001f;
      P.cage_free.inv_h = cb->fg_inv_h;
      P.cage_free.margin = cb->fg_margin;
      P.cage_free.nx = cb->fg_nx;
      P.cage_free.ny = cb->fg_ny;
      P.cage_free.nz = cb->fg_nz;
      const int m = reach_side(n, part_pairs[p]);
      if (m > 0) {
        P.cage_reach = FreeReach{nullptr, m, n, P.triangular};
        reach_at[p] = reach_total;
        reach_total += (reach_entries(n, m) + 63) & ~(size_t)63;
      }
    }
    P.bitset = bits + word_start[p];
    P.cnt = cnt;
    P.status = ctx->d_status;
    tile_start[p] = tiles;
    tiles += P.total_tiles;
  }
  tile_start[n_parts] = tiles;
  // Without room for the tables the walk starts at the points.
  const bool reaches = reach_total > 0 && ensure_slot(ctx, kSlotVisReach, reach_total * 4) == VISACD_OK;
  for (int p = 0; p < n_parts; ++p) {
    if (desc[p].cage_reach.m == 0) continue;
    if (reaches) desc[p].cage_reach.reach = slot<float>(ctx, kSlotVisReach) + reach_at[p];
    else desc[p].cage_reach = FreeReach{};
  }
  {
    VisCounters init;
    memset(&init, 0, sizeof(init));
    Stager up(ctx);
    VTRY(up.reserve(sizeof(VisParams) * (size_t)n_parts + 8 * (size_t)(n_parts + 1) + sizeof(VisCounters), 3));
    VTRY(up.put(base + o_desc, desc.data(), sizeof(VisParams) * (size_t)n_parts));
    VTRY(up.put(base + o_tiles, tile_start.data(), 8 * (size_t)(n_parts + 1)));
    VTRY(up.put(cnt, &init, sizeof(VisCounters)));
  }
  if (words) VCUDA(cudaMemsetAsync(bits, 0, (size_t)words * 4, ctx->stream));
  const VisParams* d_desc = reinterpret_cast<const VisParams*>(base + o_desc);
  const unsigned long long* d_tiles = reinterpret_cast<const unsigned long long*>(base + o_tiles);
  const unsigned long long* d_words = reinterpret_cast<const unsigned long long*>(base + o_words);
  if (tiles) {
    unsigned long long* pend = nullptr;
    uint32_t* pend_done = nullptr;
    if (any_grid) {
      VTRY(ensure_slot(ctx, kSlotVisCleared, (size_t)tiles * 12 + 256));
      pend = slot<unsigned long long>(ctx, kSlotVisCleared);
      pend_done = reinterpret_cast<uint32_t*>(pend + tiles);
      for (int p = 0; p < n_parts; ++p)
        if (desc[p].cage_reach.reach) VTRY(launch_reach(ctx, desc[p]));
      VLAUNCH(ctx, kKVisWalk, (unsigned)(ctx->sm_count * kWalkBlocks), kVisThreads, 0, visibility_multi_walk_kernel<8>,
              d_desc, n_parts, d_tiles, tiles, cnt, pend, pend_done);
    }
    VLAUNCH(ctx, kKVisibility, (unsigned)(ctx->sm_count * 8), kVisThreads, 0, (visibility_multi_kernel<8, 8>),
            d_desc, n_parts, d_tiles, tiles, cnt, ctx->d_status, pend, pend_done);
  }
  // Compaction over the concatenated bitset.
  const int64_t nw = (int64_t)words;
  VTRY(ensure_slot(ctx, kSlotWordOffsets, (size_t)(nw + 1) * 8));
  uint64_t* wo = slot<uint64_t>(ctx, kSlotWordOffsets);
  const unsigned gw = grid_for(std::max<int64_t>(nw, 1), 256, 16LL * ctx->sm_count);
  if (nw) {
    VTRY(exclusive_scan_bits(ctx, bits, wo, nw));
  } else {
    VCUDA(cudaMemsetAsync(wo, 0, 8, ctx->stream));
  }
  uint64_t* d_poff = reinterpret_cast<uint64_t*>(base + o_poff);
  VLAUNCH(ctx, kKVisPrep, 1, 256, 0, multi_part_offsets_kernel, d_words, n_parts, wo, d_poff);
  // Counters, part offsets and the status word in one wait.
  char* hb = nullptr;
  const size_t o_st = (sizeof(VisCounters) + 8 * (size_t)(n_parts + 1) + 15) & ~size_t(15);
  VTRY(pinned(ctx, o_st + 16, (void**)&hb));
  VCUDA(cudaMemcpyAsync(hb, cnt, sizeof(VisCounters), cudaMemcpyDeviceToHost, ctx->stream));
  VCUDA(cudaMemcpyAsync(hb + sizeof(VisCounters), d_poff, 8 * (size_t)(n_parts + 1), cudaMemcpyDeviceToHost,
                        ctx->stream));
  VCUDA(cudaMemcpyAsync(hb + o_st, ctx->d_status, sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx->stream));
  VCUDA(stream_wait(ctx));
  VisCounters hc;
  memcpy(&hc, hb, sizeof(hc));
  std::vector<uint64_t> poff(n_parts + 1);
  memcpy(poff.data(), hb + sizeof(VisCounters), 8 * (size_t)(n_parts + 1));
  uint32_t dev_status = 0;
  memcpy(&dev_status, hb + o_st, sizeof(uint32_t));
  VTRY(status_result(ctx, dev_status, "visibility_batch"));
  for (int p = 0; p < n_parts; ++p) n_edges[p] = (int64_t)(poff[p + 1] - poff[p]);
  const int64_t ne = (int64_t)poff[n_parts];
  VTRY(ensure_slot(ctx, kSlotEdgesOut, (size_t)(ne > 0 ? ne : 1) * 8));
  if (ne > 0) {
    VLAUNCH(ctx, kKBitEmit, gw, 256, 0, multi_emit_kernel, d_desc, n_parts, d_words, bits, nw, wo,
            slot<uint32_t>(ctx, kSlotEdgesOut));
  }
  ctx->last_n_edges = ne;
  if (stats) {
    stats->pairs_tested = (int64_t)hc.pairs;
    stats->n_edges = ne;
    stats->self_hits = (int64_t)hc.self_hits;
    stats->cage_hits = (int64_t)hc.cage_hits;
    stats->fp64_rechecks = (int64_t)hc.rechecks;
    stats->degenerate = (int64_t)hc.degenerate;
    stats->node_visits = (int64_t)hc.node_visits;
    stats->tri_tests = (int64_t)hc.tri_tests;
  }
  return VISACD_OK;
}

int visibility_impl(visacd_ctx* ctx, const float* pts, int32_t n, const uint8_t* is_new,
                    int device_ptrs, const visacd_bvh* self_bvh, const visacd_bvh* cage_bvh,
                    int64_t* n_edges, visacd_vis_stats* stats) {
  VCHECK(ctx && self_bvh && cage_bvh, VISACD_ERR_INVALID_ARG, "visibility: null argument");
  VCHECK(self_bvh->ctx && cage_bvh->ctx, VISACD_ERR_INVALID_ARG,
         "visibility: a BVH outlived the context it was built on");
  VCHECK(n >= 0 && (n == 0 || pts), VISACD_ERR_INVALID_ARG, "visibility: bad points");
  VCHECK(n <= (1 << 24), VISACD_ERR_INVALID_ARG, "visibility: n = %d above the 2^24 limit", n);
  VCHECK(self_bvh->device == ctx->device && cage_bvh->device == ctx->device,
         VISACD_ERR_INVALID_ARG, "visibility: BVH built on another device");
  VCHECK(self_bvh->depth <= kStack && cage_bvh->depth <= kStack, VISACD_ERR_INVALID_ARG,
         "visibility: BVH depth %d/%d exceeds the traversal stack (%d)", self_bvh->depth,
         cage_bvh->depth, kStack);
  VCHECK(self_bvh->nt == 0 || self_bvh->nv == n, VISACD_ERR_INVALID_ARG,
         "visibility: self BVH has %d vertices, points have %d", self_bvh->nv, n);
  VCUDA(cudaSetDevice(ctx->device));
  const float* d_pts = pts;
  const uint8_t* d_new = is_new;
  int64_t pairs = (int64_t)n * (n > 0 ? n - 1 : 0) / 2;
  int32_t n_new = 0;
  VTRY(bvh_settle(ctx, self_bvh));
  VTRY(bvh_settle(ctx, cage_bvh));
  if (is_new) {
    int64_t k = 0;
    if (device_ptrs && n > 0) {
      VTRY(ensure_slot(ctx, kSlotCounters, sizeof(VisCounters)));
      unsigned long long* d_rows = &slot<VisCounters>(ctx, kSlotCounters)->n_rows;
      unsigned long long* h_rows = nullptr;
      VTRY(pinned(ctx, sizeof(*h_rows), (void**)&h_rows));
      VCUDA(cudaMemsetAsync(d_rows, 0, sizeof(*d_rows), ctx->stream));
      VLAUNCH(ctx, kKVisPrep, grid_for(n, 256, 4LL * ctx->sm_count), 256, 0, mask_count_kernel, d_new, n, d_rows);
      VCUDA(cudaMemcpyAsync(h_rows, d_rows, sizeof(*h_rows), cudaMemcpyDeviceToHost, ctx->stream));
      VCUDA(stream_wait(ctx));
      k = (int64_t)*h_rows;
    } else {
      for (int32_t v = 0; v < n; ++v) k += is_new[v] != 0;
    }
    n_new = (int32_t)k;
    pairs -= ((int64_t)n - k) * ((int64_t)n - k - 1) / 2;
  }
  if (!device_ptrs && n > 0) {
    VTRY(ensure_slot(ctx, kSlotPoints, (size_t)n * 12));
    if (is_new) VTRY(ensure_slot(ctx, kSlotMask, (size_t)n));
    Stager up(ctx);
    VTRY(up.reserve((size_t)n * 13, 2));
    VTRY(up.put(ctx->buf[kSlotPoints].p, pts, (size_t)n * 12));
    d_pts = slot<float>(ctx, kSlotPoints);
    if (is_new) {
      VTRY(up.put(ctx->buf[kSlotMask].p, is_new, (size_t)n));
      d_new = slot<uint8_t>(ctx, kSlotMask);
    }
  }
  return vis_device(ctx, d_pts, n, d_new, self_bvh, cage_bvh, n_edges, stats, pairs, n_new, nullptr, nullptr);
}

// compute_intersection_matrix on checked input: the part, its mask and the
// cage in one upload, both BVHs and the points' order in one launch.
static int matrix_together(visacd_ctx* ctx, const float* verts, int32_t nv, const uint32_t* tris, int32_t nt,
                           const uint8_t* is_new, const float* cage_verts, int32_t ncv, const uint32_t* cage_tris,
                           int32_t nct, visacd_bvh** sb, visacd_bvh** cb, int64_t* n_edges, visacd_vis_stats* stats,
                           const uint32_t** few_edges) {
  VCUDA(cudaSetDevice(ctx->device));
  auto al = [](size_t b) { return (b + 63) & ~size_t(63); };
  const void* src[5] = {verts, tris, cage_verts, cage_tris, is_new};
  const size_t bytes[5] = {(size_t)nv * 12, (size_t)nt * 12, (size_t)ncv * 12, (size_t)nct * 12,
                           is_new ? (size_t)nv : 0};
  size_t at[5], total = 0;
  for (int k = 0; k < 5; ++k) {
    at[k] = total;
    total += al(bytes[k]);
  }
  VTRY(ensure_slot(ctx, kSlotBuildVerts, total));
  char* d = slot<char>(ctx, kSlotBuildVerts);
  Stager up(ctx);
  VTRY(up.reserve(total, 1));
  for (int k = 0; k < 5; ++k)
    if (bytes[k]) memcpy(up.host() + at[k], src[k], bytes[k]);
  VTRY(up.copy(d, total));
  const float* d_pts = reinterpret_cast<const float*>(d + at[0]);
  const uint8_t* d_new = is_new ? reinterpret_cast<const uint8_t*>(d + at[4]) : nullptr;
  OrderJob jobs[3];
  PointOrder order;
  VTRY(order_slots(ctx, d_pts, nv, d_new, order));
  VTRY(ensure_slot(ctx, kSlotTmpTris, order_scratch(nt, true) + order_scratch(nct, true) + order_scratch(nv, false)));
  char* scratch = slot<char>(ctx, kSlotTmpTris);
  VTRY(bvh_prepare(ctx, d_pts, nv, reinterpret_cast<const uint32_t*>(d + at[1]), nt, scratch, sb, jobs[0]));
  scratch += order_scratch(nt, true);
  VTRY(bvh_prepare(ctx, reinterpret_cast<const float*>(d + at[2]), ncv, reinterpret_cast<const uint32_t*>(d + at[3]),
                   nct, scratch, cb, jobs[1]));
  scratch += order_scratch(nct, true);
  jobs[2] = points_job(order, scratch);
  VTRY(order_run(ctx, jobs, 3));
  VTRY(order_nodes(ctx, jobs, 2));
  int64_t pairs = (int64_t)nv * (nv - 1) / 2;
  int32_t n_new = 0;
  if (is_new) {
    for (int32_t v = 0; v < nv; ++v) n_new += is_new[v] != 0;
    pairs -= ((int64_t)nv - n_new) * ((int64_t)nv - n_new - 1) / 2;
  }
  return vis_device(ctx, d_pts, nv, d_new, *sb, *cb, n_edges, stats, pairs, n_new, &order, few_edges);
}

}  // namespace vgpu

using namespace vgpu;

extern "C" int visacd_visibility(visacd_ctx* ctx, const float* pts, int32_t n,
                                 const uint8_t* is_new, int device_ptrs,
                                 const visacd_bvh* self_bvh, const visacd_bvh* cage_bvh,
                                 int64_t* n_edges, visacd_vis_stats* stats) {
  return visibility_impl(ctx, pts, n, is_new, device_ptrs, self_bvh, cage_bvh, n_edges, stats);
}

extern "C" int visacd_visibility_batch(visacd_ctx* ctx, int32_t n_parts, const float* const* pts,
                                       const int32_t* n_pts, const uint8_t* const* is_new,
                                       const visacd_bvh* const* self_bvhs,
                                       const visacd_bvh* const* cage_bvhs, int64_t* n_edges,
                                       visacd_vis_stats* stats) {
  return visibility_multi_impl(ctx, n_parts, pts, n_pts, is_new, self_bvhs, cage_bvhs, n_edges, stats);
}

extern "C" int visacd_visibility_edges(visacd_ctx* ctx, uint32_t* edges_out,
                                       int64_t capacity_edges) {
  VCHECK(ctx, VISACD_ERR_INVALID_ARG, "visibility_edges: null context");
  VCHECK(capacity_edges >= ctx->last_n_edges, VISACD_ERR_CAPACITY,
         "visibility_edges: capacity %lld < %lld edges", (long long)capacity_edges,
         (long long)ctx->last_n_edges);
  if (ctx->last_n_edges == 0) return VISACD_OK;
  VCHECK(edges_out, VISACD_ERR_INVALID_ARG, "visibility_edges: edges_out is NULL");
  VCUDA(cudaMemcpyAsync(edges_out, ctx->buf[kSlotEdgesOut].p, (size_t)ctx->last_n_edges * 8,
                        cudaMemcpyDeviceToHost, ctx->stream));
  VCUDA(stream_wait(ctx));
  return VISACD_OK;
}

extern "C" int visacd_visibility_edges_device(visacd_ctx* ctx, const uint32_t** d_edges,
                                              int64_t* n_edges) {
  VCHECK(ctx && d_edges && n_edges, VISACD_ERR_INVALID_ARG, "visibility_edges_device: null");
  *d_edges = slot<uint32_t>(ctx, kSlotEdgesOut);
  *n_edges = ctx->last_n_edges;
  return VISACD_OK;
}

extern "C" int visacd_compute_intersection_matrix(
    visacd_ctx* ctx, const float* verts, int32_t nv, const uint32_t* tris, int32_t nt,
    const uint8_t* is_new, const float* cage_verts, int32_t ncv, const uint32_t* cage_tris,
    int32_t nct, uint32_t* edges_out, int64_t capacity_edges, int64_t* n_edges,
    visacd_vis_stats* stats) {
  VCHECK(ctx && n_edges, VISACD_ERR_INVALID_ARG, "compute_intersection_matrix: null argument");
  visacd_bvh *sb = nullptr, *cb = nullptr;
  const uint32_t* few_edges = nullptr;
  int rc;
  // Part and cage of ordinary size: one upload, both builds and the points'
  // order in one launch. Anything else (and every refusal) one by one.
  const bool together = verts && tris && cage_verts && cage_tris && nv >= 2 && nv <= kOrderMax && nt >= 1 &&
                        nt <= kOrderMax && ncv >= 1 && nct >= 1 && nct <= kOrderMax &&
                        indices_in_range(reinterpret_cast<const int32_t*>(tris), 3LL * nt, nv) &&
                        indices_in_range(reinterpret_cast<const int32_t*>(cage_tris), 3LL * nct, ncv);
  if (together) {
    rc = matrix_together(ctx, verts, nv, tris, nt, is_new, cage_verts, ncv, cage_tris, nct, &sb, &cb, n_edges, stats,
                         &few_edges);
  } else {
    rc = bvh_build(ctx, verts, nv, tris, nt, 0, &sb);
    if (rc == VISACD_OK) rc = bvh_build(ctx, cage_verts, ncv, cage_tris, nct, 0, &cb);
    if (rc == VISACD_OK) {
      // A BVH over a mesh with no triangles still needs the vertex count check.
      if (sb->nt == 0) sb->nv = nv;
      rc = visibility_impl(ctx, verts, nv, is_new, 0, sb, cb, n_edges, stats);
    }
  }
  if (rc == VISACD_OK) {
    if (*n_edges > capacity_edges) {
      set_error("compute_intersection_matrix: %lld edges exceed capacity %lld",
                (long long)*n_edges, (long long)capacity_edges);
      rc = VISACD_ERR_CAPACITY;
    } else if (few_edges && (edges_out || *n_edges == 0)) {
      if (*n_edges) memcpy(edges_out, few_edges, (size_t)*n_edges * 8);
    } else {
      rc = visacd_visibility_edges(ctx, edges_out, capacity_edges);
    }
  }
  visacd_bvh_destroy(sb);
  visacd_bvh_destroy(cb);
  return rc;
}

// ---------------------------------------------------------------------------
// Launch-shape control and the visibility autotuner.
// ---------------------------------------------------------------------------
extern "C" int visacd_vis_variant_count(void) { return kNumVisVariants; }

extern "C" int visacd_ctx_set_vis_variant(visacd_ctx* ctx, int variant) {
  VCHECK(ctx, VISACD_ERR_INVALID_ARG, "set_vis_variant: null context");
  VCHECK(variant >= -1 && variant < kNumVisVariants, VISACD_ERR_INVALID_ARG,
         "set_vis_variant: variant %d out of range", variant);
  ctx->vis_variant_override = variant;
  return VISACD_OK;
}

extern "C" int visacd_ctx_set_vis_trace(visacd_ctx* ctx, int enable) {
  VCHECK(ctx, VISACD_ERR_INVALID_ARG, "set_vis_trace: null context");
  ctx->vis_trace = enable != 0;
  return VISACD_OK;
}

extern "C" int visacd_ctx_vis_trace_counts(const visacd_ctx* ctx, int64_t* cleared, int64_t* grid_reads) {
  VCHECK(ctx, VISACD_ERR_INVALID_ARG, "vis_trace_counts: null context");
  if (cleared) *cleared = ctx->last_vis_certified;
  if (grid_reads) *grid_reads = ctx->last_vis_trace_steps;
  return VISACD_OK;
}

extern "C" int visacd_autotune_visibility(visacd_ctx* ctx, const float* pts, int32_t n,
                                          const uint8_t* is_new, int device_ptrs,
                                          const visacd_bvh* self_bvh, const visacd_bvh* cage_bvh,
                                          int* best_variant, double* ms_per_variant) {
  VCHECK(ctx && self_bvh && cage_bvh, VISACD_ERR_INVALID_ARG, "autotune: null argument");
  VCHECK(self_bvh->ctx && cage_bvh->ctx, VISACD_ERR_INVALID_ARG,
         "autotune: a BVH outlived the context it was built on");
  const int saved_override = ctx->vis_variant_override;
  const bool saved_timing = ctx->timing;
  int best = 0;
  double best_ms = 1e300;
  int rc = VISACD_OK;
  for (int v = 0; v < kNumVisVariants && rc == VISACD_OK; ++v) {
    ctx->vis_variant_override = v;
    double ms = 0.0;
    for (int rep = 0; rep < 2 && rc == VISACD_OK; ++rep) {
      ctx->timing = true;
      rc = visacd_ctx_reset_times(ctx);
      if (rc == VISACD_OK)
        rc = visibility_impl(ctx, pts, n, is_new, device_ptrs, self_bvh, cage_bvh, nullptr, nullptr);
      const char* names[64];
      double t[64];
      int64_t cnt[64];
      int nk = 0;
      if (rc == VISACD_OK) rc = visacd_ctx_kernel_times(ctx, names, t, cnt, 64, &nk);
      ms = 0.0;
      for (int k = 0; k < nk && k < 64; ++k)
        if (strcmp(names[k], kernel_name(kKVisibility)) == 0 || strcmp(names[k], kernel_name(kKVisWalk)) == 0)
          ms += t[k];
    }
    if (ms_per_variant) ms_per_variant[v] = ms;
    if (ms < best_ms) {
      best_ms = ms;
      best = v;
    }
  }
  ctx->vis_variant_override = saved_override;
  ctx->timing = saved_timing;
  visacd_ctx_reset_times(ctx);
  if (rc != VISACD_OK) return rc;
  ctx->vis_tuned[vis_shape_class(n, is_new != nullptr, self_bvh, cage_bvh)] = best;
  if (best_variant) *best_variant = best;
  return VISACD_OK;
}
