// Per-part mesh clipping on the GPU (the cap triangulation stays on the host).
//
// Semantics of lib/src/clip.cpp:190-741, bit-exact with this project's host
// restatement (FP64 with explicit round-to-nearest intrinsics in the host's
// operation order):
//  1. clip_classify: per triangle, the sides of its vertices (1e-6 test) and
//     its case. Triangles strictly on one side (|sum of sides| = 3, including
//     the all-on-plane case oriented by the face normal) are "simple": they
//     keep their vertices and emit themselves. All others touch the plane and
//     get a record: the case and the border points it asks for (FP64, spread
//     over the whole grid: one SM's FP64 rate is what bounded the resolver
//     when it computed them).
//  2. clip_resolve: one CTA gives every request its border point. The
//     reference deduplicates them in triangle order: by vertex key, by edge
//     key and by position (1e-4 per coordinate, first match wins). Here the
//     keys' first requests are found with a hash table, numbered by a scan,
//     near positions found by comparing all first requests, and the keep-first
//     rule settled in rounds over the (few) near pairs. Triangles whose case
//     overwrites an edge's point (the plane through a vertex of a crossed
//     triangle), very many near pairs and very large cuts take the ordered
//     walk instead: one warp in triangle order. Emits each touching
//     triangle's pieces, border edges (unique unordered pairs, first
//     occurrence) and the kept-vertex flags.
//  3. Order-preserving offsets over per-triangle output counts and per-vertex
//     kept flags (tile sums, then every tile adds up the sums before it), then
//     scatter + remap into part-local indices.
#include "common.cuh"

namespace vgpu {

constexpr int kClipResolveThreads = 512;

struct ClipCounters {
  unsigned n_touch;     // touching triangles
  unsigned n_border;    // border points
  unsigned n_bedges;    // unique border edges
  unsigned overflow;    // hash/table overflow (the call fails)
  unsigned n_pos, n_neg;    // output triangles per side
  unsigned nv_pos, nv_neg;  // kept original vertices per side
};

struct PieceSlot {   // pieces of one touching triangle (<= 3 per side)
  int pos[3][3];
  int neg[3][3];
  int npos, nneg;
};

__device__ __forceinline__ double dm(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double da(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double ds(double a, double b) { return __dsub_rn(a, b); }

// ((p0 a + p1 b) + p2 c) + d, the host's order.
__device__ __forceinline__ int side_of(const double* p, const double* pl) {
  double r = da(da(da(dm(p[0], pl[0]), dm(p[1], pl[1])), dm(p[2], pl[2])), pl[3]);
  if (r > 1e-6) return 1;
  if (r < -1e-6) return -1;
  return 0;
}

// Orientation of a triangle lying in the plane (host face_normal + the sign
// rule of lib/include/core.hpp:169-176).
__device__ int coplanar_side(const double* p0, const double* p1, const double* p2, const double* pl) {
  double v0 = ds(p1[0], p0[0]), v1 = ds(p1[1], p0[1]), v2 = ds(p1[2], p0[2]);
  double w0 = ds(p2[0], p0[0]), w1 = ds(p2[1], p0[1]), w2 = ds(p2[2], p0[2]);
  double n0 = ds(dm(v1, w2), dm(v2, w1));
  double n1 = ds(dm(v2, w0), dm(v0, w2));
  double n2 = ds(dm(v0, w1), dm(v1, w0));
  double l = __dsqrt_rn(da(da(dm(n0, n0), dm(n1, n1)), dm(n2, n2)));
  double a0 = __ddiv_rn(n0, l), a1 = __ddiv_rn(n1, l), a2 = __ddiv_rn(n2, l);
  if (dm(a0, pl[0]) > 0 || dm(a1, pl[1]) > 0 || dm(a2, pl[2]) > 0) return -1;
  return 1;
}

// Plane-line intersection of p1-p2 in the host's formula order
// (lib/include/core.hpp:187-210 form), accepted inside the widened bbox.
__device__ bool intersect_segment(const double* pl, const double* p1, const double* p2, double* pi) {
  const double a = pl[0], b = pl[1], c = pl[2], d = pl[3], eps = 1e-6;
  double den = da(da(da(da(ds(dm(a, p2[0]), dm(a, p1[0])), dm(b, p2[1])), -dm(b, p1[1])), dm(c, p2[2])),
                  -dm(c, p1[2]));
  double n0 = ds(ds(ds(da(da(dm(dm(p1[0], b), p2[1]), dm(dm(p1[0], c), p2[2])), dm(p1[0], d)),
                        dm(dm(p2[0], b), p1[1])),
                     dm(dm(p2[0], c), p1[2])),
                  dm(p2[0], d));
  double n1 = ds(ds(ds(da(da(dm(dm(a, p2[0]), p1[1]), dm(dm(c, p1[1]), p2[2])), dm(p1[1], d)),
                        dm(dm(a, p1[0]), p2[1])),
                     dm(dm(c, p1[2]), p2[1])),
                  dm(p2[1], d));
  double n2 = ds(ds(ds(da(da(dm(dm(a, p2[0]), p1[2]), dm(dm(b, p2[1]), p1[2])), dm(p1[2], d)),
                        dm(dm(a, p1[0]), p2[2])),
                     dm(dm(b, p1[1]), p2[2])),
                  dm(p2[2], d));
  pi[0] = __ddiv_rn(n0, den);
  pi[1] = __ddiv_rn(n1, den);
  pi[2] = __ddiv_rn(n2, den);
  for (int k = 0; k < 3; ++k) {
    double lo = fmin(ds(p1[k], eps), ds(p2[k], eps)), hi = fmax(da(p1[k], eps), da(p2[k], eps));
    if (!(lo <= pi[k] && pi[k] <= hi)) return false;
  }
  return true;
}

// A touching triangle's case (classify) and the points of the edges it crosses.
enum : int {
  kTouchNone = 0,     // emits nothing
  kTouchOneOff = 1,   // one vertex (a) off the plane, two on it
  kTouchTwoOff = 2,   // one vertex (a) on the plane, two off it
  kTouchCross = 3,    // edges a and a + 1 crossed, vertex a + 1 between them
  kTouchVertex = 4,   // the plane through vertex a, the opposite edge crossed
};
struct ClipTouch {
  double pi[2][3];  // kTouchCross: the crossings of edges a and a + 1
  int kind;
  int a;
  int pos;          // kTouchOneOff/TwoOff: 1 on the positive side; kTouchCross: vertex a + 1 is
  int pad;
};

// code: 0 simple pos, 1 simple neg, 2 touching. For simple triangles the kept
// flags of the three vertices are raised here. Blocks of 64: a decomposition's
// part has a few thousand triangles, and the touching ones' FP64 work is
// spread over as many SMs as there are blocks.
__global__ void __launch_bounds__(64) clip_classify_kernel(const double* __restrict__ v, const int* __restrict__ t,
                                                           int nt, const double* __restrict__ plp,
                                                           unsigned char* __restrict__ code,
                                                           ClipTouch* __restrict__ touch,
                                                           unsigned char* __restrict__ keep_pos,
                                                           unsigned char* __restrict__ keep_neg) {
  const double pl[4] = {plp[0], plp[1], plp[2], plp[3]};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nt; i += gridDim.x * blockDim.x) {
    const int id[3] = {t[3 * (int64_t)i], t[3 * (int64_t)i + 1], t[3 * (int64_t)i + 2]};
    double p[3][3];
    int s[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
#pragma unroll
      for (int x = 0; x < 3; ++x) p[k][x] = v[3 * (int64_t)id[k] + x];
      s[k] = side_of(p[k], pl);
    }
    if (s[0] == 0 && s[1] == 0 && s[2] == 0) s[0] = s[1] = s[2] = coplanar_side(p[0], p[1], p[2], pl);
    const int sum = s[0] + s[1] + s[2];
    if (sum == 3 || sum == -3) {
      code[i] = sum == 3 ? 0 : 1;
      unsigned char* k = sum == 3 ? keep_pos : keep_neg;
      k[id[0]] = 1;
      k[id[1]] = 1;
      k[id[2]] = 1;
      continue;
    }
    code[i] = 2;
    const int nzero = (s[0] == 0) + (s[1] == 0) + (s[2] == 0);
    const bool one_pos = sum == 2 || (sum == 1 && nzero == 2);
    const bool one_neg = sum == -2 || (sum == -1 && nzero == 2);
    ClipTouch r;
    r.kind = kTouchNone;
    r.a = r.pos = r.pad = 0;
    if (one_pos || one_neg) {
      r.pos = one_pos ? 1 : 0;
      const bool one_off = sum == 1 || sum == -1;
      r.kind = one_off ? kTouchOneOff : kTouchTwoOff;
      if (one_off) r.a = s[0] != 0 ? 0 : (s[1] != 0 ? 1 : 2);
      else r.a = s[0] == 0 ? 0 : (s[1] == 0 ? 1 : 2);
    } else {
      double pi[3][3];
      bool f[3];
#pragma unroll
      for (int e = 0; e < 3; ++e) f[e] = intersect_segment(pl, p[e], p[(e + 1) % 3], pi[e]);
      int e = -1;
      if (f[0] && f[1] && !f[2]) e = 0;
      else if (f[1] && f[2] && !f[0]) e = 1;
      else if (f[2] && f[0] && !f[1]) e = 2;
      if (e >= 0) {
        r.kind = kTouchCross;
        r.a = e;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          if (k == e) {
            r.pos = s[(k + 1) % 3] == 1 ? 1 : 0;
            for (int x = 0; x < 3; ++x) {
              r.pi[0][x] = pi[k][x];
              r.pi[1][x] = pi[(k + 1) % 3][x];
            }
          }
        }
      } else if (f[0] && f[1] && f[2]) {
        const bool all_nz = s[0] != 0 && s[1] != 0 && s[2] != 0;
        auto same = [](const double* x, const double* y) {
          const double eps = (double)1e-5f;
          return fabs(ds(x[0], y[0])) < eps && fabs(ds(x[1], y[1])) < eps && fabs(ds(x[2], y[2])) < eps;
        };
        int k = -1;
        if (s[0] == 0 || (all_nz && same(pi[0], pi[2]))) k = 0;
        else if (s[1] == 0 || (all_nz && same(pi[0], pi[1]))) k = 1;
        else if (s[2] == 0 || (all_nz && same(pi[1], pi[2]))) k = 2;
        if (k >= 0) {
          r.kind = kTouchVertex;
          r.a = k;
        }
      }
    }
    touch[i] = r;
  }
}

// ---- the ordered resolver (one CTA) ----------------------------------------
struct Resolver {
  const double* v;
  double* border;       // 3 doubles per border point
  int* vmap;            // mesh vertex -> border point (-1)
  int* ekeys;           // edge hash: key pairs (a, b), -1 empty
  int* evals;           // edge hash values
  int ecap;             // power of two
  int2* bedge;          // unique border edges (1-based), in order
  int* bkeys;           // unordered-pair hash for edge dedup
  int bcap;
  int max_border;
  ClipCounters* cnt;
  unsigned* n_border;   // border point count (cnt->n_border, or a shared-memory copy)
  unsigned* n_bedges;   // border edge count (likewise)
};

// Shared-memory mode of the resolver: up to kSmemTouch touching triangles have
// at most 3 border points each, at most 6 directed-edge entries each and at
// most one border edge each, so tables of these capacities never fill.
constexpr int kSmemTouch = 1024;
constexpr int kSmemBorder = 3 * kSmemTouch + 16;
constexpr int kSmemEcap = 8192;
constexpr int kSmemBcap = 4096;
constexpr int kChunk = 32;
constexpr size_t kResolveSmem = (size_t)kSmemBorder * 24 + (size_t)kSmemEcap * 12 + (size_t)kSmemBcap * 8 +
                                (size_t)kChunk * 18 * 8 + (size_t)kChunk * 7 * 4 + 16;

// One warp resolves the touching triangles in order. Lane 0 owns every table
// update; the position scan runs across the 32 lanes (first match = smallest
// index with all three coordinates within 1e-4).
__device__ int find_near(Resolver& R, const double* p, int n) {
  int best = 0x7fffffff;
  for (int i = (int)(threadIdx.x & 31); i < n; i += 32) {
    const double* q = R.border + 3 * (int64_t)i;
    if (fabs(ds(q[0], p[0])) < 1e-4 && fabs(ds(q[1], p[1])) < 1e-4 && fabs(ds(q[2], p[2])) < 1e-4) {
      best = i;
      break;
    }
  }
  best = __reduce_min_sync(0xffffffffu, best);
  return best == 0x7fffffff ? -1 : best;
}

__device__ __forceinline__ unsigned hash2(int a, int b) {
  unsigned h = (unsigned)a * 0x9E3779B1u ^ ((unsigned)b + 0x7F4A7C15u) * 0x85EBCA77u;
  return h ^ (h >> 15);
}

// Directed edge table (thread 0 only).
__device__ int edge_get(Resolver& R, int a, int b) {
  unsigned m = (unsigned)R.ecap - 1u, h = hash2(a, b) & m;
  for (int probe = 0; probe < R.ecap; ++probe, h = (h + 1) & m) {
    if (R.ekeys[2 * h] == -1) return -1;
    if (R.ekeys[2 * h] == a && R.ekeys[2 * h + 1] == b) return R.evals[h];
  }
  return -1;
}
__device__ void edge_set(Resolver& R, int a, int b, int val) {
  unsigned m = (unsigned)R.ecap - 1u, h = hash2(a, b) & m;
  for (int probe = 0; probe < R.ecap; ++probe, h = (h + 1) & m) {
    if (R.ekeys[2 * h] == -1 || (R.ekeys[2 * h] == a && R.ekeys[2 * h + 1] == b)) {
      R.ekeys[2 * h] = a;
      R.ekeys[2 * h + 1] = b;
      R.evals[h] = val;
      return;
    }
  }
  R.cnt->overflow = 1;
}

__device__ __forceinline__ bool lane0() { return (threadIdx.x & 31) == 0; }

// Append a new border point (lane 0) or report overflow.
__device__ int append_border(Resolver& R, const double* p, int n) {
  if (n < R.max_border) {
    R.border[3 * n] = p[0];
    R.border[3 * n + 1] = p[1];
    R.border[3 * n + 2] = p[2];
    *R.n_border = n + 1;
    return n;
  }
  R.cnt->overflow = 1;
  return 0;
}

// Border point of a mesh vertex (whole warp calls; result broadcast).
__device__ int vertex_point(Resolver& R, int id) {
  int have = lane0() ? R.vmap[id] : 0;
  have = __shfl_sync(0xffffffffu, have, 0);
  if (have >= 0) return have;
  const int n = (int)*(volatile unsigned*)R.n_border;
  int f = find_near(R, R.v + 3 * (int64_t)id, n);
  if (lane0()) {
    if (f < 0) f = append_border(R, R.v + 3 * (int64_t)id, n);
    R.vmap[id] = f;
  }
  f = __shfl_sync(0xffffffffu, f, 0);
  __syncwarp();
  return f;
}

// Border point where edge (a, b) crosses the plane (whole warp).
__device__ int edge_point(Resolver& R, int a, int b, const double* p) {
  int have = 0;
  if (lane0()) {
    have = edge_get(R, a, b);
    if (have < 0) have = edge_get(R, b, a);
  }
  have = __shfl_sync(0xffffffffu, have, 0);
  if (have >= 0) return have;
  const int n = (int)*(volatile unsigned*)R.n_border;
  int f = find_near(R, p, n);
  if (lane0()) {
    if (f < 0) f = append_border(R, p, n);
    edge_set(R, a, b, f);
    edge_set(R, b, a, f);
  }
  f = __shfl_sync(0xffffffffu, f, 0);
  __syncwarp();
  return f;
}

// Unique unordered border edge, in first-occurrence order (thread 0 only).
__device__ void add_bedge(Resolver& R, int a, int b) {
  int lo = min(a, b), hi = max(a, b);
  unsigned m = (unsigned)R.bcap - 1u, h = hash2(lo, hi) & m;
  for (int probe = 0; probe < R.bcap; ++probe, h = (h + 1) & m) {
    if (R.bkeys[2 * h] == lo && R.bkeys[2 * h + 1] == hi) return;
    if (R.bkeys[2 * h] == -1) {
      R.bkeys[2 * h] = lo;
      R.bkeys[2 * h + 1] = hi;
      unsigned k = *R.n_bedges;
      R.bedge[k] = make_int2(a, b);
      *R.n_bedges = k + 1;
      return;
    }
  }
  R.cnt->overflow = 1;
}

__device__ __forceinline__ int bref(int b) { return -b - 1; }

// Empties the tables the ordered walk uses (the whole block): the touching
// triangles' vertices, and above kSmemTouch global edge tables of the capacity these
// triangles need, with the load factor of the full ones (a quarter at most). Emptied
// to their full size by the one warp, they took 10 ms for 980,000 triangles of which
// 1,400 touch the plane, beside 16 for the walk.
__device__ void ordered_tables(Resolver& R, const int* __restrict__ t, const int* __restrict__ list, int ntouch) {
  const int tid = threadIdx.x, nth = blockDim.x;
  for (int i = tid; i < 3 * ntouch; i += nth) R.vmap[t[3 * (int64_t)list[i / 3] + i % 3]] = -1;
  if (ntouch <= kSmemTouch) return;
  int ecap = 64, bcap = 64;
  while (ecap < R.ecap && ecap < 24 * (int64_t)ntouch) ecap <<= 1;
  while (bcap < R.bcap && bcap < 12 * (int64_t)ntouch) bcap <<= 1;
  R.ecap = ecap;
  R.bcap = bcap;
  for (int64_t i = tid; i < 2LL * ecap; i += nth) R.ekeys[i] = -1;
  for (int64_t i = tid; i < 2LL * bcap; i += nth) R.bkeys[i] = -1;
}

// The ordered walk (one warp): the general form of the resolver. With at most
// kSmemTouch touching triangles the tables, the border points and the
// counters live in shared memory (copied out at the end); otherwise in the
// global buffers sized by the triangle count. Either way the triangles are
// staged 32 at a time, one lane each, together with everything about them
// that does not depend on the tables (sides with the coplanar rule, the three
// edge-plane intersections).
__device__ __noinline__ void resolve_ordered(const double* __restrict__ v, const int* __restrict__ t,
                                             const double* __restrict__ plp, const int* __restrict__ list, int ntouch,
                                             Resolver R, PieceSlot* __restrict__ slots,
                                             unsigned char* __restrict__ keep_pos,
                                             unsigned char* __restrict__ keep_neg) {
  extern __shared__ __align__(16) unsigned char rsm[];
  double* sm_border = reinterpret_cast<double*>(rsm);
  int* sm_ekeys = reinterpret_cast<int*>(sm_border + 3 * kSmemBorder);
  int* sm_evals = sm_ekeys + 2 * kSmemEcap;
  int* sm_bkeys = sm_evals + kSmemEcap;
  double* ch_p = reinterpret_cast<double*>(sm_bkeys + 2 * kSmemBcap);  // kChunk x 9 vertex coordinates
  double* ch_pi = ch_p + kChunk * 9;                                   // kChunk x 9 edge intersections
  int* ch_id = reinterpret_cast<int*>(ch_pi + kChunk * 9);             // kChunk x 3
  int* ch_s = ch_id + kChunk * 3;                                      // kChunk x 3
  int* ch_f = ch_s + kChunk * 3;                                       // kChunk intersection flags
  unsigned* sm_cnt = reinterpret_cast<unsigned*>(ch_f + kChunk);       // n_border, n_bedges
  const int lane = threadIdx.x & 31;
  const double pl[4] = {plp[0], plp[1], plp[2], plp[3]};
  double* const global_border = R.border;
  const bool smem = ntouch <= kSmemTouch;
  if (smem) {
    for (int i = lane; i < 2 * kSmemEcap; i += 32) sm_ekeys[i] = -1;
    for (int i = lane; i < 2 * kSmemBcap; i += 32) sm_bkeys[i] = -1;
    if (lane == 0) sm_cnt[0] = sm_cnt[1] = 0;
    R.border = sm_border;
    R.ekeys = sm_ekeys;
    R.evals = sm_evals;
    R.ecap = kSmemEcap;
    R.bkeys = sm_bkeys;
    R.bcap = kSmemBcap;
    R.max_border = kSmemBorder;
    R.n_border = sm_cnt;
    R.n_bedges = sm_cnt + 1;
  } else {
    R.n_border = &R.cnt->n_border;
    R.n_bedges = &R.cnt->n_bedges;
  }
  __syncwarp();
  for (int li = 0; li < ntouch; ++li) {
    const int cc = li % kChunk;
    if (cc == 0) {
      __syncwarp();
      if (li + lane < ntouch) {
        const int tr = list[li + lane];
        int sl[3];
        for (int k = 0; k < 3; ++k) {
          const int vk = t[3 * tr + k];
          ch_id[3 * lane + k] = vk;
          for (int a = 0; a < 3; ++a) ch_p[9 * lane + 3 * k + a] = v[3 * (int64_t)vk + a];
          sl[k] = side_of(ch_p + 9 * lane + 3 * k, pl);
        }
        const double* q = ch_p + 9 * lane;
        if (sl[0] == 0 && sl[1] == 0 && sl[2] == 0) sl[0] = sl[1] = sl[2] = coplanar_side(q, q + 3, q + 6, pl);
        int fl = 0;
        for (int e = 0; e < 3; ++e)
          if (intersect_segment(pl, q + 3 * e, q + 3 * ((e + 1) % 3), ch_pi + 9 * lane + 3 * e)) fl |= 1 << e;
        for (int k = 0; k < 3; ++k) ch_s[3 * lane + k] = sl[k];
        ch_f[lane] = fl;
      }
      __syncwarp();
    }
    const int id[3] = {ch_id[3 * cc], ch_id[3 * cc + 1], ch_id[3 * cc + 2]};
    const int s[3] = {ch_s[3 * cc], ch_s[3 * cc + 1], ch_s[3 * cc + 2]};
    const int sum = s[0] + s[1] + s[2];
    const int nzero = (s[0] == 0) + (s[1] == 0) + (s[2] == 0);
    PieceSlot out;
    out.npos = out.nneg = 0;
    auto emit = [&](bool pos, int x, int y, int z) {
      if (pos) {
        out.pos[out.npos][0] = x; out.pos[out.npos][1] = y; out.pos[out.npos][2] = z; ++out.npos;
      } else {
        out.neg[out.nneg][0] = x; out.neg[out.nneg][1] = y; out.neg[out.nneg][2] = z; ++out.nneg;
      }
    };
    auto keep = [&](bool pos, int vid) {
      if (lane0()) (pos ? keep_pos : keep_neg)[vid] = 1;
    };
    const bool one_pos = sum == 2 || (sum == 1 && nzero == 2);
    const bool one_neg = sum == -2 || (sum == -1 && nzero == 2);
    if (one_pos || one_neg) {
      const int sg = one_pos ? 1 : -1;
      if (sum == sg) {
        int k = s[0] != 0 ? 0 : (s[1] != 0 ? 1 : 2);
        int k1 = (k + 1) % 3, k2 = (k + 2) % 3;
        int b1, b2;
        if (sg > 0) {
          b1 = vertex_point(R, id[k1]);
          b2 = vertex_point(R, id[k2]);
        } else {
          b2 = vertex_point(R, id[k2]);
          b1 = vertex_point(R, id[k1]);
        }
        if (b1 != b2) {
          if (lane0()) {
            if (sg > 0) add_bedge(R, b1 + 1, b2 + 1);
            else add_bedge(R, b2 + 1, b1 + 1);
          }
          emit(sg > 0, id[k], bref(b1), bref(b2));
          keep(sg > 0, id[k]);
        }
      } else {
        int z = s[0] == 0 ? 0 : (s[1] == 0 ? 1 : 2);
        int bz = vertex_point(R, id[z]);
        if (z == 2) emit(sg > 0, id[0], id[1], bref(bz));
        else if (z == 0) emit(sg > 0, id[1], id[2], bref(bz));
        else emit(sg > 0, id[0], bref(bz), id[2]);
        for (int k = 0; k < 3; ++k)
          if (k != z) keep(sg > 0, id[k]);
      }
    } else {
      const double* pi[3] = {ch_pi + 9 * cc, ch_pi + 9 * cc + 3, ch_pi + 9 * cc + 6};
      const int fl = ch_f[cc];
      const bool f[3] = {(fl & 1) != 0, (fl & 2) != 0, (fl & 4) != 0};
      int e = -1;
      if (f[0] && f[1] && !f[2]) e = 0;
      else if (f[1] && f[2] && !f[0]) e = 1;
      else if (f[2] && f[0] && !f[1]) e = 2;
      if (e >= 0) {
        const int a = e, vv = (e + 1) % 3, c = (e + 2) % 3;
        edge_point(R, id[a], id[vv], pi[a]);
        edge_point(R, id[vv], id[c], pi[vv]);
        int fa = 0, fv = 0;
        if (lane0()) {
          fa = edge_get(R, id[a], id[vv]);
          fv = edge_get(R, id[vv], id[c]);
        }
        fa = __shfl_sync(0xffffffffu, fa, 0);
        fv = __shfl_sync(0xffffffffu, fv, 0);
        const bool apex_pos = s[vv] == 1;
        if (fv != fa) {
          if (lane0()) {
            if (apex_pos) add_bedge(R, fv + 1, fa + 1);
            else add_bedge(R, fa + 1, fv + 1);
          }
          keep(apex_pos, id[vv]);
          keep(!apex_pos, id[a]);
          keep(!apex_pos, id[c]);
          emit(apex_pos, id[vv], bref(fv), bref(fa));
          if (e == 0) {
            emit(!apex_pos, id[a], bref(fa), bref(fv));
            emit(!apex_pos, bref(fv), id[c], id[a]);
          } else {
            emit(!apex_pos, id[c], bref(fa), bref(fv));
            emit(!apex_pos, bref(fa), id[c], id[a]);
          }
        } else {
          keep(!apex_pos, id[a]);
          keep(!apex_pos, id[c]);
          emit(!apex_pos, e == 0 ? bref(fv) : bref(fa), id[c], id[a]);
        }
      } else if (f[0] && f[1] && f[2]) {
        const bool all_nz = s[0] != 0 && s[1] != 0 && s[2] != 0;
        auto same = [](const double* x, const double* y) {
          const double eps = (double)1e-5f;
          return fabs(ds(x[0], y[0])) < eps && fabs(ds(x[1], y[1])) < eps && fabs(ds(x[2], y[2])) < eps;
        };
        int k = -1;
        if (s[0] == 0 || (all_nz && same(pi[0], pi[2]))) k = 0;
        else if (s[1] == 0 || (all_nz && same(pi[0], pi[1]))) k = 1;
        else if (s[2] == 0 || (all_nz && same(pi[1], pi[2]))) k = 2;
        if (k >= 0) {
          const int k1 = (k + 1) % 3, k2 = (k + 2) % 3;
          const int bk = vertex_point(R, id[k]);
          if (lane0()) {
            edge_set(R, id[k], id[k1], bk);
            edge_set(R, id[k1], id[k], bk);
            edge_set(R, id[k2], id[k], bk);
            edge_set(R, id[k], id[k2], bk);
          }
          __syncwarp();
          edge_point(R, id[k1], id[k2], pi[k1]);
          int fo = lane0() ? edge_get(R, id[k1], id[k2]) : 0;
          fo = __shfl_sync(0xffffffffu, fo, 0);
          const int test = (k == 0) ? s[1] : s[0];
          const int u = (k == 1) ? k2 : k1;
          const int other = (k == 1) ? k1 : k2;
          int A, Bp;
          if (k == 1) { A = bk; Bp = fo; } else { A = fo; Bp = bk; }
          if (A != Bp) {
            if (lane0()) {
              if (test == 1) add_bedge(R, A + 1, Bp + 1);
              else add_bedge(R, Bp + 1, A + 1);
            }
            keep(test == 1, id[u]);
            keep(test != 1, id[other]);
            emit(test == 1, id[u], bref(A), bref(Bp));
            emit(test != 1, id[other], bref(Bp), bref(A));
          }
        }
      }
    }
    if (lane0()) slots[li] = out;
    __syncwarp();
  }
  if (smem) {
    const unsigned nb = sm_cnt[0];
    for (unsigned i = lane; i < 3 * nb; i += 32) global_border[i] = sm_border[i];
    if (lane == 0) {
      R.cnt->n_border = nb;
      R.cnt->n_bedges = sm_cnt[1];
    }
  }
}

// ---- the resolver: first requests, near pairs, numbering (one CTA) ----------
// Up to kParTouch touching triangles (two requests each). What bounds it is
// latency: about a dozen block-wide steps and one pass over all pairs of first
// requests in FP32 (FP64 only decides the pairs within 1e-4 and its rounding).
// A body of 8,000 vertices with 354 touching triangles: 0.041 ms, 0.855 ms as
// the ordered walk (about 2.4 us a triangle: hash probes, a position scan and
// the table updates form one dependent chain). The ordered walk stays for what
// this form cannot express: an overwritten edge point, and tables beyond the
// shared memory of one SM.
constexpr int kParTouch = 2048;
constexpr int kParReq = 2 * kParTouch;
constexpr int kParHash = 2 * kParReq;  // load factor at most 1/2
constexpr int kParNear = 4096;
struct ParShared {
  unsigned long long key[kParHash];
  int val[kParHash];              // first request of the key, later its number
  int list[kParTouch];            // touching triangles, in order
  unsigned short slot[kParReq];   // hash slot of each request, 0xffff none
  float fx[kParReq], fy[kParReq], fz[kParReq];  // positions of the first requests, in order
  unsigned short seq[kParReq];    // their requests
  int alias[kParReq];             // smallest kept near predecessor
  int bidx[kParReq];              // border point
  unsigned near[kParNear];        // near pairs (later << 16 | earlier)
  unsigned char state[kParReq];   // 0 undecided, 1 kept, 2 dropped
  unsigned char wait[kParReq];    // a near predecessor is undecided
  unsigned wsum[kClipResolveThreads / 32];
  unsigned n_near;
};
constexpr size_t kClipSmem = sizeof(ParShared) > kResolveSmem ? sizeof(ParShared) : kResolveSmem;
static_assert(kClipSmem <= 227 * 1024, "shared memory of one CTA");
constexpr unsigned long long kNoKey = ~0ull;
constexpr int kNoAlias = 0x7fffffff;

// Exclusive prefix of one count per thread, and the block's total.
__device__ __forceinline__ unsigned block_prefix(unsigned c, unsigned* wsum, unsigned& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned x = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();  // wsum may still be read
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  unsigned before = 0;
  total = 0;
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
    const unsigned s = wsum[w];
    if (w < warp) before += s;
    total += s;
  }
  return before + x - c;
}

__device__ __forceinline__ unsigned hash64(unsigned long long k) {
  return hash2((int)(unsigned)(k >> 32), (int)(unsigned)k);
}

// Slot of key k, inserted if new (the table never fills).
__device__ __forceinline__ int par_insert(ParShared& S, unsigned long long k) {
  unsigned h = hash64(k) & (kParHash - 1);
  for (int probe = 0; probe < kParHash; ++probe, h = (h + 1) & (kParHash - 1)) {
    const unsigned long long old = atomicCAS(&S.key[h], kNoKey, k);
    if (old == kNoKey || old == k) return (int)h;
  }
  return 0;
}

// Request q (0 or 1) of a touching triangle: its key (vertex, or unordered
// edge) and where its position is; false when there is none.
__device__ __forceinline__ bool par_request(const ClipTouch* __restrict__ touch, const int* __restrict__ t,
                                            const double* __restrict__ v, int tri, int q, unsigned long long& key,
                                            const double*& pos) {
  const ClipTouch& r = touch[tri];
  const int kind = r.kind, a = r.a;
  const int* id = t + 3 * (int64_t)tri;
  if (kind == kTouchCross) {
    const int e = q == 0 ? a : (a + 1) % 3;
    const unsigned x = (unsigned)id[e], y = (unsigned)id[(e + 1) % 3];
    key = ((unsigned long long)min(x, y) << 32) | max(x, y);
    pos = r.pi[q];
    return true;
  }
  int k;
  if (kind == kTouchOneOff) k = (a + 1 + (r.pos ? q : 1 - q)) % 3;  // pos: a+1 then a+2; neg: the reverse
  else if (kind == kTouchTwoOff && q == 0) k = a;
  else return false;
  key = 0xffffffff00000000ull | (unsigned)id[k];
  pos = v + 3 * (int64_t)id[k];
  return true;
}

// All touching triangles in parallel. False when the ordered walk has to run.
__device__ __noinline__ bool resolve_parallel(ParShared& S, const double* __restrict__ v, const int* __restrict__ t,
                                              const ClipTouch* __restrict__ touch, int ntouch, Resolver R,
                                              PieceSlot* __restrict__ slots, unsigned char* __restrict__ keep_pos,
                                              unsigned char* __restrict__ keep_neg) {
  const int tid = threadIdx.x, nth = blockDim.x;
  bool special = false;
  for (int r = tid; r < ntouch; r += nth) special |= touch[S.list[r]].kind == kTouchVertex;
  for (int i = tid; i < kParHash; i += nth) {
    S.key[i] = kNoKey;
    S.val[i] = 0x7fffffff;
  }
  if (tid == 0) S.n_near = 0;
  if (__syncthreads_or(special)) return false;
  // First request of every key.
  const int nreq = 2 * ntouch;
  for (int i = tid; i < nreq; i += nth) {
    unsigned long long key;
    const double* pos;
    S.slot[i] = 0xffff;
    if (par_request(touch, t, v, S.list[i >> 1], i & 1, key, pos)) {
      const int h = par_insert(S, key);
      S.slot[i] = (unsigned short)h;
      atomicMin(&S.val[h], i);
    }
  }
  __syncthreads();
  // Numbered in request order (a contiguous run of requests per thread).
  const int per = (nreq + nth - 1) / nth;
  const int q0 = min(nreq, tid * per), q1 = min(nreq, q0 + per);
  unsigned c = 0, U;
  for (int i = q0; i < q1; ++i) c += S.slot[i] != 0xffff && S.val[S.slot[i]] == i;
  unsigned u = block_prefix(c, S.wsum, U);
  float big = 0.f;
  for (int i = q0; i < q1; ++i) {
    if (S.slot[i] == 0xffff || S.val[S.slot[i]] != i) continue;
    unsigned long long key;
    const double* pos;
    par_request(touch, t, v, S.list[i >> 1], i & 1, key, pos);
    const float x = (float)pos[0], y = (float)pos[1], z = (float)pos[2];
    S.fx[u] = x;
    S.fy[u] = y;
    S.fz[u] = z;
    big = fmaxf(big, fmaxf(fabsf(x), fmaxf(fabsf(y), fabsf(z))));
    S.seq[u] = (unsigned short)i;
    S.state[u] = 1;
    S.alias[u] = kNoAlias;
    ++u;
  }
  __syncthreads();
  // Keys take their numbers (each first request is its key's only writer).
  for (unsigned k = tid; k < U; k += nth) S.val[S.slot[S.seq[k]]] = (int)k;
  // FP32 filter: coordinates rounded to float are off by at most 2^-24 of the
  // largest each, the difference by as much again.
#pragma unroll
  for (int o = 16; o; o >>= 1) big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, o));
  if ((tid & 31) == 0) S.wsum[tid >> 5] = __float_as_uint(big);
  __syncthreads();
  for (int w = 0; w < (nth >> 5); ++w) big = fmaxf(big, __uint_as_float(S.wsum[w]));
  const float thr = 1.0001e-4f + big * 2.3841858e-7f;
  auto position = [&](unsigned k) {
    unsigned long long key;
    const double* pos = nullptr;
    const int i = S.seq[k];
    par_request(touch, t, v, S.list[i >> 1], i & 1, key, pos);
    return pos;
  };
  for (unsigned k = tid; k < U; k += nth) {
    const float x = S.fx[k], y = S.fy[k], z = S.fz[k];
    for (unsigned j = 0; j < k; ++j) {
      if (fabsf(S.fx[j] - x) > thr || fabsf(S.fy[j] - y) > thr || fabsf(S.fz[j] - z) > thr) continue;
      const double *p = position(k), *q = position(j);
      if (fabs(ds(q[0], p[0])) < 1e-4 && fabs(ds(q[1], p[1])) < 1e-4 && fabs(ds(q[2], p[2])) < 1e-4) {
        const unsigned at = atomicAdd(&S.n_near, 1u);
        if (at < kParNear) S.near[at] = (k << 16) | j;
      }
    }
  }
  __syncthreads();
  const unsigned nn = S.n_near;
  if (nn > kParNear) return false;
  // Keep-first: a request makes a point unless an earlier near one did. The
  // earliest undecided one decides in every round.
  if (nn) {
    for (unsigned i = tid; i < nn; i += nth) S.state[S.near[i] >> 16] = 0;
    __syncthreads();
    for (unsigned round = 0; round <= U; ++round) {
      for (unsigned k = tid; k < U; k += nth) {
        S.wait[k] = 0;
        S.alias[k] = kNoAlias;
      }
      __syncthreads();
      for (unsigned i = tid; i < nn; i += nth) {
        const unsigned k = S.near[i] >> 16, j = S.near[i] & 0xffffu;
        if (S.state[j] == 1) atomicMin(&S.alias[k], (int)j);
        else if (S.state[j] == 0) S.wait[k] = 1;
      }
      __syncthreads();
      int left = 0;
      for (unsigned k = tid; k < U; k += nth) {
        if (S.state[k]) continue;
        if (S.alias[k] != kNoAlias) S.state[k] = 2;
        else if (!S.wait[k]) S.state[k] = 1;
        else left = 1;
      }
      if (!__syncthreads_or(left)) break;
    }
    // Every state is settled: the smallest kept near predecessor.
    for (unsigned i = tid; i < nn; i += nth) {
      const unsigned k = S.near[i] >> 16, j = S.near[i] & 0xffffu;
      if (S.state[j] == 1) atomicMin(&S.alias[k], (int)j);
    }
    __syncthreads();
  }
  // Border points: the kept ones, in order.
  const unsigned uper = (U + nth - 1) / nth;
  const unsigned u0 = min(U, tid * uper), u1 = min(U, u0 + uper);
  c = 0;
  for (unsigned k = u0; k < u1; ++k) c += S.state[k] == 1;
  unsigned nb;
  unsigned b = block_prefix(c, S.wsum, nb);
  for (unsigned k = u0; k < u1; ++k) {
    if (S.state[k] != 1) continue;
    const double* p = position(k);
    R.border[3 * b] = p[0];
    R.border[3 * b + 1] = p[1];
    R.border[3 * b + 2] = p[2];
    S.bidx[k] = (int)b++;
  }
  __syncthreads();
  for (unsigned k = tid; k < U; k += nth)
    if (S.state[k] == 2) S.bidx[k] = S.bidx[S.alias[k]];
  __syncthreads();
  int* value = reinterpret_cast<int*>(S.fx);  // border point of each request
  for (int i = tid; i < nreq; i += nth) value[i] = S.slot[i] == 0xffff ? -1 : S.bidx[S.val[S.slot[i]]];
  __syncthreads();
  for (int i = tid; i < kParHash; i += nth) {
    S.key[i] = kNoKey;
    S.val[i] = 0x7fffffff;
  }
  __syncthreads();
  // Pieces, kept vertices and the border edge of every triangle.
  int2* edge = reinterpret_cast<int2*>(S.alias);  // kParTouch entries (alias and bidx are done)
  static_assert(sizeof(S.alias) >= sizeof(int2) * kParTouch, "edge table");
  for (int r = tid; r < ntouch; r += nth) {
    const int tri = S.list[r];
    const ClipTouch& tr = touch[tri];
    const int kind = tr.kind, a = tr.a;
    const bool pos = tr.pos != 0;
    const int id[3] = {t[3 * (int64_t)tri], t[3 * (int64_t)tri + 1], t[3 * (int64_t)tri + 2]};
    PieceSlot out;
    out.npos = out.nneg = 0;
    int2 be = make_int2(0, 0);
    auto emit = [&](bool p, int x, int y, int z) {
      int* o = p ? out.pos[out.npos++] : out.neg[out.nneg++];
      o[0] = x;
      o[1] = y;
      o[2] = z;
    };
    auto keep = [&](bool p, int vid) { (p ? keep_pos : keep_neg)[vid] = 1; };
    const int v0 = value[2 * r], v1 = value[2 * r + 1];
    if (kind == kTouchOneOff) {
      // Requests run a+1, a+2 on the positive side and a+2, a+1 on the other.
      const int b1 = pos ? v0 : v1, b2 = pos ? v1 : v0;
      if (b1 != b2) {
        be = pos ? make_int2(b1 + 1, b2 + 1) : make_int2(b2 + 1, b1 + 1);
        emit(pos, id[a], bref(b1), bref(b2));
        keep(pos, id[a]);
      }
    } else if (kind == kTouchTwoOff) {
      if (a == 2) emit(pos, id[0], id[1], bref(v0));
      else if (a == 0) emit(pos, id[1], id[2], bref(v0));
      else emit(pos, id[0], bref(v0), id[2]);
      for (int k = 0; k < 3; ++k)
        if (k != a) keep(pos, id[k]);
    } else if (kind == kTouchCross) {
      const int vv = (a + 1) % 3, cc = (a + 2) % 3;
      const int fa = v0, fv = v1;
      if (fv != fa) {
        be = pos ? make_int2(fv + 1, fa + 1) : make_int2(fa + 1, fv + 1);
        keep(pos, id[vv]);
        keep(!pos, id[a]);
        keep(!pos, id[cc]);
        emit(pos, id[vv], bref(fv), bref(fa));
        if (a == 0) {
          emit(!pos, id[a], bref(fa), bref(fv));
          emit(!pos, bref(fv), id[cc], id[a]);
        } else {
          emit(!pos, id[cc], bref(fa), bref(fv));
          emit(!pos, bref(fa), id[cc], id[a]);
        }
      } else {
        keep(!pos, id[a]);
        keep(!pos, id[cc]);
        emit(!pos, a == 0 ? bref(fv) : bref(fa), id[cc], id[a]);
      }
    }
    slots[r] = out;
    edge[r] = be;
    if (be.x) {
      const int h =
          par_insert(S, ((unsigned long long)(unsigned)min(be.x, be.y) << 32) | (unsigned)max(be.x, be.y));
      S.slot[r] = (unsigned short)h;
      atomicMin(&S.val[h], r);
    }
  }
  __syncthreads();
  const int tper = (ntouch + nth - 1) / nth;
  const int r0 = min(ntouch, tid * tper), r1 = min(ntouch, r0 + tper);
  c = 0;
  for (int r = r0; r < r1; ++r) c += edge[r].x && S.val[S.slot[r]] == r;
  unsigned ne;
  unsigned at = block_prefix(c, S.wsum, ne);
  for (int r = r0; r < r1; ++r)
    if (edge[r].x && S.val[S.slot[r]] == r) R.bedge[at++] = edge[r];
  if (tid == 0) {
    R.cnt->n_border = nb;
    R.cnt->n_bedges = ne;
  }
  return true;
}

__global__ void __launch_bounds__(kClipResolveThreads) clip_resolve_kernel(
    const double* __restrict__ v, const int* __restrict__ t, int nt, const double* __restrict__ plp,
    const unsigned char* __restrict__ code, const ClipTouch* __restrict__ touch, Resolver R, int* __restrict__ list,
    int* __restrict__ tslot, PieceSlot* __restrict__ slots, unsigned char* __restrict__ keep_pos,
    unsigned char* __restrict__ keep_neg) {
  extern __shared__ __align__(16) unsigned char rsm[];
  ParShared& S = *reinterpret_cast<ParShared*>(rsm);
  // The touching triangles in order: every thread a contiguous run of codes,
  // sixteen at a time (the code array is padded to a multiple of 16).
  const int runs = (nt + 15) / 16, per = (runs + (int)blockDim.x - 1) / (int)blockDim.x;
  const int g0 = min(runs, (int)threadIdx.x * per), g1 = min(runs, g0 + per);
  auto touching = [&](int g, unsigned& m) {
    const uint4 w = reinterpret_cast<const uint4*>(code)[g];
    const unsigned x[4] = {w.x, w.y, w.z, w.w};
    m = 0;
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (((x[k >> 2] >> (8 * (k & 3))) & 0xffu) == 2u && 16 * g + k < nt) m |= 1u << k;
  };
  unsigned c = 0, m, total;
  for (int g = g0; g < g1; ++g) {
    touching(g, m);
    c += __popc(m);
  }
  unsigned at = block_prefix(c, S.wsum, total);
  const int ntouch = (int)total;
  for (int g = g0; g < g1; ++g) {
    touching(g, m);
    for (; m; m &= m - 1) {
      const int i = 16 * g + __ffs(m) - 1;
      list[at] = i;
      tslot[i] = (int)at;
      if (at < kParTouch) S.list[at] = i;
      ++at;
    }
  }
  if (threadIdx.x == 0) R.cnt->n_touch = total;
  __syncthreads();
  if (ntouch <= kParTouch && resolve_parallel(S, v, t, touch, ntouch, R, slots, keep_pos, keep_neg)) return;
  __syncthreads();
  ordered_tables(R, t, list, ntouch);
  __syncthreads();
  if (threadIdx.x < 32) resolve_ordered(v, t, plp, list, ntouch, R, slots, keep_pos, keep_neg);
}

// ---- outputs ------------------------------------------------------------------
// Three launches (tile sums, vertex maps, triangles); each tile adds up the
// sums before it itself, which for the few hundred tiles of a large mesh is
// cheaper than a launch. The four separate scans this replaced took 14
// launches: the call's other kernels went from 0.13 to 0.046 ms on the body
// above, and the whole call from 1.09 to 0.27 ms (Python side included).
constexpr int kOutThreads = 256;
constexpr int kOutItems = 4;
constexpr int kOutTile = kOutThreads * kOutItems;

// (pos, neg) output triangles of triangle i, packed in one word each.
__device__ __forceinline__ unsigned long long tri_counts(const unsigned char* __restrict__ code,
                                                         const int* __restrict__ tslot,
                                                         const PieceSlot* __restrict__ slots, int i) {
  const unsigned char c = code[i];
  if (c == 0) return 1ull;
  if (c == 1) return 1ull << 32;
  const PieceSlot& s = slots[tslot[i]];
  return (unsigned long long)(unsigned)s.npos | ((unsigned long long)(unsigned)s.nneg << 32);
}
__device__ __forceinline__ unsigned long long keep_counts(const unsigned char* __restrict__ kpos,
                                                          const unsigned char* __restrict__ kneg, int i) {
  return (unsigned long long)kpos[i] | ((unsigned long long)kneg[i] << 32);
}

// Exclusive prefix over the block of one packed pair of counts per thread.
__device__ __forceinline__ unsigned long long out_prefix(unsigned long long c, unsigned long long& total) {
  __shared__ unsigned long long ws[kOutThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long x = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();
  if (lane == 31) ws[warp] = x;
  __syncthreads();
  unsigned long long before = 0;
  total = 0;
#pragma unroll
  for (int w = 0; w < kOutThreads / 32; ++w) {
    if (w < warp) before += ws[w];
    total += ws[w];
  }
  return before + x - c;
}
// Sum of the tile sums before tile `upto`.
__device__ __forceinline__ unsigned long long tiles_before(const unsigned long long* __restrict__ sums, int upto) {
  unsigned long long s = 0, total;
  for (int k = threadIdx.x; k < upto; k += kOutThreads) s += sums[k];
  out_prefix(s, total);
  return total;
}

// Output counts of every tile of 1024 triangles, then of every tile of 1024
// vertices (halves of 64 bits: pos low, neg high).
__global__ void __launch_bounds__(kOutThreads) clip_sums_kernel(
    const unsigned char* __restrict__ code, const int* __restrict__ tslot, const PieceSlot* __restrict__ slots, int nt,
    int tri_tiles, const unsigned char* __restrict__ kpos, const unsigned char* __restrict__ kneg, int nv,
    unsigned long long* __restrict__ tri_sums, unsigned long long* __restrict__ vert_sums) {
  const bool tri = (int)blockIdx.x < tri_tiles;
  const int tile = tri ? blockIdx.x : blockIdx.x - tri_tiles;
  unsigned long long c = 0, total;
  for (int k = 0; k < kOutItems; ++k) {
    const int64_t i = (int64_t)tile * kOutTile + k * kOutThreads + threadIdx.x;
    if (i < (tri ? nt : nv)) c += tri ? tri_counts(code, tslot, slots, (int)i) : keep_counts(kpos, kneg, (int)i);
  }
  out_prefix(c, total);
  if (threadIdx.x == 0) (tri ? tri_sums : vert_sums)[tile] = total;
}

// 1-based maps (0 = absent) and the kept vertices of each side.
__global__ void __launch_bounds__(kOutThreads) clip_maps_kernel(
    const unsigned char* __restrict__ kpos, const unsigned char* __restrict__ kneg, int nv, int vert_tiles,
    const unsigned long long* __restrict__ vert_sums, int* __restrict__ map_pos, int* __restrict__ map_neg,
    ClipCounters* __restrict__ cnt) {
  unsigned long long at = tiles_before(vert_sums, blockIdx.x), own[kOutItems], c = 0, total;
  const int64_t i0 = (int64_t)blockIdx.x * kOutTile + (int64_t)threadIdx.x * kOutItems;
#pragma unroll
  for (int k = 0; k < kOutItems; ++k) {
    own[k] = i0 + k < nv ? keep_counts(kpos, kneg, (int)(i0 + k)) : 0ull;
    c += own[k];
  }
  unsigned long long x = at + out_prefix(c, total);
#pragma unroll
  for (int k = 0; k < kOutItems; ++k) {
    if (i0 + k < nv) {
      map_pos[i0 + k] = (unsigned)own[k] ? (int)(unsigned)x + 1 : 0;
      map_neg[i0 + k] = own[k] >> 32 ? (int)(x >> 32) + 1 : 0;
    }
    x += own[k];
  }
  if ((int)blockIdx.x == vert_tiles - 1 && threadIdx.x == 0) {
    cnt->nv_pos = (unsigned)(at + total);
    cnt->nv_neg = (unsigned)((at + total) >> 32);
  }
}

// Scatter + remap: original vertex -> map - 1, border point b -> n_side + b.
__global__ void __launch_bounds__(kOutThreads) clip_scatter_kernel(
    const int* __restrict__ t, const unsigned char* __restrict__ code, const int* __restrict__ tslot,
    const PieceSlot* __restrict__ slots, int nt, int tri_tiles, const unsigned long long* __restrict__ tri_sums,
    const int* __restrict__ map_pos, const int* __restrict__ map_neg, int* __restrict__ out_pos,
    int* __restrict__ out_neg, ClipCounters* __restrict__ cnt) {
  const int npos_v = (int)cnt->nv_pos, nneg_v = (int)cnt->nv_neg;
  const unsigned long long at = tiles_before(tri_sums, blockIdx.x);
  unsigned long long own[kOutItems], c = 0, total;
  const int64_t i0 = (int64_t)blockIdx.x * kOutTile + (int64_t)threadIdx.x * kOutItems;
#pragma unroll
  for (int k = 0; k < kOutItems; ++k) {
    own[k] = i0 + k < nt ? tri_counts(code, tslot, slots, (int)(i0 + k)) : 0ull;
    c += own[k];
  }
  unsigned long long x = at + out_prefix(c, total);
  auto rp = [&](int w) { return w >= 0 ? map_pos[w] - 1 : npos_v + (-w - 1); };
  auto rn = [&](int w) { return w >= 0 ? map_neg[w] - 1 : nneg_v + (-w - 1); };
#pragma unroll
  for (int k = 0; k < kOutItems; ++k) {
    const int64_t i = i0 + k;
    if (i < nt) {
      const unsigned char cd = code[i];
      int* op = out_pos + 3 * (int64_t)(unsigned)x;
      int* on = out_neg + 3 * (int64_t)(x >> 32);
      if (cd == 0) {
        op[0] = rp(t[3 * i]);
        op[1] = rp(t[3 * i + 1]);
        op[2] = rp(t[3 * i + 2]);
      } else if (cd == 1) {
        on[0] = rn(t[3 * i]);
        on[1] = rn(t[3 * i + 1]);
        on[2] = rn(t[3 * i + 2]);
      } else {
        const PieceSlot& s = slots[tslot[i]];
        for (int q = 0; q < s.npos; ++q)
          for (int a = 0; a < 3; ++a) op[3 * q + a] = rp(s.pos[q][a]);
        for (int q = 0; q < s.nneg; ++q)
          for (int a = 0; a < 3; ++a) on[3 * q + a] = rn(s.neg[q][a]);
      }
    }
    x += own[k];
  }
  if ((int)blockIdx.x == tri_tiles - 1 && threadIdx.x == 0) {
    cnt->n_pos = (unsigned)(at + total);
    cnt->n_neg = (unsigned)((at + total) >> 32);
  }
}

}  // namespace vgpu

using namespace vgpu;

static size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

extern "C" int visacd_clip(visacd_ctx* ctx, const double* verts, int32_t nv, const int32_t* tris,
                           int32_t nt, const double* plane, visacd_clip_result* res) {
  VCHECK(ctx && res && plane, VISACD_ERR_INVALID_ARG, "visacd_clip: null argument");
  VCHECK(nv >= 0 && nt >= 0 && (nv == 0 || verts) && (nt == 0 || tris), VISACD_ERR_INVALID_ARG,
         "visacd_clip: bad mesh");
  memset(res, 0, sizeof(*res));
  if (nt == 0 || nv == 0) return VISACD_OK;
  VCHECK(indices_in_range(tris, 3LL * nt, nv), VISACD_ERR_INVALID_ARG, "visacd_clip: triangle index out of range");
  VCUDA(cudaSetDevice(ctx->device));
  // Border points are bounded by the touching triangles (3 each).
  const int max_border = 3 * nt + 16;
  int ecap = 64;
  while (ecap < 8 * max_border) ecap <<= 1;
  int bcap = 64;
  while (bcap < 4 * max_border) bcap <<= 1;
  const int tri_tiles = (nt + kOutTile - 1) / kOutTile, vert_tiles = (nv + kOutTile - 1) / kOutTile;
  size_t off = 0;
  auto carve = [&](size_t b) { size_t o = off; off += align256(b); return o; };
  // The uploaded block (one copy), the zeroed block (one memset), the rest.
  const size_t o_pl = carve(32), o_v = carve((size_t)nv * 24), o_t = carve((size_t)nt * 12);
  const size_t upload = off;
  const size_t o_kp = carve(nv), o_kn = carve(nv), o_cnt = carve(sizeof(ClipCounters));
  const size_t zero_end = off;
  const size_t o_code = carve(((size_t)nt + 15) & ~size_t(15)), o_touch = carve((size_t)nt * sizeof(ClipTouch)),
               o_list = carve((size_t)nt * 4), o_tslot = carve((size_t)nt * 4),
               o_border = carve((size_t)max_border * 24), o_vmap = carve((size_t)nv * 4),
               o_ek = carve((size_t)ecap * 8), o_ev = carve((size_t)ecap * 4),
               o_be = carve((size_t)max_border * 8), o_bk = carve((size_t)bcap * 8),
               o_slots = carve((size_t)nt * sizeof(PieceSlot)), o_ts = carve((size_t)tri_tiles * 8),
               o_vs = carve((size_t)vert_tiles * 8), o_outp = carve((size_t)nt * 3 * 12),
               o_outn = carve((size_t)nt * 3 * 12), o_mapp = carve((size_t)nv * 4), o_mapn = carve((size_t)nv * 4);
  VTRY(ensure_slot(ctx, kSlotClip, off));
  char* B = slot<char>(ctx, kSlotClip);
  double* dv = (double*)(B + o_v);
  int* dt = (int*)(B + o_t);
  double* dpl = (double*)(B + o_pl);
  unsigned char* code = (unsigned char*)(B + o_code);
  ClipTouch* touch = (ClipTouch*)(B + o_touch);
  int *list = (int*)(B + o_list), *tslot = (int*)(B + o_tslot);
  unsigned char *kp = (unsigned char*)(B + o_kp), *kn = (unsigned char*)(B + o_kn);
  ClipCounters* cnt = (ClipCounters*)(B + o_cnt);
  Resolver R;
  R.v = dv;
  R.border = (double*)(B + o_border);
  R.vmap = (int*)(B + o_vmap);
  R.ekeys = (int*)(B + o_ek);
  R.evals = (int*)(B + o_ev);
  R.ecap = ecap;
  R.bedge = (int2*)(B + o_be);
  R.bkeys = (int*)(B + o_bk);
  R.bcap = bcap;
  R.max_border = max_border;
  R.cnt = cnt;
  R.n_border = &cnt->n_border;
  R.n_bedges = &cnt->n_bedges;
  PieceSlot* slots = (PieceSlot*)(B + o_slots);
  unsigned long long *ts = (unsigned long long*)(B + o_ts), *vs = (unsigned long long*)(B + o_vs);
  int *outp = (int*)(B + o_outp), *outn = (int*)(B + o_outn), *mapp = (int*)(B + o_mapp),
      *mapn = (int*)(B + o_mapn);
  cudaStream_t st = ctx->stream;
  Stager up(ctx);
  VTRY(up.reserve(upload, 1));
  std::memcpy(up.host() + o_pl, plane, 32);
  std::memcpy(up.host() + o_v, verts, (size_t)nv * 24);
  std::memcpy(up.host() + o_t, tris, (size_t)nt * 12);
  VTRY(up.copy(B, upload));
  VCUDA(cudaMemsetAsync(B + o_kp, 0, zero_end - o_kp, st));
  VLAUNCH(ctx, kKClip, grid_for(nt, 64, 32LL * ctx->sm_count), 64, 0, clip_classify_kernel, dv, dt, nt, dpl, code,
          touch, kp, kn);
  VCUDA(cudaFuncSetAttribute(clip_resolve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClipSmem));
  VLAUNCH(ctx, kKClipResolve, 1, kClipResolveThreads, kClipSmem, clip_resolve_kernel, dv, dt, nt, dpl, code,
          touch, R, list, tslot, slots, kp, kn);
  VLAUNCH(ctx, kKClip, (unsigned)(tri_tiles + vert_tiles), kOutThreads, 0, clip_sums_kernel, code, tslot, slots, nt,
          tri_tiles, kp, kn, nv, ts, vs);
  VLAUNCH(ctx, kKClip, (unsigned)vert_tiles, kOutThreads, 0, clip_maps_kernel, kp, kn, nv, vert_tiles, vs, mapp,
          mapn, cnt);
  VLAUNCH(ctx, kKClip, (unsigned)tri_tiles, kOutThreads, 0, clip_scatter_kernel, dt, code, tslot, slots, nt,
          tri_tiles, ts, mapp, mapn, outp, outn, cnt);
  // Counts back to the host.
  ClipCounters* h = nullptr;
  VTRY(pinned(ctx, sizeof(ClipCounters), (void**)&h));
  VCUDA(cudaMemcpyAsync(h, cnt, sizeof(ClipCounters), cudaMemcpyDeviceToHost, st));
  VCUDA(stream_wait(ctx));
  VCHECK(!h->overflow, VISACD_ERR_CAPACITY, "visacd_clip: internal table overflow");
  ctx->clip_out.n_pos = (int32_t)h->n_pos;
  ctx->clip_out.n_neg = (int32_t)h->n_neg;
  ctx->clip_out.nv_pos = (int32_t)h->nv_pos;
  ctx->clip_out.nv_neg = (int32_t)h->nv_neg;
  ctx->clip_out.n_border = (int32_t)h->n_border;
  ctx->clip_out.n_border_edges = (int32_t)h->n_bedges;
  ctx->clip_out.n_touching = (int32_t)h->n_touch;
  ctx->clip_nv = nv;
  ctx->clip_ptrs[0] = outp;
  ctx->clip_ptrs[1] = outn;
  ctx->clip_ptrs[2] = mapp;
  ctx->clip_ptrs[3] = mapn;
  ctx->clip_ptrs[4] = R.border;
  ctx->clip_ptrs[5] = R.bedge;
  *res = ctx->clip_out;
  return VISACD_OK;
}

extern "C" int visacd_clip_fetch(visacd_ctx* ctx, int32_t* pos_tris, int32_t* neg_tris,
                                 int32_t* pos_map, int32_t* neg_map, double* border,
                                 int32_t* border_edges) {
  VCHECK(ctx, VISACD_ERR_INVALID_ARG, "visacd_clip_fetch: null context");
  const visacd_clip_result& r = ctx->clip_out;
  void* const dst[6] = {pos_tris, neg_tris, pos_map, neg_map, border, border_edges};
  const void* const src[6] = {ctx->clip_ptrs[0], ctx->clip_ptrs[1], ctx->clip_ptrs[2],
                              ctx->clip_ptrs[3], ctx->clip_ptrs[4], ctx->clip_ptrs[5]};
  const size_t bytes[6] = {(size_t)r.n_pos * 12, (size_t)r.n_neg * 12,    (size_t)ctx->clip_nv * 4,
                           (size_t)ctx->clip_nv * 4, (size_t)r.n_border * 24, (size_t)r.n_border_edges * 8};
  return fetch(ctx, 6, dst, src, bytes);
}
