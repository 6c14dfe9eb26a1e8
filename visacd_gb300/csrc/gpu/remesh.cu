// SDF remeshing on the GPU: the iso-surface at distance `level` outside a
// mesh, on a grid of voxel size 1/scale — the cage / manifold step that
// replaces OpenVDB in lib/src/preprocess.cpp:18-67.
//
// Same algorithm and arithmetic as the host restatement (manifold_preprocess in
// csrc/host/remesh.cpp), so the output mesh is identical bit for bit:
//  1. sdf_tri_prep_kernel computes each triangle's set-up once (voxel box, ray
//     boxes, FP32 bounds and planes).
//  2. Crossings: sdf_cross_kernel marks, for every ray along an axis through
//     voxel centres (offset by 1.2345679e-6 / 2.3456789e-6 voxels) that crosses
//     a triangle at x, the first voxel whose centre lies beyond x (one toggle
//     bit per axis); sdf_parity_yz_kernel and sdf_inside_kernel run the prefix
//     parities along the rays. Inside = at least two of the three odd.
//  3. Distances: sdf_ub_kernel gives the voxels that matter an FP32 upper
//     bound of their distance, then sdf_dist_kernel the exact FP64
//     point-triangle distance (rounded to float) unless a lower bound rules
//     the triangle out, combined with atomicMin (non-negative floats order
//     like their bit patterns). The boxes are cut into work items of 256
//     voxels. Which voxels matter: see class_cut.
//  4. Surface nets: a vertex per sign-changing cell at the mean of its edge
//     crossings (cells in linear order, exclusive scan), two triangles per
//     sign-changing grid edge whose four cells all have vertices (voxels in
//     linear order, x / y / z edges, exclusive scan).
#include "common.cuh"
#include "geom64.cuh"

namespace vgpu {

namespace {

constexpr float kSdfU = 5.9604645e-8f;  // 2^-24

struct SdfGrid {
  int org[3], dim[3];
  double band;
  float fiso;
  double scale;
  float margin;  // FP32 lower-bound margin (voxels): 1e-3 + 1e-6 max |grid coordinate|
  float cut_out, low_out;  // outside voxels need their exact distance between these (class_cut)
  double reach;            // the voxel boxes of triangles are grown by this
};

// The output depends on a voxel's exact distance d only where a grid edge
// joins a voxel with f < iso to one with f >= iso (f = -d for inside voxels, d
// otherwise); elsewhere only the side counts. So with iso > 0:
//  * a voxel next to one of the other class needs it (kClassEdge);
//  * any other inside voxel does not: its neighbours are inside, f <= 0 < iso;
//  * any other outside voxel needs it for iso - 1 <= d < iso + 1, since the
//    distances of neighbours differ by at most 1: below, its neighbours are
//    all on the f < iso side, above all on the other.
// Elsewhere a voxel keeps the band or its upper bound, both on the right side.
// So boxes grown by cut_out instead of the band find every distance that is
// needed, but those of kClassEdge voxels farther out (a mesh that is not closed):
// sdf_far_kernel marks these kClassFar and sdf_far_dist_kernel, which does
// nothing without them, goes over the boxes grown by the band.
//
// Thin triangles (SdfTri::thin): the exact formula's closest point may lie off the
// triangle, or be NaN, and what it gives is the result. So they bound nothing, and the
// above holds for the other triangles alone; the thin ones are evaluated at every voxel
// of their boxes grown by the band that is not on its side already (inside and no
// kClassEdge, or an upper bound below iso - 1). What they bring below iso may have a
// neighbour whose other distances were not needed: sdf_far_kernel marks that too.
enum : uint8_t { kClassOut = 0, kClassIn = 1, kClassEdge = 2, kClassFar = 4 };
__device__ __forceinline__ float class_cut(const SdfGrid& g, uint8_t c) {
  return (c & kClassEdge) ? 3.0e38f : ((c & kClassIn) ? 0.f : g.cut_out);
}

__device__ __forceinline__ size_t vid(const SdfGrid& g, int i, int j, int k) {
  return ((size_t)k * g.dim[1] + j) * g.dim[0] + i;
}

__device__ __forceinline__ void load_tri(const double* __restrict__ P, const int32_t* __restrict__ T, int t,
                                         double (&A)[3], double (&B)[3], double (&C)[3]) {
  const int a = T[3 * (size_t)t], b = T[3 * (size_t)t + 1], c = T[3 * (size_t)t + 2];
  for (int k = 0; k < 3; ++k) {
    A[k] = P[3 * (size_t)a + k];
    B[k] = P[3 * (size_t)b + k];
    C[k] = P[3 * (size_t)c + k];
  }
}

__device__ __forceinline__ double min3(double a, double b, double c) { return fmin(fmin(a, b), c); }
__device__ __forceinline__ double max3(double a, double b, double c) { return fmax(fmax(a, b), c); }

// The rays a triangle covers: its box projected on the grid plane.
__device__ __forceinline__ bool ray_box(const double (&A)[3], const double (&B)[3], const double (&C)[3],
                                        const SdfGrid& g, int u, int w, int& u0, int& w0, int& eu, int& ew) {
  u0 = max(0, (int)floor(min3(A[u], B[u], C[u]) - g.org[u]));
  const int u1 = min(g.dim[u] - 1, (int)ceil(max3(A[u], B[u], C[u]) - g.org[u]));
  w0 = max(0, (int)floor(min3(A[w], B[w], C[w]) - g.org[w]));
  const int w1 = min(g.dim[w] - 1, (int)ceil(max3(A[w], B[w], C[w]) - g.org[w]));
  eu = u1 - u0 + 1;
  ew = w1 - w0 + 1;
  return eu > 0 && ew > 0;
}

// Lower-bound pre-filter of the exact distance: a voxel whose lower bound
// (FP32, less twice a margin of 1e-3 voxel plus 1e-6 of the largest grid
// coordinate, which covers the FP32 rounding of the plane evaluations) is not
// below the voxel's current minimum cannot lower it — the exact FP64 distance
// is at least as large, and rounding to float is monotone — so its FP64
// evaluation is skipped. The stored result is the same minimum as without the
// filter. The bound is the larger of the gap to the triangle's bounding box
// and sqrt(p^2 + s^2), with p the distance to the triangle's plane and s the
// largest distance beyond one of its edges in the plane: with n the unit
// normal and m_e the unit in-plane normal of edge e pointing away from the
// triangle (offset so that no vertex lies beyond it), every triangle point x
// has |q - x|^2 >= (n.(q - x))^2 + (m_e.(q - x))^2 >= p^2 + s_e^2.
// Per-triangle set-up of the distances (one thread per triangle, once): the
// voxel box grown by the reach, the vertices in FP32, the FP32 bounding box, and the FP32 plane
// and edge planes of the lower bound.
struct SdfTri {
  int lo[3], ext[3];      // voxel box (ext[0] <= 0: nothing in the grid)
  float blo[3], bhi[3];   // bounding box rounded outwards
  float4 pl;              // unit normal, offset; w of fe[0] = -1e30 without a plane
  float4 fe[3];           // unit in-plane edge normals, offsets (no vertex beyond)
  int has_plane, thin, pad[2];
  int ray[3][4];          // per axis: first ray and extents over (u, w); extents 0: none
  float v[3][3], vabs;    // vertices in FP32, their largest coordinate
  int pad2[2];
};

// What the passes share beside the voxels.
struct SdfFlags {
  unsigned n_wide;  // listed triangles of sdf_cross_wide_kernel
  unsigned n_far;   // whether sdf_far_dist_kernel has work
  unsigned thin;    // whether a triangle is thin
  unsigned pad;
};

// Box voxels per work item of the distance passes (one warp); fewer where all of them
// take the exact formula.
constexpr int kSdfChunk = 256, kSdfThinChunk = 32;

__device__ __forceinline__ void box_range(const SdfGrid& g, int a, double mn, double mx, double by, int& lo, int& ext) {
  lo = max(0, (int)floor(mn - by) - g.org[a]);
  ext = min(g.dim[a] - 1, (int)ceil(mx + by) - g.org[a]) - lo + 1;
}

__global__ void sdf_tri_prep_kernel(const double* __restrict__ P, const int32_t* __restrict__ T, int nt, SdfGrid g,
                                    SdfTri* __restrict__ out, uint32_t* __restrict__ chunks,
                                    SdfFlags* __restrict__ flags) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nt; t += gridDim.x * blockDim.x) {
    double A[3], B[3], C[3];
    load_tri(P, T, t, A, B, C);
    SdfTri r;
    // unit normal and plane offset (FP32 copies; degenerate triangles get none)
    const double ux = B[0] - A[0], uy = B[1] - A[1], uz = B[2] - A[2];
    const double vx = C[0] - A[0], vy = C[1] - A[1], vz = C[2] - A[2];
    double nx = uy * vz - uz * vy, ny = uz * vx - ux * vz, nz = ux * vy - uy * vx;
    const double nl = sqrt(nx * nx + ny * ny + nz * nz);
    r.has_plane = nl > 1e-12;
    // Thin: the exact formula's closest point may be off by 1e-3 voxels or lie outside
    // (its weights are quotients of products of this size, with an error of some 1e-14
    // of L^2 (L + band)^2), or be NaN.
    const double wx = C[0] - B[0], wy = C[1] - B[1], wz = C[2] - B[2];
    const double l2 = fmax(fmax(ux * ux + uy * uy + uz * uz, vx * vx + vy * vy + vz * vz), wx * wx + wy * wy + wz * wz);
    const double len = sqrt(l2), reachable = len + g.band;
    r.thin = !(nl * nl >= 1e-11 * l2 * len * reachable * reachable);
    if (r.thin) flags->thin = 1u;
    for (int a = 0; a < 3; ++a) {
      const double mn = min3(A[a], B[a], C[a]), mx = max3(A[a], B[a], C[a]);
      box_range(g, a, mn, mx, r.thin ? g.band : g.reach, r.lo[a], r.ext[a]);
      r.blo[a] = __double2float_rd(mn);
      r.bhi[a] = __double2float_ru(mx);
    }
    if (r.ext[0] <= 0 || r.ext[1] <= 0 || r.ext[2] <= 0) r.ext[0] = 0;
    r.pl = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int e = 0; e < 3; ++e) r.fe[e] = make_float4(0.f, 0.f, 0.f, -1e30f);
    if (r.has_plane) {
      nx /= nl;
      ny /= nl;
      nz /= nl;
      r.pl = make_float4((float)nx, (float)ny, (float)nz, (float)-(nx * A[0] + ny * A[1] + nz * A[2]));
      const double* V[3] = {A, B, C};
      for (int e = 0; e < 3; ++e) {
        const double* P0 = V[e];
        const double* P1 = V[(e + 1) % 3];
        const double* P2 = V[(e + 2) % 3];
        const double ex = P1[0] - P0[0], ey = P1[1] - P0[1], ez = P1[2] - P0[2];
        double mx = ny * ez - nz * ey, my = nz * ex - nx * ez, mz = nx * ey - ny * ex;
        const double ml = sqrt(mx * mx + my * my + mz * mz);
        if (!(ml > 1e-12)) continue;
        mx /= ml;
        my /= ml;
        mz /= ml;
        if (mx * (P2[0] - P0[0]) + my * (P2[1] - P0[1]) + mz * (P2[2] - P0[2]) > 0) {
          mx = -mx;
          my = -my;
          mz = -mz;
        }
        const double top = fmax(fmax(mx * A[0] + my * A[1] + mz * A[2], mx * B[0] + my * B[1] + mz * B[2]),
                                mx * C[0] + my * C[1] + mz * C[2]);
        r.fe[e] = make_float4((float)mx, (float)my, (float)mz, (float)-top);
      }
    }
    for (int ax = 0; ax < 3; ++ax) {
      const int u = (ax + 1) % 3, w = (ax + 2) % 3;
      int eu, ew;
      if (!ray_box(A, B, C, g, u, w, r.ray[ax][0], r.ray[ax][1], eu, ew)) eu = ew = 0;
      r.ray[ax][2] = eu;
      r.ray[ax][3] = ew;
    }
    r.vabs = 0.f;
    for (int a = 0; a < 3; ++a) {
      r.v[0][a] = (float)A[a];
      r.v[1][a] = (float)B[a];
      r.v[2][a] = (float)C[a];
      r.vabs = fmaxf(r.vabs, fmaxf(fabsf(r.v[0][a]), fmaxf(fabsf(r.v[1][a]), fabsf(r.v[2][a]))));
    }
    out[t] = r;
    const int chunk = r.thin ? kSdfThinChunk : kSdfChunk;
    chunks[t] = r.ext[0] > 0 ? (uint32_t)((r.ext[0] * r.ext[1] * r.ext[2] + chunk - 1) / chunk) : 0u;
  }
}

// Work items of the distance passes: (triangle, chunk of kSdfChunk voxels of
// its box), numbered by the scanned chunk counts. Each warp takes a contiguous
// range of items, so a triangle with a large box (the long triangles of a
// clipped part's cap) is spread over many warps instead of holding one while
// the rest of the grid idles.
struct SdfItems {
  const uint64_t* off;  // nt + 1 scanned chunk counts
  int nt;
};

__device__ __forceinline__ void item_range(const SdfItems& W, long long& w0, long long& w1) {
  const long long total = (long long)W.off[W.nt];
  const long long warps = ((long long)gridDim.x * blockDim.x) >> 5;
  const long long per = (total + warps - 1) / warps;
  w0 = (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * per;
  w1 = min(total, w0 + per);
}

// Position of a lane in a box walked 32 voxels at a time, x fastest: stepped
// with carries, as three divisions per voxel cost more than the bounds.
struct BoxWalk {
  int i, j, k, e0, e1, si, sj, sk;
  __device__ __forceinline__ BoxWalk(const int (&ext)[3], int q) : e0(ext[0]), e1(ext[1]) {
    i = q % e0;
    j = (q / e0) % e1;
    k = q / (e0 * e1);
    si = 32 % e0;
    sj = (32 / e0) % e1;
    sk = 32 / (e0 * e1);
  }
  __device__ __forceinline__ void step() {
    i += si;
    const int ci = i >= e0;
    i -= ci ? e0 : 0;
    j += sj + ci;
    const int cj = j >= e1;
    j -= cj ? e1 : 0;
    k += sk + cj;
  }
};

// Triangle of item w (off[t] <= w < off[t + 1]).
__device__ __forceinline__ int item_triangle(const SdfItems& W, long long w) {
  int lo = 0, hi = W.nt;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if ((long long)W.off[mid] <= w) lo = mid;
    else hi = mid;
  }
  return lo;
}

// FP32 upper bound of the distance from q to triangle (A, B, C): the distance
// to a point of the triangle chosen in FP32 by the closest-point regions
// (Ericson, Real-Time Collision Detection 5.1.5), taken as A + v AB + w AC
// with v, w clamped to v, w >= 0, v + w <= 1 so that the exact point with
// these weights lies on the triangle; `slack` covers the FP32 rounding of the
// point and of the distance.
__device__ float tri_dist_ub32(float qx, float qy, float qz, const float (&A)[3], const float (&B)[3],
                               const float (&C)[3], float slack) {
  const float ab[3] = {B[0] - A[0], B[1] - A[1], B[2] - A[2]};
  const float ac[3] = {C[0] - A[0], C[1] - A[1], C[2] - A[2]};
  const float ap[3] = {qx - A[0], qy - A[1], qz - A[2]};
  const float bp[3] = {qx - B[0], qy - B[1], qz - B[2]};
  const float cp[3] = {qx - C[0], qy - C[1], qz - C[2]};
  auto dot = [](const float (&x)[3], const float (&y)[3]) { return x[0] * y[0] + x[1] * y[1] + x[2] * y[2]; };
  const float d1 = dot(ab, ap), d2 = dot(ac, ap), d3 = dot(ab, bp), d4 = dot(ac, bp), d5 = dot(ab, cp),
              d6 = dot(ac, cp);
  float v = 0.f, w = 0.f;
  const float vc = d1 * d4 - d3 * d2, vb = d5 * d2 - d1 * d6, va = d3 * d6 - d5 * d4;
  if (d1 <= 0.f && d2 <= 0.f) {
  } else if (d3 >= 0.f && d4 <= d3) {
    v = 1.f;
  } else if (vc <= 0.f && d1 >= 0.f && d3 <= 0.f) {
    v = d1 / (d1 - d3);
  } else if (d6 >= 0.f && d5 <= d6) {
    w = 1.f;
  } else if (vb <= 0.f && d2 >= 0.f && d6 <= 0.f) {
    w = d2 / (d2 - d6);
  } else if (va <= 0.f && (d4 - d3) >= 0.f && (d5 - d6) >= 0.f) {
    w = (d4 - d3) / ((d4 - d3) + (d5 - d6));
    v = 1.f - w;
  } else {
    const float den = 1.f / (va + vb + vc);
    v = vb * den;
    w = vc * den;
  }
  v = fminf(fmaxf(v, 0.f), 1.f);  // NaN (degenerate triangle) becomes 0
  w = fminf(fmaxf(w, 0.f), 1.f - v);
  const float px = A[0] + v * ab[0] + w * ac[0], py = A[1] + v * ab[1] + w * ac[1], pz = A[2] + v * ab[2] + w * ac[2];
  const float ex = qx - px, ey = qy - py, ez = qz - pz;
  return __fadd_ru(__fmul_ru(__fsqrt_ru(__fadd_ru(__fadd_ru(__fmul_ru(ex, ex), __fmul_ru(ey, ey)), __fmul_ru(ez, ez))),
                             1.0f + 1.0f / 65536.0f),
                   slack);
}

// FP32 band voxel bound between the triangle's lower bound and its FP32 upper
// bound (first pass): ub[v] ends at or above the voxel's exact distance, so
// the exact pass can skip every triangle whose lower bound reaches it.
__device__ __forceinline__ float sdf_lower_bound(const SdfTri& r, float qx, float qy, float qz) {
  const float gx = fmaxf(fmaxf(r.blo[0] - qx, qx - r.bhi[0]), 0.f);
  const float gy = fmaxf(fmaxf(r.blo[1] - qy, qy - r.bhi[1]), 0.f);
  const float gz = fmaxf(fmaxf(r.blo[2] - qz, qz - r.bhi[2]), 0.f);
  float lb = sqrtf(gx * gx + gy * gy + gz * gz);
  if (r.has_plane) {
    const float pd = fabsf(r.pl.x * qx + r.pl.y * qy + r.pl.z * qz + r.pl.w);
    float se = 0.f;
    for (int e = 0; e < 3; ++e) se = fmaxf(se, r.fe[e].x * qx + r.fe[e].y * qy + r.fe[e].z * qz + r.fe[e].w);
    lb = fmaxf(lb, sqrtf(pd * pd + se * se));
  }
  return lb;
}

__global__ void __launch_bounds__(128) sdf_ub_kernel(SdfItems W, SdfGrid g, const SdfTri* __restrict__ prep,
                                                     const uint8_t* __restrict__ cls, uint32_t* __restrict__ ub) {
  const int lane = threadIdx.x & 31;
  long long w0, w1;
  item_range(W, w0, w1);
  int t = w0 < w1 ? item_triangle(W, w0) : 0;
  for (long long w = w0; w < w1; ++w) {
    while ((long long)W.off[t + 1] <= w) ++t;
    const SdfTri& r = prep[t];
    if (r.thin) continue;
    // rounding of the vertices to float, of the chosen point and of its
    // distance: a few units of 2^-24 of the largest coordinate involved
    const int n = r.ext[0] * r.ext[1] * r.ext[2];
    const int c0 = (int)(w - (long long)W.off[t]) * kSdfChunk, c1 = min(n, c0 + kSdfChunk);
    BoxWalk at(r.ext, c0 + lane);
    for (int q0 = c0 + lane; q0 < c1; q0 += 32, at.step()) {
      const int i = r.lo[0] + at.i, j = r.lo[1] + at.j, k = r.lo[2] + at.k;
      const size_t v = vid(g, i, j, k);
      const float cut = class_cut(g, cls[v]);
      if (cut <= 0.f) continue;
      const float qx = (float)(g.org[0] + i), qy = (float)(g.org[1] + j), qz = (float)(g.org[2] + k);
      const float lb = sdf_lower_bound(r, qx, qy, qz);
      const float cur = fminf(cut, __uint_as_float(*(volatile const uint32_t*)&ub[v]));
      if (lb - 2.0f * g.margin >= cur) continue;
      const float qa = fmaxf(fabsf(qx), fmaxf(fabsf(qy), fabsf(qz)));
      const float slack = 64.0f * kSdfU * fmaxf(r.vabs, qa) + g.margin;
      atomicMin(&ub[v], __float_as_uint(tri_dist_ub32(qx, qy, qz, r.v[0], r.v[1], r.v[2], slack)));
    }
  }
}

// Resident blocks per SM of the two passes, and their grids: one wave, since every
// warp has its share of the items from the start (with 8 blocks per SM of which 5
// are resident, 1.6 waves, the exact pass took 24 us more).
constexpr int kDistBlocks = 6, kUbBlocks = 9;

// The (triangle, voxel) pairs that the lower bound leaves, kept per warp over
// all of its items and evaluated in FP64 32 at a time: the FP64 pipe, slow on
// this part, runs with full warps, and no warp waits for another. 20,480
// triangles, 740,000 voxels: with a list per block and barriers around it, boxes
// grown by the band and three divisions per voxel this pass took 383 us and the
// FP32 one 212; with the queue, cut_out and BoxWalk 158 and 83.
struct PairQueue {
  int t[64];
  uint32_t v[64];
};

// Appends the lanes' pairs (keep) to n and evaluates 32 when there are as many,
// or what is left (flush).
__device__ __forceinline__ void queue_pairs(PairQueue& Q, int& n, bool keep, int t, uint32_t v, bool flush,
                                            const double* __restrict__ P, const int32_t* __restrict__ T,
                                            const SdfGrid& g, uint32_t* __restrict__ dist) {
  const int lane = threadIdx.x & 31;
  const unsigned m = __ballot_sync(0xffffffffu, keep);
  if (keep) {
    const int at = n + __popc(m & ((1u << lane) - 1u));
    Q.t[at] = t;
    Q.v[at] = v;
  }
  n += __popc(m);
  while (n >= 32 || (flush && n > 0)) {
    __syncwarp();
    const int first = n > 32 ? n - 32 : 0;
    if (first + lane < n) {
      const uint32_t e = Q.v[first + lane];
      double A[3], B[3], C[3];
      load_tri(P, T, Q.t[first + lane], A, B, C);
      const int i = (int)(e % g.dim[0]), j = (int)((e / g.dim[0]) % g.dim[1]),
                k = (int)(e / ((uint32_t)g.dim[0] * g.dim[1]));
      const double q[3] = {(double)(g.org[0] + i), (double)(g.org[1] + j), (double)(g.org[2] + k)};
      atomicMin(&dist[e], __float_as_uint(__double2float_rn(point_tri_dist(q, A, B, C))));
    }
    n = first;
    __syncwarp();
  }
}

__global__ void __launch_bounds__(128, kDistBlocks) sdf_dist_kernel(const double* __restrict__ P, const int32_t* __restrict__ T,
                                                       SdfItems W, SdfGrid g, const SdfTri* __restrict__ prep,
                                                       const uint8_t* __restrict__ cls, const uint32_t* __restrict__ ub,
                                                       uint32_t* __restrict__ dist) {
  __shared__ PairQueue queues[4];
  PairQueue& Q = queues[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  int nq = 0;
  long long w0, w1;
  item_range(W, w0, w1);
  int t = w0 < w1 ? item_triangle(W, w0) : 0;
  for (long long w = w0; w < w1; ++w) {
    while ((long long)W.off[t + 1] <= w) ++t;
    const SdfTri& r = prep[t];
    const int n = r.ext[0] * r.ext[1] * r.ext[2];
    const int chunk = r.thin ? kSdfThinChunk : kSdfChunk;
    const int c0 = (int)(w - (long long)W.off[t]) * chunk, c1 = min(n, c0 + chunk);
    BoxWalk at(r.ext, c0 + lane);
    for (int base = c0; base < c1; base += 32, at.step()) {
      bool keep = false;
      size_t v = 0;
      if (base + lane < c1) {
        const int i = r.lo[0] + at.i, j = r.lo[1] + at.j, k = r.lo[2] + at.k;
        v = vid(g, i, j, k);
        const uint8_t c = cls[v];
        const float up = __uint_as_float(ub[v]);
        float cur = fminf(up, class_cut(g, c));
        // an outside voxel whose upper bound is this low has no neighbour on
        // the other side
        if (c == kClassOut && up < g.low_out) cur = 0.f;
        if (cur > 0.f) {
          const float lb = r.thin ? -3.0e38f
                                  : sdf_lower_bound(r, (float)(g.org[0] + i), (float)(g.org[1] + j),
                                                    (float)(g.org[2] + k));
          keep = lb - 2.0f * g.margin < fminf(cur, __uint_as_float(*(volatile const uint32_t*)&dist[v]));
        }
      }
      queue_pairs(Q, nq, keep, t, (uint32_t)v, w == w1 - 1 && base + 32 >= c1, P, T, g, dist);
    }
  }
}

__global__ void sdf_far_kernel(SdfGrid g, size_t n, const uint32_t* __restrict__ dist, const uint32_t* __restrict__ ub,
                               uint8_t* __restrict__ cls, SdfFlags* __restrict__ flags) {
  const bool thin = flags->thin != 0;
  const size_t sy = g.dim[0], sz = (size_t)g.dim[0] * g.dim[1];
  auto field = [&](size_t v) { return fminf(__uint_as_float(dist[v]), __uint_as_float(ub[v])); };
  for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (size_t)gridDim.x * blockDim.x) {
    const uint8_t c = cls[v];
    if (!(c & kClassEdge) && !(thin && c == kClassOut)) continue;
    if ((double)field(v) < g.reach) continue;
    if (!(c & kClassEdge)) {  // (its neighbours are outside too)
      const int i = (int)(v % sy), j = (int)(v / sy % g.dim[1]), k = (int)(v / sz);
      if (!((i > 0 && field(v - 1) < g.fiso) || (i + 1 < g.dim[0] && field(v + 1) < g.fiso) ||
            (j > 0 && field(v - sy) < g.fiso) || (j + 1 < g.dim[1] && field(v + sy) < g.fiso) ||
            (k > 0 && field(v - sz) < g.fiso) || (k + 1 < g.dim[2] && field(v + sz) < g.fiso)))
        continue;
    }
    cls[v] = c | kClassFar;
    flags->n_far = 1u;
  }
}

// Exact distances of the kClassFar voxels. The box grown by the band is at most two
// voxels longer an axis than the one of the work items: a triangle of few items is
// one warp's, the box of a larger one is shared out over its items. (With a warp per
// triangle the distance passes of an open box, ten faces of 200 x 200 voxels, took
// 7.0 ms, 0.78 so. Runs of items for the small triangles too took 5 to 10 % of the
// call more on a bowl: a warp's triangles then lie together, and so do the voxels.)
constexpr int kFarRun = 8, kFarWhole = 16;
__global__ void __launch_bounds__(128, kDistBlocks)
    sdf_far_dist_kernel(const double* __restrict__ P, const int32_t* __restrict__ T, SdfItems W, SdfGrid g,
                        const SdfTri* __restrict__ prep, const uint8_t* __restrict__ cls,
                        const unsigned* __restrict__ n_far, uint32_t* __restrict__ dist) {
  __shared__ PairQueue queues[4];
  PairQueue& Q = queues[threadIdx.x >> 5];
  if (*n_far == 0) return;
  const int lane = threadIdx.x & 31, warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5),
            warps = (int)((gridDim.x * blockDim.x) >> 5);
  int nq = 0;
  // Items a to b (of `items`) of triangle t's box.
  auto part = [&](int t, long long a, long long b, long long items) {
    double A[3], B[3], C[3];
    load_tri(P, T, t, A, B, C);
    int lo[3], ext[3];
#pragma unroll
    for (int x = 0; x < 3; ++x)
      box_range(g, x, min3(A[x], B[x], C[x]), max3(A[x], B[x], C[x]), g.band, lo[x], ext[x]);
    const SdfTri& r = prep[t];
    if (r.thin || ext[0] <= 0 || ext[1] <= 0 || ext[2] <= 0) return;
    const long long n = ext[0] * ext[1] * ext[2];
    const int c0 = (int)(n * a / items), c1 = (int)(n * b / items);
    BoxWalk at(ext, c0 + lane);
    for (int base = c0; base < c1; base += 32, at.step()) {
      bool keep = false;
      size_t v = 0;
      if (base + lane < c1) {
        const int i = lo[0] + at.i, j = lo[1] + at.j, k = lo[2] + at.k;
        v = vid(g, i, j, k);
        if (cls[v] & kClassFar) {
          const float lb = sdf_lower_bound(r, (float)(g.org[0] + i), (float)(g.org[1] + j), (float)(g.org[2] + k));
          keep = lb - 2.0f * g.margin < __uint_as_float(*(volatile const uint32_t*)&dist[v]);
        }
      }
      // (a triangle's pairs are not kept waiting: what they find spares others)
      queue_pairs(Q, nq, keep, t, (uint32_t)v, base + 32 >= c1, P, T, g, dist);
    }
  };
  // Pass 0: the small triangles; pass 1: runs of items, those of large ones.
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    const long long total = pass ? (long long)W.off[W.nt] : W.nt;
    const int run = pass ? kFarRun : 1;
    for (long long w0 = (long long)warp * run; w0 < total; w0 += (long long)warps * run) {
      const long long w1 = min(w0 + run, total);
      int t = pass ? item_triangle(W, w0) : (int)w0;
      for (long long w = w0; w < w1; ++t) {
        const long long first = (long long)W.off[t], last = (long long)W.off[t + 1];
        const long long a = pass ? w : first, b = pass ? min(w1, last) : last;
        w = pass ? b : w1;
        if (a < b && (last - first > kFarWhole) == (pass == 1)) part(t, a - first, b - first, last - first);
      }
    }
  }
}

// Crossings of rays (grid column (ku, kw) along axis ax) with triangles. What an
// FP32 form of the three orientations cannot rule out is kept per warp and
// evaluated in FP64 32 at a time, as in PairQueue.
struct RayQueue {
  int t[64], ku[64], kw[64];
};

// Crossing of one ray with triangle t: toggles the first voxel whose centre lies
// beyond the crossing. Component 0, 1, 2 of the vertices: along u, w, ax.
__device__ __forceinline__ void cross_ray(const double* __restrict__ P, const int32_t* __restrict__ T, int t,
                                          const SdfGrid& g, int ax, int u, int w, int ku, int kw,
                                          uint32_t* __restrict__ toggle) {
  double V[3][3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double* v = P + 3 * (int64_t)T[3 * (size_t)t + k];
    V[k][0] = v[u];
    V[k][1] = v[w];
    V[k][2] = v[ax];
  }
  const double(&A)[3] = V[0], (&B)[3] = V[1], (&C)[3] = V[2];
  const double ou = 1.2345679e-6, ow = 2.3456789e-6;
  const double y = da((double)(g.org[u] + ku), ou), z = da((double)(g.org[w] + kw), ow);
  const double e0 = ds(dm(ds(B[0], A[0]), ds(z, A[1])), dm(ds(B[1], A[1]), ds(y, A[0])));
  const double e1 = ds(dm(ds(C[0], B[0]), ds(z, B[1])), dm(ds(C[1], B[1]), ds(y, B[0])));
  const double e2 = ds(dm(ds(A[0], C[0]), ds(z, C[1])), dm(ds(A[1], C[1]), ds(y, C[0])));
  const bool in = (e0 > 0 && e1 > 0 && e2 > 0) || (e0 < 0 && e1 < 0 && e2 < 0);
  if (!in) return;
  const double sw = da(da(e0, e1), e2);
  const double x = __ddiv_rn(da(da(dm(e1, A[2]), dm(e2, B[2])), dm(e0, C[2])), sw);
  // first voxel s whose centre org + s lies beyond x (integers compare exactly)
  const int org = g.org[ax], dim = g.dim[ax];
  int s = (int)floor(x - (double)org) + 1;
  while (s > 0 && (double)(org + s - 1) > x) --s;
  while (s < dim && !((double)(org + s) > x)) ++s;
  if (s < 0) s = 0;
  if (s >= dim) return;
  const int gi = ax == 0 ? s : (u == 0 ? ku : kw), gj = ax == 1 ? s : (u == 1 ? ku : kw),
            gk = ax == 2 ? s : (u == 2 ? ku : kw);
  atomicXor(&toggle[vid(g, gi, gj, gk)], 1u << ax);
}

// False when two of the orientations certainly have different signs. Coordinates
// are off by at most c (rounding to FP32, and the rays' offsets), differences of
// one triangle's box by twice that; the products' own rounding is far below m's
// second term.
__device__ __forceinline__ bool ray_may_cross(const SdfTri& r, const SdfGrid& g, int u, int w, int eu, int ew, int ku,
                                              int kw) {
  const float y = (float)(g.org[u] + ku), z = (float)(g.org[w] + kw);
  const float Au = r.v[0][u], Aw = r.v[0][w], Bu = r.v[1][u], Bw = r.v[1][w], Cu = r.v[2][u], Cw = r.v[2][w];
  const float c = 8.0f * kSdfU * (r.vabs + fabsf(y) + fabsf(z)) + 5e-6f;
  const float m = 8.0f * c * (float)(eu + ew + 2) + 1e-6f * (float)(eu + 1) * (float)(ew + 1);
  const float e0 = (Bu - Au) * (z - Aw) - (Bw - Aw) * (y - Au);
  const float e1 = (Cu - Bu) * (z - Bw) - (Cw - Bw) * (y - Bu);
  const float e2 = (Au - Cu) * (z - Cw) - (Aw - Cw) * (y - Cu);
  return !((e0 < -m || e1 < -m || e2 < -m) && (e0 > m || e1 > m || e2 > m));
}

__device__ __forceinline__ void queue_rays(RayQueue& Q, int& n, bool keep, int t, int ku, int kw, bool flush,
                                           const double* __restrict__ P, const int32_t* __restrict__ T,
                                           const SdfGrid& g, int ax, int u, int w, uint32_t* __restrict__ toggle) {
  const int lane = threadIdx.x & 31;
  const unsigned m = __ballot_sync(0xffffffffu, keep);
  if (keep) {
    const int at = n + __popc(m & ((1u << lane) - 1u));
    Q.t[at] = t;
    Q.ku[at] = ku;
    Q.kw[at] = kw;
  }
  n += __popc(m);
  while (n >= 32 || (flush && n > 0)) {
    __syncwarp();
    const int first = n > 32 ? n - 32 : 0;
    if (first + lane < n)
      cross_ray(P, T, Q.t[first + lane], g, ax, u, w, Q.ku[first + lane], Q.kw[first + lane], toggle);
    n = first;
    __syncwarp();
  }
}

// Triangles covering at most kCrossSmall rays (nearly all): kCrossLanes lanes
// each, over its rays, blockIdx.y the axis. Larger ones (the long triangles of
// clipped parts' caps, big faces) are listed with their axis and take one block
// each (sdf_cross_wide_kernel). All three axes in one launch with one bit each,
// and the parities' rays next to each other in x, took crossings and votes of
// 20,480 triangles on 740,000 voxels from 321 to 116 us; of that 82 were this
// kernel with every ray in FP64 in its own lane, and are 49 now.
constexpr int kCrossSmall = 32;
constexpr int kCrossLanes = 8;

__global__ void __launch_bounds__(128) sdf_cross_kernel(const double* __restrict__ P, const int32_t* __restrict__ T,
                                                        int nt, SdfGrid g, const SdfTri* __restrict__ prep,
                                                        uint32_t* __restrict__ toggle, int* __restrict__ wide,
                                                        unsigned* __restrict__ n_wide) {
  __shared__ RayQueue queues[4];
  RayQueue& Q = queues[threadIdx.x >> 5];
  const int ax = blockIdx.y, u = (ax + 1) % 3, w = (ax + 2) % 3;
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  const int sub = gid % kCrossLanes;
  const int groups = (gridDim.x * blockDim.x) / kCrossLanes;
  int nq = 0;
  for (int t0 = (gid - (int)(threadIdx.x & 31)) / kCrossLanes; t0 < nt; t0 += groups) {  // the warp's first triangle
    const int t = t0 + (int)(threadIdx.x & 31) / kCrossLanes;
    int4 r = make_int4(0, 0, 0, 0);
    if (t < nt) r = *reinterpret_cast<const int4*>(prep[t].ray[ax]);
    int n = r.z * r.w;
    if (n > kCrossSmall) {
      if (sub == 0) wide[atomicAdd(n_wide, 1u)] = 3 * t + ax;
      n = 0;
    }
    const int most = __reduce_max_sync(0xffffffffu, n);
    for (int q0 = 0; q0 < most; q0 += kCrossLanes) {
      const int q = q0 + sub;
      int ku = 0, kw = 0;
      bool keep = false;
      if (q < n) {
        kw = r.y + q / r.z;
        ku = r.x + q % r.z;
        keep = ray_may_cross(prep[t], g, u, w, r.z, r.w, ku, kw);
      }
      queue_rays(Q, nq, keep, t, ku, kw, false, P, T, g, ax, u, w, toggle);
    }
  }
  queue_rays(Q, nq, false, 0, 0, 0, true, P, T, g, ax, u, w, toggle);
}

__global__ void __launch_bounds__(128) sdf_cross_wide_kernel(const double* __restrict__ P,
                                                             const int32_t* __restrict__ T, SdfGrid g,
                                                             const SdfTri* __restrict__ prep,
                                                             const int* __restrict__ wide,
                                                             const unsigned* __restrict__ n_wide,
                                                             uint32_t* __restrict__ toggle) {
  __shared__ RayQueue queues[4];
  RayQueue& Q = queues[threadIdx.x >> 5];
  const int nw = (int)*n_wide;
  for (int k = blockIdx.x; k < nw; k += gridDim.x) {
    const int t = wide[k] / 3, ax = wide[k] % 3, u = (ax + 1) % 3, w = (ax + 2) % 3;
    const int4 r = *reinterpret_cast<const int4*>(prep[t].ray[ax]);
    const int n = r.z * r.w;
    int nq = 0;
    for (int q0 = 0; q0 < n; q0 += blockDim.x) {
      const int q = q0 + threadIdx.x;
      int ku = 0, kw = 0;
      bool keep = false;
      if (q < n) {
        kw = r.y + q / r.z;
        ku = r.x + q % r.z;
        keep = ray_may_cross(prep[t], g, u, w, r.z, r.w, ku, kw);
      }
      queue_rays(Q, nq, keep, t, ku, kw, q0 + (int)blockDim.x >= n, P, T, g, ax, u, w, toggle);
    }
  }
}

// Prefix parities along y (blockIdx.y 0) and z (1): one thread per ray, rays
// next to each other in x, eight loads in flight.
__global__ void __launch_bounds__(64) sdf_parity_yz_kernel(SdfGrid g, const uint32_t* __restrict__ toggle,
                                                           uint8_t* __restrict__ par_y, uint8_t* __restrict__ par_z) {
  const int ax = 1 + (int)blockIdx.y;
  const int ncol = g.dim[0] * (ax == 1 ? g.dim[2] : g.dim[1]), n = ax == 1 ? g.dim[1] : g.dim[2];
  const size_t stride = ax == 1 ? (size_t)g.dim[0] : (size_t)g.dim[0] * g.dim[1];
  uint8_t* out = ax == 1 ? par_y : par_z;
  for (int col = blockIdx.x * blockDim.x + threadIdx.x; col < ncol; col += gridDim.x * blockDim.x) {
    const int i = col % g.dim[0], o = col / g.dim[0];
    const size_t base = ax == 1 ? vid(g, i, 0, o) : vid(g, i, o, 0);
    uint32_t par = 0;
    for (int s = 0; s < n; s += 8) {
      uint32_t t[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) t[q] = s + q < n ? toggle[base + (size_t)(s + q) * stride] >> ax : 0u;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        par ^= t[q];
        if (s + q < n) out[base + (size_t)(s + q) * stride] = (uint8_t)(par & 1u);
      }
    }
  }
}

// Prefix parity along x (one warp per row, 32 voxels at a time by ballot) and
// the class of every voxel: inside when at least two parities are odd.
__global__ void __launch_bounds__(128) sdf_inside_kernel(SdfGrid g, const uint32_t* __restrict__ toggle,
                                                         const uint8_t* __restrict__ par_y,
                                                         const uint8_t* __restrict__ par_z,
                                                         uint8_t* __restrict__ inside) {
  const int lane = threadIdx.x & 31;
  const int rows = g.dim[1] * g.dim[2], warps = (gridDim.x * blockDim.x) >> 5;
  for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += warps) {
    const size_t base = (size_t)r * g.dim[0];
    uint32_t carry = 0;
    for (int i0 = 0; i0 < g.dim[0]; i0 += 32) {
      const int i = i0 + lane;
      const bool in_grid = i < g.dim[0];
      const unsigned m = __ballot_sync(0xffffffffu, in_grid && (toggle[base + i] & 1u));
      const uint32_t px = (carry + __popc(m & (0xffffffffu >> (31 - lane)))) & 1u;
      if (in_grid) inside[base + i] = px + par_y[base + i] + par_z[base + i] >= 2u ? kClassIn : kClassOut;
      carry += __popc(m);
    }
  }
}

// Marks voxels with a neighbour of the other class (all: every voxel, when
// the range of class_cut does not apply), and starts both distance arrays at the
// band.
__global__ void sdf_class_kernel(SdfGrid g, const uint8_t* __restrict__ inside, int all, uint32_t band,
                                 uint8_t* __restrict__ cls, uint32_t* __restrict__ ub, uint32_t* __restrict__ dist) {
  const size_t n = (size_t)g.dim[0] * g.dim[1] * g.dim[2];
  const size_t sy = g.dim[0], sz = (size_t)g.dim[0] * g.dim[1];
  for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(v % g.dim[0]), j = (int)((v / g.dim[0]) % g.dim[1]), k = (int)(v / sz);
    const uint8_t c = inside[v];
    const bool edge = all || (i > 0 && inside[v - 1] != c) || (i + 1 < g.dim[0] && inside[v + 1] != c) ||
                      (j > 0 && inside[v - sy] != c) || (j + 1 < g.dim[1] && inside[v + sy] != c) ||
                      (k > 0 && inside[v - sz] != c) || (k + 1 < g.dim[2] && inside[v + sz] != c);
    cls[v] = c | (edge ? kClassEdge : 0);
    ub[v] = band;
    dist[v] = band;
  }
}

// The field: the exact distance where it was needed (the upper bound is never
// below it), a value on its side elsewhere.
__global__ void sdf_field_kernel(const uint32_t* __restrict__ dist, const uint32_t* __restrict__ ub,
                                 const uint8_t* __restrict__ cls, size_t n, float* __restrict__ f) {
  for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (size_t)gridDim.x * blockDim.x) {
    const float d = fminf(__uint_as_float(dist[v]), __uint_as_float(ub[v]));
    f[v] = (cls[v] & kClassIn) ? -d : d;
  }
}

__constant__ int kCorner[8][3] = {{0, 0, 0}, {1, 0, 0}, {0, 1, 0}, {1, 1, 0},
                                  {0, 0, 1}, {1, 0, 1}, {0, 1, 1}, {1, 1, 1}};
__device__ __forceinline__ int corner_values(const SdfGrid& g, const float* __restrict__ f, int i, int j, int k,
                                             float (&cv)[8]) {
  int nin = 0;
  for (int c = 0; c < 8; ++c) {
    cv[c] = f[vid(g, i + kCorner[c][0], j + kCorner[c][1], k + kCorner[c][2])];
    nin += cv[c] < g.fiso;
  }
  return nin;
}

__global__ void sdf_cell_flag_kernel(SdfGrid g, const float* __restrict__ f, uint32_t* __restrict__ flag) {
  const int cx = g.dim[0] - 1, cy = g.dim[1] - 1, cz = g.dim[2] - 1;
  const size_t n = (size_t)cx * cy * cz;
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(c % cx), j = (int)((c / cx) % cy), k = (int)(c / ((size_t)cx * cy));
    float cv[8];
    const int nin = corner_values(g, f, i, j, k, cv);
    flag[c] = (nin != 0 && nin != 8) ? 1u : 0u;
  }
}

// Vertex number of every cell (-1: none) and the cells that have one, in order.
__global__ void sdf_cell_list_kernel(size_t n, const uint32_t* __restrict__ flag, const uint64_t* __restrict__ off,
                                     int32_t* __restrict__ cell_vertex, uint32_t* __restrict__ cells) {
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
    const bool has = flag[c] != 0;
    const int vtx = (int)off[c];
    cell_vertex[c] = has ? vtx : -1;
    if (has) cells[vtx] = (uint32_t)c;
  }
}

// One thread per vertex, over the list, so that FP64 runs with full warps: of
// the cells themselves only about one in twenty-five has a vertex, and the same
// arithmetic over all of 740,000 took 189 us; over the list, 23.
__global__ void __launch_bounds__(64) sdf_cell_vertex_kernel(SdfGrid g, const float* __restrict__ f,
                                                             const uint32_t* __restrict__ cells, size_t n,
                                                             double* __restrict__ out_v) {
  const int cx = g.dim[0] - 1, cy = g.dim[1] - 1;
  for (size_t vtx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; vtx < n; vtx += (size_t)gridDim.x * blockDim.x) {
    const size_t c = cells[vtx];
    const int i = (int)(c % cx), j = (int)((c / cx) % cy), k = (int)(c / ((size_t)cx * cy));
    float cv[8];
    corner_values(g, f, i, j, k, cv);
    double acc[3] = {0, 0, 0};
    int ncross = 0;
#pragma unroll
    for (int e = 0; e < 12; ++e) {
      // Edges 0-3 run along x, 4-7 along y, 8-11 along z, between corners numbered x + 2 y + 4 z.
      constexpr int kC[12][2] = {{0, 1}, {2, 3}, {4, 5}, {6, 7}, {0, 2}, {1, 3},
                                 {4, 6}, {5, 7}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};
      const int c0 = kC[e][0], c1 = kC[e][1];
      if ((cv[c0] < g.fiso) == (cv[c1] < g.fiso)) continue;
      const double t = __ddiv_rn((double)__fsub_rn(g.fiso, cv[c0]), (double)__fsub_rn(cv[c1], cv[c0]));
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const int s0 = (c0 >> a) & 1, s1 = (c1 >> a) & 1;
        acc[a] = da(acc[a], da((double)s0, dm(t, (double)(s1 - s0))));
      }
      ++ncross;
    }
    const int ijk[3] = {i, j, k};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double m = __ddiv_rn(acc[a], (double)ncross);
      out_v[3 * vtx + a] = __ddiv_rn(da((double)(g.org[a] + ijk[a]), m), g.scale);
    }
  }
}

// Quads of interior voxel (i, j, k) in the host's order (+x, +y, +z edges),
// each as two triangles; returns the triangle count, writes them when out.
__device__ __forceinline__ int voxel_quads(const SdfGrid& g, const float* __restrict__ f,
                                           const int32_t* __restrict__ cv, int i, int j, int k,
                                           int32_t* __restrict__ out) {
  const int cx = g.dim[0] - 1, cy = g.dim[1] - 1;
  auto cid = [&](int a, int b, int c) { return ((size_t)c * cy + b) * cx + a; };
  const bool in0 = f[vid(g, i, j, k)] < g.fiso;
  int n = 0;
  auto emit = [&](int q0, int q1, int q2, int q3, bool flip) {
    if (q0 < 0 || q1 < 0 || q2 < 0 || q3 < 0) return;
    if (flip) {
      const int t = q1;
      q1 = q3;
      q3 = t;
    }
    if (out) {
      out[3 * n] = q0;
      out[3 * n + 1] = q1;
      out[3 * n + 2] = q2;
      out[3 * n + 3] = q0;
      out[3 * n + 4] = q2;
      out[3 * n + 5] = q3;
    }
    n += 2;
  };
  if (in0 != (f[vid(g, i + 1, j, k)] < g.fiso))
    emit(cv[cid(i, j - 1, k - 1)], cv[cid(i, j, k - 1)], cv[cid(i, j, k)], cv[cid(i, j - 1, k)], !in0);
  if (in0 != (f[vid(g, i, j + 1, k)] < g.fiso))
    emit(cv[cid(i - 1, j, k - 1)], cv[cid(i - 1, j, k)], cv[cid(i, j, k)], cv[cid(i, j, k - 1)], !in0);
  if (in0 != (f[vid(g, i, j, k + 1)] < g.fiso))
    emit(cv[cid(i - 1, j - 1, k)], cv[cid(i, j - 1, k)], cv[cid(i, j, k)], cv[cid(i - 1, j, k)], !in0);
  return n;
}

__global__ void sdf_quad_kernel(SdfGrid g, const float* __restrict__ f, const int32_t* __restrict__ cell_vertex,
                                uint32_t* __restrict__ count, const uint64_t* __restrict__ off,
                                int32_t* __restrict__ out_t) {
  const int ix = g.dim[0] - 2, iy = g.dim[1] - 2, iz = g.dim[2] - 2;
  const size_t n = (size_t)ix * iy * iz;
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (size_t)gridDim.x * blockDim.x) {
    const int i = 1 + (int)(r % ix), j = 1 + (int)((r / ix) % iy), k = 1 + (int)(r / ((size_t)ix * iy));
    if (off)
      voxel_quads(g, f, cell_vertex, i, j, k, out_t + 3 * (size_t)off[r]);
    else
      count[r] = (uint32_t)voxel_quads(g, f, cell_vertex, i, j, k, nullptr);
  }
}

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

}  // namespace
}  // namespace vgpu

using namespace vgpu;

extern "C" int visacd_sdf_remesh(visacd_ctx* ctx, const double* verts, int32_t nv, const int32_t* tris, int32_t nt,
                                 double scale, double level, int32_t* out_nv, int32_t* out_nt) {
  VCHECK(ctx && out_nv && out_nt, VISACD_ERR_INVALID_ARG, "sdf_remesh: null argument");
  VCHECK(nv >= 0 && nt >= 0 && (nt == 0 || (verts && tris)), VISACD_ERR_INVALID_ARG, "sdf_remesh: bad sizes");
  VCHECK(scale > 0, VISACD_ERR_INVALID_ARG, "sdf_remesh: scale must be positive");
  ctx->sdf_nv = ctx->sdf_nt = 0;
  *out_nv = *out_nt = 0;
  if (nt == 0 || nv == 0) return VISACD_OK;
  VCHECK(indices_in_range(tris, 3LL * nt, nv), VISACD_ERR_INVALID_ARG, "sdf_remesh: triangle index out of range");
  VCUDA(cudaSetDevice(ctx->device));
  // Grid (host arithmetic of manifold_preprocess).
  std::vector<double> P(3 * (size_t)nv);
  double lo[3] = {1e308, 1e308, 1e308}, hi[3] = {-1e308, -1e308, -1e308};
  for (int32_t i = 0; i < nv; ++i)
    for (int a = 0; a < 3; ++a) {
      const double x = verts[3 * (size_t)i + a] * scale;
      P[3 * (size_t)i + a] = x;
      lo[a] = std::min(lo[a], x);
      hi[a] = std::max(hi[a], x);
    }
  const double iso = level * scale;
  SdfGrid g;
  g.band = std::max(iso, 0.0) + 2.0;
  g.fiso = (float)iso;
  g.scale = scale;
  for (int a = 0; a < 3; ++a) {
    g.org[a] = (int)std::floor(lo[a] - g.band - 2.0);
    g.dim[a] = (int)std::ceil(hi[a] + g.band + 2.0) - g.org[a] + 1;
  }
  VCHECK(g.dim[0] >= 3 && g.dim[1] >= 3 && g.dim[2] >= 3, VISACD_ERR_INVALID_ARG, "sdf_remesh: degenerate grid");
  double qmax = 0;
  for (int a = 0; a < 3; ++a)
    qmax = std::max(qmax, std::max(std::fabs((double)g.org[a]), std::fabs((double)g.org[a] + g.dim[a])));
  g.margin = (float)(1e-3 + 1e-6 * qmax);
  // The range of class_cut, wider by 0.01 for the rounding of the distances to
  // float and by the lower bounds' margin; it does not hold for iso <= 0.
  const bool all_exact = !(iso > 0.0);
  g.cut_out = (float)(iso + 1.0 + 0.01) + 2.0f * g.margin;
  g.low_out = (float)(iso - 1.0 - 0.01);
  g.reach = all_exact ? g.band : std::min(g.band, (double)g.cut_out);
  const size_t nvox = (size_t)g.dim[0] * g.dim[1] * g.dim[2];
  VCHECK(nvox <= ((size_t)1 << 30), VISACD_ERR_CAPACITY, "sdf_remesh: grid of %zu voxels is too large", nvox);
  const size_t ncell = (size_t)(g.dim[0] - 1) * (g.dim[1] - 1) * (g.dim[2] - 1);
  const size_t nint = (size_t)(g.dim[0] - 2) * (g.dim[1] - 2) * (g.dim[2] - 2);
  // Scratch layout in one buffer.
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t o = at;
    at += align256(bytes);
    return o;
  };
  const size_t oP = take(P.size() * 8), oT = take(3 * (size_t)nt * 4);
  const size_t upload = at;
  const size_t oTog = take(nvox * 4), oFlags = take(sizeof(SdfFlags));
  const size_t zero_end = at;
  const size_t oPrep = take((size_t)nt * sizeof(SdfTri)), oWide = take(3 * (size_t)nt * 4), oChunks = take((size_t)nt * 4), oChunkOff = take(((size_t)nt + 1) * 8), oDist = take(nvox * 4),
               oUb = take(nvox * 4), oPy = take(nvox), oPz = take(nvox), oIn = take(nvox), oCls = take(nvox),
               oF = take(nvox * 4), oFlag = take(ncell * 4), oCoff = take((ncell + 1) * 8), oCv = take(ncell * 4),
               oQcnt = take(nint * 4), oQoff = take((nint + 1) * 8);
  VTRY(ensure_slot(ctx, kSlotSdf, at));
  char* base = slot<char>(ctx, kSlotSdf);
  double* dP = (double*)(base + oP);
  int32_t* dT = (int32_t*)(base + oT);
  uint32_t* dist = (uint32_t*)(base + oDist);
  uint32_t *tog = (uint32_t*)(base + oTog), *ub = (uint32_t*)(base + oUb);
  uint8_t *par_y = (uint8_t*)(base + oPy), *par_z = (uint8_t*)(base + oPz), *inside = (uint8_t*)(base + oIn),
          *cls = (uint8_t*)(base + oCls);
  float* f = (float*)(base + oF);
  uint32_t* flag = (uint32_t*)(base + oFlag);
  uint64_t* coff = (uint64_t*)(base + oCoff);
  int32_t* cv = (int32_t*)(base + oCv);
  uint32_t* qcnt = (uint32_t*)(base + oQcnt);
  uint64_t* qoff = (uint64_t*)(base + oQoff);
  cudaStream_t st = ctx->stream;
  Stager up(ctx);
  VTRY(up.reserve(upload, 1));
  std::memcpy(up.host() + oP, P.data(), P.size() * 8);
  std::memcpy(up.host() + oT, tris, 3 * (size_t)nt * 4);
  VTRY(up.copy(base, upload));
  VCUDA(cudaMemsetAsync(base + oTog, 0, zero_end - oTog, st));
  const unsigned gv = grid_for((int64_t)nvox, 256, 16 * (int64_t)ctx->sm_count);
  const float band_f = (float)g.band;
  uint32_t band_bits;
  std::memcpy(&band_bits, &band_f, 4);
  SdfTri* prep = (SdfTri*)(base + oPrep);
  uint32_t* chunks = (uint32_t*)(base + oChunks);
  uint64_t* chunk_off = (uint64_t*)(base + oChunkOff);
  SdfFlags* flags = (SdfFlags*)(base + oFlags);
  unsigned *n_wide = &flags->n_wide, *n_far = &flags->n_far;
  VLAUNCH(ctx, kKSdfDist, grid_for(nt, 64, 32 * (int64_t)ctx->sm_count), 64, 0, sdf_tri_prep_kernel, dP, dT, nt,
          g, prep, chunks, flags);
  // Crossings of all three axes, the triangles covering many rays one block
  // each, then the parities and classes.
  int* wide = (int*)(base + oWide);
  VLAUNCH(ctx, kKSdfCross, dim3(grid_for((int64_t)kCrossLanes * nt, 128, 16 * (int64_t)ctx->sm_count), 3), 128, 0,
          sdf_cross_kernel, dP, dT, nt, g, (const SdfTri*)prep, tog, wide, n_wide);
  VLAUNCH(ctx, kKSdfCross, (unsigned)std::min<int64_t>(3LL * nt, 4 * (int64_t)ctx->sm_count), 128, 0,
          sdf_cross_wide_kernel, dP, dT, g, (const SdfTri*)prep, (const int*)wide, (const unsigned*)n_wide, tog);
  VLAUNCH(ctx, kKSdfCross,
          dim3(grid_for((int64_t)g.dim[0] * std::max(g.dim[1], g.dim[2]), 64, 32 * (int64_t)ctx->sm_count), 2), 64, 0,
          sdf_parity_yz_kernel, g, (const uint32_t*)tog, par_y, par_z);
  VLAUNCH(ctx, kKSdfCross, grid_for(32LL * g.dim[1] * g.dim[2], 128, 16 * (int64_t)ctx->sm_count), 128, 0,
          sdf_inside_kernel, g, (const uint32_t*)tog, (const uint8_t*)par_y, (const uint8_t*)par_z, inside);
  VLAUNCH(ctx, kKSdf, gv, 256, 0, sdf_class_kernel, g, (const uint8_t*)inside, all_exact ? 1 : 0,
          band_bits, cls, ub, dist);
  VTRY(exclusive_scan_u32_to_u64(ctx, chunks, chunk_off, nt));
  SdfItems items;
  items.off = chunk_off;
  items.nt = nt;
  const unsigned gw = (unsigned)(kDistBlocks * (int64_t)ctx->sm_count);
  // First pass: FP32 upper bounds per voxel, then the exact pass.
  VLAUNCH(ctx, kKSdfDist, (unsigned)(kUbBlocks * (int64_t)ctx->sm_count), 128, 0, sdf_ub_kernel, items, g, (const SdfTri*)prep, (const uint8_t*)cls, ub);
  VLAUNCH(ctx, kKSdfDist, gw, 128, 0, sdf_dist_kernel, dP, dT, items, g, (const SdfTri*)prep, (const uint8_t*)cls,
          (const uint32_t*)ub, dist);
  if (g.reach < g.band) {
    VLAUNCH(ctx, kKSdf, gv, 256, 0, sdf_far_kernel, g, nvox, (const uint32_t*)dist, (const uint32_t*)ub, cls, flags);
    VLAUNCH(ctx, kKSdfDist, gw, 128, 0, sdf_far_dist_kernel, dP, dT, items, g, (const SdfTri*)prep, (const uint8_t*)cls,
            (const unsigned*)n_far, dist);
  }
  VLAUNCH(ctx, kKSdf, gv, 256, 0, sdf_field_kernel, (const uint32_t*)dist, (const uint32_t*)ub, (const uint8_t*)cls,
          nvox, f);
  const unsigned gc = grid_for((int64_t)ncell, 256, 16 * (int64_t)ctx->sm_count);
  VLAUNCH(ctx, kKSdf, gc, 256, 0, sdf_cell_flag_kernel, g, f, flag);
  VTRY(exclusive_scan_u32_to_u64(ctx, flag, coff, (int64_t)ncell));
  const unsigned gq = grid_for((int64_t)nint, 256, 16 * (int64_t)ctx->sm_count);
  uint64_t* totals = nullptr;
  VTRY(pinned(ctx, 2 * sizeof(uint64_t), (void**)&totals));
  VCUDA(cudaMemcpyAsync(&totals[0], coff + ncell, 8, cudaMemcpyDeviceToHost, st));
  VCUDA(stream_wait(ctx));
  VCHECK(totals[0] < (1ull << 31), VISACD_ERR_CAPACITY, "sdf_remesh: too many vertices");
  // (the vertices, then the list of their cells)
  VTRY(ensure_slot(ctx, kSlotSdfOut, align256(totals[0] * 24) + totals[0] * 4 + 256));
  double* out_v = slot<double>(ctx, kSlotSdfOut);
  uint32_t* cells = reinterpret_cast<uint32_t*>(slot<char>(ctx, kSlotSdfOut) + align256(totals[0] * 24));
  VLAUNCH(ctx, kKSdf, gc, 256, 0, sdf_cell_list_kernel, ncell, flag, coff, cv, cells);
  if (totals[0])
    VLAUNCH(ctx, kKSdf, grid_for((int64_t)totals[0], 64, 32 * (int64_t)ctx->sm_count), 64, 0, sdf_cell_vertex_kernel,
            g, f, (const uint32_t*)cells, (size_t)totals[0], out_v);
  VLAUNCH(ctx, kKSdf, gq, 256, 0, sdf_quad_kernel, g, f, cv, qcnt, (const uint64_t*)nullptr,
          (int32_t*)nullptr);
  VTRY(exclusive_scan_u32_to_u64(ctx, qcnt, qoff, (int64_t)nint));
  VCUDA(cudaMemcpyAsync(&totals[1], qoff + nint, 8, cudaMemcpyDeviceToHost, st));
  VCUDA(stream_wait(ctx));
  VCHECK(totals[1] < (1ull << 31), VISACD_ERR_CAPACITY, "sdf_remesh: too many triangles");
  VTRY(ensure_slot(ctx, kSlotSdfTris, align256(totals[1] * 12) + 256));
  VLAUNCH(ctx, kKSdf, gq, 256, 0, sdf_quad_kernel, g, f, cv, qcnt, qoff, slot<int32_t>(ctx, kSlotSdfTris));
  ctx->sdf_nv = (int32_t)totals[0];
  ctx->sdf_nt = (int32_t)totals[1];
  *out_nv = ctx->sdf_nv;
  *out_nt = ctx->sdf_nt;
  return VISACD_OK;
}

extern "C" int visacd_sdf_fetch(visacd_ctx* ctx, double* verts, int32_t* tris) {
  VCHECK(ctx, VISACD_ERR_INVALID_ARG, "sdf_fetch: null context");
  VCUDA(cudaSetDevice(ctx->device));
  VCHECK(ctx->sdf_nv == 0 || verts, VISACD_ERR_INVALID_ARG, "sdf_fetch: null vertex buffer");
  VCHECK(ctx->sdf_nt == 0 || tris, VISACD_ERR_INVALID_ARG, "sdf_fetch: null triangle buffer");
  void* const dst[2] = {verts, tris};
  const void* const src[2] = {slot<double>(ctx, kSlotSdfOut), slot<int32_t>(ctx, kSlotSdfTris)};
  const size_t bytes[2] = {(size_t)ctx->sdf_nv * 24, (size_t)ctx->sdf_nt * 12};
  return fetch(ctx, 2, dst, src, bytes);
}
