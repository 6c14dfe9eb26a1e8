// Device side of the segment visibility test, shared by the single-part and
// the batched visibility kernels: segment setup, conservative slab test,
// FP32 segment-triangle test with its rounding bound, FP64 re-decision, and the
// warp-packet any-hit traversal (see vis.cu for the design notes).
#pragma once

#include <math.h>

#include "bvh.cuh"

namespace vgpu {

constexpr int kVisThreads = 128;
constexpr int kStack = 64;
constexpr float kU = 5.9604645e-8f;  // 2^-24
constexpr float kTmin = 0.001f;      // reference tmin (ray_segments.cu:99)

struct VisCounters {
  unsigned long long work;
  unsigned long long pairs, edges, self_hits, cage_hits, rechecks, degenerate;
  unsigned long long node_visits, tri_tests;  // per-warp node fetches, per-lane triangle tests
  unsigned pmin[3], pmax[3];  // orderable point bounds
  unsigned long long n_rows;  // rows of the tile space (masked mode)
  unsigned long long certified, trace_steps;  // free-space walks: segments cleared, grid reads
  unsigned long long walk_work;               // tile counter of the walk kernel
  unsigned long long pending;                 // tiles the walk left to the traversal
};

// A cage's free-space grid as the visibility kernel reads it (freegrid.cu).
struct FreeGridView {
  const float* lb;          // null: no grid
  cudaTextureObject_t tex;  // the same bounds as a 3D texture (border 0)
  float ox, oy, oz, h_up, inv_h, margin;  // h_up: the cell size times (1 + 1e-6)
  int32_t nx, ny, nz;
};

// Lower bound of the distance to the cage from the point at cell coordinates
// (u, v, w) (x = o + u h): the bound B of the centre of the cell the point
// falls in, less h x the point's distance to that centre in cells. Outside
// the grid the texture's border gives B = 0, so the result is negative.
__device__ __forceinline__ float free_bound(const FreeGridView& g, float u, float v, float w) {
  const float B = tex3D<float>(g.tex, u, v, w);
  // u - floor(u) is exact; so is subtracting 0.5 from it.
  const float rx = (u - floorf(u)) - 0.5f, ry = (v - floorf(v)) - 0.5f, rz = (w - floorf(w)) - 0.5f;
  // |r| from the hardware reciprocal square root (2 ulp), rounded up through
  // the factor folded into h_up = h (1 + 1e-6).
  const float q = rx * rx + ry * ry + rz * rz;
  return B - q * rsqrtf(q + 1e-30f) * g.h_up;
}

constexpr int kTraceSteps = 32;  // rounds (two grid reads each) before a segment goes to the BVH

// Free reach of the points by direction: the directions are 6 x m x m cells of a
// cube around the point (axis of the largest component, its sign, and m x m
// squares of the two other components over it), and reach[cell * n + row] is a
// length along the axis up to which every segment from the point with a
// direction in the cell stays free of the cage. Most of a walk's reads are the
// first, short advances away from the surface, and they are much the same for
// all segments of a cell, so a table of n x 6 m^2 reaches spares them to n^2 / 2.
struct FreeReach {
  const float* reach;  // null: none
  int m, n;
  int by_pos;          // rows are sorted positions (else vertex ids)
};

// Half the width of a cell's squares, with room for the rounding of the
// components by which a direction is sorted into it (about 2e-6).
__device__ __forceinline__ float reach_half(int m) { return 1.0f / (float)m + 1e-5f; }

// The reach of point p in a cell. Walking along the cell's middle direction c
// (largest component 1, length |c|), a point at axis length a of any segment of
// the cell is within a w of the walk's, w = sqrt(2) reach_half. With Q = lb -
// margin at the walk's point at a, all of them are free up to the a' with
// a' w + (a' - a) |c| <= Q. Roundings are directed as in trace_free, whose margin
// covers the rounding of the walk's points.
__device__ __forceinline__ float cell_reach(const FreeGridView& g, float px, float py, float pz, int m, int cell) {
  const int iu = cell % m, iv = (cell / m) % m, face = cell / (m * m);
  const float u = (float)(2 * iu + 1 - m) / (float)m, v = (float)(2 * iv + 1 - m) / (float)m;
  const float one = (face & 1) ? -1.f : 1.f;
  const int axis = face >> 1;
  const float cx = axis == 0 ? one : (axis == 1 ? v : u), cy = axis == 0 ? u : (axis == 1 ? one : v),
              cz = axis == 0 ? v : (axis == 1 ? u : one);
  const float w = __fmul_ru(1.4142137f, reach_half(m));
  const float c = __fsqrt_ru(__fadd_ru(__fadd_ru(1.f, __fmul_ru(u, u)), __fmul_ru(v, v))) * 1.000001f;
  const float inv = __frcp_rd(__fadd_ru(w, c));
  const float u0 = (px - g.ox) * g.inv_h, v0 = (py - g.oy) * g.inv_h, w0 = (pz - g.oz) * g.inv_h;
  const float du = cx * g.inv_h, dv = cy * g.inv_h, dw = cz * g.inv_h;
  float a = 0.f;
  for (int k = 0; k < kTraceSteps; ++k) {
    const float Q = __fsub_rd(free_bound(g, fmaf(a, du, u0), fmaf(a, dv, v0), fmaf(a, dw, w0)), g.margin);
    const float next = __fmul_rd(__fadd_rd(Q, __fmul_rd(a, c)), inv);
    if (!(next > a)) break;
    const bool slow = next < 1.02f * a;
    a = next;
    if (slow) break;
  }
  return a * (1.f - 1e-6f);
}

// The free ends of the segment p -> q (as trace_free) from the table.
__device__ __forceinline__ void cone_start(const FreeReach& T, uint32_t rp, uint32_t rq, float dx, float dy, float dz,
                                           float& t0, float& s0) {
  const float ax = fabsf(dx), ay = fabsf(dy), az = fabsf(dz);
  const int axis = ax >= ay ? (ax >= az ? 0 : 2) : (ay >= az ? 1 : 2);
  const float da = axis == 0 ? dx : (axis == 1 ? dy : dz);
  const float db = axis == 0 ? dy : (axis == 1 ? dz : dx);
  const float dc = axis == 0 ? dz : (axis == 1 ? dx : dy);
  const float len = fabsf(da);
  t0 = 0.f;
  s0 = 1.f;
  if (!(len > 1e-30f && len < 1e30f)) return;
  // Below 1 / len: the factor is eight times the hardware reciprocal's error.
  float inv;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(len * 1.000001f));
  const int m = T.m, top = m - 1;
  const float half = 0.5f * (float)m;
  const int iu = min(max((int)(fmaf(db, inv, 1.f) * half), 0), top);
  const int iv = min(max((int)(fmaf(dc, inv, 1.f) * half), 0), top);
  const int face = 2 * axis + (da < 0.f ? 1 : 0);
  const int cp = (face * m + iv) * m + iu, cq = ((face ^ 1) * m + (top - iv)) * m + (top - iu);
  // (at most 2^28 entries)
  t0 = __fmul_rd(T.reach[(uint32_t)cp * (uint32_t)T.n + rp], inv);
  s0 = __fsub_ru(1.f, __fmul_rd(T.reach[(uint32_t)cq * (uint32_t)T.n + rq], inv));
}


// Free-space walk of the segment p -> q (d = q - p rounded, len its FP32
// length) through a cage's grid, from both ends at once (two independent
// chains of dependent reads). The point at t has cell coordinates
// u0 + t du with u0 = (p - o) / h and du = d / h; from it the walk may
// advance by (lb - margin) / |q - p| in either direction, lb = free_bound:
// no cage triangle lies within lb of the point. The margin covers the FP32
// rounding of those coordinates against the true point of the segment (below
// 2e-4 cells for grids of at most 256 cells a side), of the cell centres, a
// cell read on either side of a face the point lies on, and leaves every
// covered point at least that far from the cage. True when the two covered
// parts [0, t] and [s, 1] meet: the segment cannot hit the cage. Roundings
// are directed so that the parts covered are never overstated. `steps`
// counts the grid reads.
// t0 and s0 > t0: [0, t0] and [s0, 1] are known to be free (cone_start).
__device__ __forceinline__ bool trace_free(const FreeGridView& g, float px, float py, float pz, float dx, float dy,
                                           float dz, float len, float t0, float s0, unsigned long long& steps) {
  // 1 / |q - p| rounded down; |q - p| <= len (1 + 17u).
  const float inv_len = __frcp_rd(__fmul_ru(len, 1.000001f));
  const float u0 = (px - g.ox) * g.inv_h, v0 = (py - g.oy) * g.inv_h, w0 = (pz - g.oz) * g.inv_h;
  const float du = dx * g.inv_h, dv = dy * g.inv_h, dw = dz * g.inv_h;
  float t = t0, s = s0;
  for (int k = 0; k < kTraceSteps; ++k) {
    const float lb0 = free_bound(g, fmaf(t, du, u0), fmaf(t, dv, v0), fmaf(t, dw, w0));
    const float lb1 = free_bound(g, fmaf(s, du, u0), fmaf(s, dv, v0), fmaf(s, dw, w0));
    steps += 2;
    if (!(lb0 > g.margin) || !(lb1 > g.margin)) return false;
    t = __fadd_rd(t, __fmul_rd(__fsub_rd(lb0, g.margin), inv_len));
    s = __fsub_ru(s, __fmul_rd(__fsub_rd(lb1, g.margin), inv_len));
    if (t >= s) return true;
  }
  return false;
}

// What the traversal keeps of a lane's segment p -> q (d = q - p rounded): per
// axis 1 / d, |1 / d| and -p / d in registers, for a box test of three FMAs per
// axis, and what a leaf test needs in shared memory (two 16-byte reads).
struct SegLeaf {
  float4 p[32];  // p, and edge_factor of d
  float4 d[32];  // d
};
struct Seg {
  float ix, iy, iz;
  float ax, ay, az;
  float nx, ny, nz;
  int vi, vj;    // endpoint vertex ids (p = pts[vi], q = pts[vj])
  bool exclude;  // skip triangles incident to vi or vj (self test)
  SegLeaf* leaf; // the warp's
};

__device__ __forceinline__ unsigned f2o_v(float f) {
  unsigned b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float o2f_v(unsigned o) {
  unsigned b = (o & 0x80000000u) ? (o & 0x7fffffffu) : ~o;
  return __uint_as_float(b);
}

__device__ __forceinline__ float max3f(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// 1 / d, with |d| taken as `least` at least.
__device__ __forceinline__ float inv_guard(float d, float least) {
  return __frcp_rn(fabsf(d) < least ? copysignf(least, d) : d);
}

__device__ __forceinline__ float edge_factor(float dx, float dy, float dz) {
  const float d1 = fabsf(dx) + fabsf(dy) + fabsf(dz);
  return 17.0f * kU * d1 * (1.0f + 4.0f * kU);
}
__device__ __forceinline__ float seg_length(float dx, float dy, float dz) {
  return __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)));
}

__device__ __forceinline__ void make_seg(Seg& s, float3 p, float3 q, int vi, int vj, float least, SegLeaf* leaf) {
  const float dx = __fsub_rn(q.x, p.x), dy = __fsub_rn(q.y, p.y), dz = __fsub_rn(q.z, p.z);
  s.ix = inv_guard(dx, least);
  s.iy = inv_guard(dy, least);
  s.iz = inv_guard(dz, least);
  s.ax = fabsf(s.ix);
  s.ay = fabsf(s.iy);
  s.az = fabsf(s.iz);
  s.nx = -(p.x * s.ix);
  s.ny = -(p.y * s.iy);
  s.nz = -(p.z * s.iz);
  s.vi = vi;
  s.vj = vj;
  s.exclude = true;
  s.leaf = leaf;
  // (each lane writes and reads its own)
  leaf->p[threadIdx.x & 31] = make_float4(p.x, p.y, p.z, edge_factor(dx, dy, dz));
  leaf->d[threadIdx.x & 31] = make_float4(dx, dy, dz, 0.f);
}

// Conservative slab test of the segment (t in [0, 1]) against the box with
// centre c and half extents e. Leaf boxes are widened by 2^-19 of the mesh's
// largest |coordinate| M, 32 units of FP32 rounding; with |p|, |q| <= 4 M the
// test's own error is at most 24 units (in position: one of |p| for p / d, one
// each of the two FMA results, of |x - p| for 1 / d and for the rounding of d), so
// no slack is needed. A component of d below seg_least counts as that: it moves the
// segment by far less than the widening, so the interval it gives is still too
// large. box_hit_wide serves points farther out.
__device__ __forceinline__ bool box_hit(const Seg& s, float cx, float cy, float cz, float ex, float ey, float ez) {
  const float tx = fmaf(cx, s.ix, s.nx), ty = fmaf(cy, s.iy, s.ny), tz = fmaf(cz, s.iz, s.nz);
  const float tn = max3f(fmaf(-ex, s.ax, tx), fmaf(-ey, s.ay, ty), fmaxf(fmaf(-ez, s.az, tz), 0.f));
  const float tf = min3f(fmaf(ex, s.ax, tx), fmaf(ey, s.ay, ty), fminf(fmaf(ez, s.az, tz), 1.f));
  return tn <= tf;
}
__device__ __forceinline__ bool box_hit_wide(const Seg& s, const float3& p, float cx, float cy, float cz, float ex,
                                             float ey, float ez) {
  const float t0x = __fmul_rn(__fsub_rn(__fsub_rd(cx, ex), p.x), s.ix), t1x = __fmul_rn(__fsub_rn(__fadd_ru(cx, ex), p.x), s.ix);
  const float t0y = __fmul_rn(__fsub_rn(__fsub_rd(cy, ey), p.y), s.iy), t1y = __fmul_rn(__fsub_rn(__fadd_ru(cy, ey), p.y), s.iy);
  const float t0z = __fmul_rn(__fsub_rn(__fsub_rd(cz, ez), p.z), s.iz), t1z = __fmul_rn(__fsub_rn(__fadd_ru(cz, ez), p.z), s.iz);
  const float tn = max3f(fminf(t0x, t1x), fminf(t0y, t1y), fmaxf(fminf(t0z, t1z), 0.f));
  float tf = min3f(fmaxf(t0x, t1x), fmaxf(t0y, t1y), fminf(fmaxf(t0z, t1z), 1.f));
  tf = fmaf(fabsf(tf), 4e-6f, tf);
  return tn <= tf;
}
// The least |component| of a segment's direction: its inverse times a coordinate
// (of 4 M at most) does not overflow.
__device__ __forceinline__ float seg_least(float amax0, float amax1) {
  return fmaxf(1e-30f, 1e-37f * fmaxf(amax0, amax1));
}
// Whether box_hit serves a segment made with `least` against a mesh whose largest
// |coordinate| is amax (also false for coordinates that are not finite).
__device__ __forceinline__ bool box_test_holds(float3 p, float3 q, float amax, float least) {
  const float m = fmaxf(fmaxf(fmaxf(fabsf(p.x), fabsf(p.y)), fmaxf(fabsf(p.z), fabsf(q.x))),
                        fmaxf(fabsf(q.y), fabsf(q.z)));
  // (fmax drops NaNs: those fail the sum)
  return amax <= 1e30f && (least <= 1e-30f || least <= 1e-7f * amax) && m <= 4.f * amax &&
         fabsf(p.x + p.y + p.z + q.x + q.y + q.z) < INFINITY;
}

// FP64 segment-triangle decision from the FP32 inputs; identical formula to the
// oracle. Explicit round-to-nearest intrinsics keep contraction out.
static __device__ bool tri_test64(float ox, float oy, float oz, float qx, float qy, float qz,
                                        float4 a, float4 b, float4 c) {
  double Ax = __dsub_rn(a.x, ox), Ay = __dsub_rn(a.y, oy), Az = __dsub_rn(a.z, oz);
  double Bx = __dsub_rn(b.x, ox), By = __dsub_rn(b.y, oy), Bz = __dsub_rn(b.z, oz);
  double Cx = __dsub_rn(c.x, ox), Cy = __dsub_rn(c.y, oy), Cz = __dsub_rn(c.z, oz);
  double Dx = __dsub_rn(qx, ox), Dy = __dsub_rn(qy, oy), Dz = __dsub_rn(qz, oz);
  double BCx = __dsub_rn(__dmul_rn(By, Cz), __dmul_rn(Bz, Cy));
  double BCy = __dsub_rn(__dmul_rn(Bz, Cx), __dmul_rn(Bx, Cz));
  double BCz = __dsub_rn(__dmul_rn(Bx, Cy), __dmul_rn(By, Cx));
  double CAx = __dsub_rn(__dmul_rn(Cy, Az), __dmul_rn(Cz, Ay));
  double CAy = __dsub_rn(__dmul_rn(Cz, Ax), __dmul_rn(Cx, Az));
  double CAz = __dsub_rn(__dmul_rn(Cx, Ay), __dmul_rn(Cy, Ax));
  double ABx = __dsub_rn(__dmul_rn(Ay, Bz), __dmul_rn(Az, By));
  double ABy = __dsub_rn(__dmul_rn(Az, Bx), __dmul_rn(Ax, Bz));
  double ABz = __dsub_rn(__dmul_rn(Ax, By), __dmul_rn(Ay, Bx));
  double Wa = __dadd_rn(__dadd_rn(__dmul_rn(Dx, BCx), __dmul_rn(Dy, BCy)), __dmul_rn(Dz, BCz));
  double Wb = __dadd_rn(__dadd_rn(__dmul_rn(Dx, CAx), __dmul_rn(Dy, CAy)), __dmul_rn(Dz, CAz));
  double Wc = __dadd_rn(__dadd_rn(__dmul_rn(Dx, ABx), __dmul_rn(Dy, ABy)), __dmul_rn(Dz, ABz));
  double det = __dadd_rn(__dadd_rn(Wa, Wb), Wc);
  if (!(det != 0.0)) return false;
  bool inside = (Wa >= 0.0 && Wb >= 0.0 && Wc >= 0.0) || (Wa <= 0.0 && Wb <= 0.0 && Wc <= 0.0);
  if (!inside) return false;
  double vol = __dadd_rn(__dadd_rn(__dmul_rn(Ax, BCx), __dmul_rn(Ay, BCy)), __dmul_rn(Az, BCz));
  double len = __dsqrt_rn(
      __dadd_rn(__dadd_rn(__dmul_rn(Dx, Dx), __dmul_rn(Dy, Dy)), __dmul_rn(Dz, Dz)));
  double tmin = (double)kTmin;
  double lhs = __dmul_rn(vol, len), rhs = __dmul_rn(tmin, det);
  if (det > 0.0) return lhs >= rhs && vol <= det;
  return lhs <= rhs && vol >= det;
}

// ---- double-float arithmetic: a value as the unevaluated sum h + l of two
// FP32 numbers (about 46 bits). GB300 does about two FP64 operations per clock
// and SM, so the tests the FP32 filter leaves open go through these first.
struct DF {
  float h, l;
};
// a - b, exactly (Knuth's two-sum).
__device__ __forceinline__ DF df_diff(float a, float b) {
  const float s = __fsub_rn(a, b), t = __fsub_rn(s, a);
  return {s, __fsub_rn(__fsub_rn(a, __fsub_rn(s, t)), __fadd_rn(b, t))};
}
__device__ __forceinline__ DF df_norm(float h, float l) {  // |h| >= |l| or h == 0
  const float s = __fadd_rn(h, l);
  return {s, __fsub_rn(l, __fsub_rn(s, h))};
}
// x y within 2^-44 |x y|.
__device__ __forceinline__ DF df_mul(DF x, DF y) {
  const float p = __fmul_rn(x.h, y.h);
  const float e = __fmaf_rn(x.h, y.l, __fmaf_rn(x.l, y.h, __fmaf_rn(x.h, y.h, -p)));
  return df_norm(p, e);
}
// x + y within 2^-44 (|x| + |y|).
__device__ __forceinline__ DF df_add(DF x, DF y) {
  const float s = __fadd_rn(x.h, y.h), t = __fsub_rn(s, x.h);
  const float e = __fadd_rn(__fsub_rn(x.h, __fsub_rn(s, t)), __fsub_rn(y.h, t));
  return df_norm(s, __fadd_rn(e, __fadd_rn(x.l, y.l)));
}
__device__ __forceinline__ DF df_neg(DF x) { return {-x.h, -x.l}; }
// a b - c d, and the product of the vectors a . b.
__device__ __forceinline__ DF df_det(DF a, DF b, DF c, DF d) { return df_add(df_mul(a, b), df_neg(df_mul(c, d))); }
__device__ __forceinline__ DF df_dot(DF ax, DF ay, DF az, DF bx, DF by, DF bz) {
  return df_add(df_add(df_mul(ax, bx), df_mul(ay, by)), df_mul(az, bz));
}

// The segment-triangle decision in double-float: 1 hit, 0 miss, 2 undecided.
// With L the largest component of the vertex vectors and |D| the 1-norm of the
// direction, the differences are exact, a component of a cross product is
// within 2^-42 L^2, an edge function within 2.5 x 2^-42 |D| L^2 and the volume
// within 2^-40 L^3; the bounds below are four times that, far above the FP64
// formula's own rounding (2^-49), so a sign beyond them is the sign FP64 finds.
// Sizes outside 2^-20 .. 2^20 (where low parts could underflow) stay undecided.
static __device__ int tri_filter_df(float ox, float oy, float oz, float qx, float qy, float qz, float4 a, float4 b,
                                    float4 c) {
  const DF Ax = df_diff(a.x, ox), Ay = df_diff(a.y, oy), Az = df_diff(a.z, oz);
  const DF Bx = df_diff(b.x, ox), By = df_diff(b.y, oy), Bz = df_diff(b.z, oz);
  const DF Cx = df_diff(c.x, ox), Cy = df_diff(c.y, oy), Cz = df_diff(c.z, oz);
  const DF Dx = df_diff(qx, ox), Dy = df_diff(qy, oy), Dz = df_diff(qz, oz);
  const float L = fmaxf(fmaxf(fmaxf(fabsf(Ax.h), fabsf(Ay.h)), fmaxf(fabsf(Az.h), fabsf(Bx.h))),
                        fmaxf(fmaxf(fmaxf(fabsf(By.h), fabsf(Bz.h)), fmaxf(fabsf(Cx.h), fabsf(Cy.h))), fabsf(Cz.h)));
  const float d1 = fabsf(Dx.h) + fabsf(Dy.h) + fabsf(Dz.h);
  if (!(L >= 9.5367432e-7f && L <= 1048576.f && d1 >= 9.5367432e-7f && d1 <= 1048576.f)) return 2;
  const DF BCx = df_det(By, Cz, Bz, Cy), BCy = df_det(Bz, Cx, Bx, Cz), BCz = df_det(Bx, Cy, By, Cx);
  const DF Wa = df_dot(Dx, Dy, Dz, BCx, BCy, BCz);
  const DF Wb = df_dot(Dx, Dy, Dz, df_det(Cy, Az, Cz, Ay), df_det(Cz, Ax, Cx, Az), df_det(Cx, Ay, Cy, Ax));
  const DF Wc = df_dot(Dx, Dy, Dz, df_det(Ay, Bz, Az, By), df_det(Az, Bx, Ax, Bz), df_det(Ax, By, Ay, Bx));
  const float Ew = 9.0949470e-13f * 2.5f * d1 * L * L;  // 4 x 2.5 x 2^-42
  const float mx = fmaxf(Wa.h, fmaxf(Wb.h, Wc.h)), mn = fminf(Wa.h, fminf(Wb.h, Wc.h));
  if (mx > Ew && mn < -Ew) return 0;
  const bool pos = mn > Ew, neg = mx < -Ew;
  if (!(pos || neg)) return 2;
  DF det = df_add(df_add(Wa, Wb), Wc), vol = df_dot(Ax, Ay, Az, BCx, BCy, BCz);
  if (neg) {
    det = df_neg(det);
    vol = df_neg(vol);
  }
  const float Ev = 3.6379788e-12f * L * L * L;  // 4 x 2^-40
  const float Ed = 4.0f * Ew;
  // vol <= det
  const float g1 = df_add(det, df_neg(vol)).h;
  const float e1 = Ed + Ev + 1e-6f * fabsf(g1);
  // vol |D| >= tmin det; |D| in FP32, within 2^-21
  const float dx = Dx.h, dy = Dy.h, dz = Dz.h;
  const float len = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)));
  const float g2 = vol.h * len - kTmin * det.h;
  const float e2 = Ev * len + kTmin * Ed + 1e-6f * (fabsf(vol.h) * len + kTmin * fabsf(det.h));
  if (g1 < -e1 || g2 < -e2) return 0;
  if (g1 > e1 && g2 > e2) return 1;
  return 2;
}

// A test the FP32 filter left open: double-float, then FP64. The answer is the
// FP64 formula's.
static __device__ __noinline__ bool tri_recheck(float ox, float oy, float oz, float qx, float qy, float qz, float4 a,
                                                float4 b, float4 c) {
  const int r = tri_filter_df(ox, oy, oz, qx, qy, qz, a, b, c);
  return r == 2 ? tri_test64(ox, oy, oz, qx, qy, qz, a, b, c) : r == 1;
}

// FP32 filter of the segment p -> p + d (d = q - p rounded, kw = edge_factor of d):
// 1 certain hit, 0 certain miss, 2 undecided (tri_recheck).
__device__ __forceinline__ int tri_test32(float ox, float oy, float oz, float dx, float dy, float dz, float kw,
                                          float4 a, float4 b, float4 c) {
  float Ax = __fsub_rn(a.x, ox), Ay = __fsub_rn(a.y, oy), Az = __fsub_rn(a.z, oz);
  float Bx = __fsub_rn(b.x, ox), By = __fsub_rn(b.y, oy), Bz = __fsub_rn(b.z, oz);
  float Cx = __fsub_rn(c.x, ox), Cy = __fsub_rn(c.y, oy), Cz = __fsub_rn(c.z, oz);
  float L = max3f(max3f(fabsf(Ax), fabsf(Ay), fabsf(Az)), max3f(fabsf(Bx), fabsf(By), fabsf(Bz)),
                  max3f(fabsf(Cx), fabsf(Cy), fabsf(Cz)));
  float BCx = By * Cz - Bz * Cy, BCy = Bz * Cx - Bx * Cz, BCz = Bx * Cy - By * Cx;
  float CAx = Cy * Az - Cz * Ay, CAy = Cz * Ax - Cx * Az, CAz = Cx * Ay - Cy * Ax;
  float ABx = Ay * Bz - Az * By, ABy = Az * Bx - Ax * Bz, ABz = Ax * By - Ay * Bx;
  float Wa = dx * BCx + dy * BCy + dz * BCz;
  float Wb = dx * CAx + dy * CAy + dz * CAz;
  float Wc = dx * ABx + dy * ABy + dz * ABz;
  float L2 = L * L;
  float Ew = kw * L2;
  float mx = max3f(Wa, Wb, Wc), mn = min3f(Wa, Wb, Wc);
  if (mx > Ew && mn < -Ew) return 0;  // edge functions of strictly opposite sign
  bool allpos = mn > Ew, allneg = mx < -Ew;
  if (!(allpos || allneg)) return 2;
  float sg = allpos ? 1.f : -1.f;
  float det_s = sg * ((Wa + Wb) + Wc);
  float vol_s = sg * (Ax * BCx + Ay * BCy + Az * BCz);
  float Ev = 49.0f * kU * L2 * L;
  float Edet = 3.0f * Ew + 2.02f * kU * det_s;
  float g1 = det_s - vol_s;
  float e1 = Edet + Ev + 2.0f * kU * fabsf(g1);
  const float len = seg_length(dx, dy, dz);
  float g2 = vol_s * len - kTmin * det_s;
  float e2 = (Ev + 6.0f * kU * fabsf(vol_s)) * len + kTmin * (Edet + 2.0f * kU * det_s) +
             2.0f * kU * fabsf(g2);
  if (g1 < -e1 || g2 < -e2) return 0;
  if (g1 > e1 && g2 > e2) return 1;
  return 2;
}

__device__ __forceinline__ bool leaf_hit(const float4* __restrict__ tris, int leaf, const Seg& s,
                                         const float* __restrict__ pts, unsigned& rechecks) {
  float4 a = __ldg(&tris[3 * leaf]), b = __ldg(&tris[3 * leaf + 1]), c = __ldg(&tris[3 * leaf + 2]);
  if (s.exclude) {
    int ia = __float_as_int(a.w), ib = __float_as_int(b.w), ic = __float_as_int(c.w);
    if (ia == s.vi || ia == s.vj || ib == s.vi || ib == s.vj || ic == s.vi || ic == s.vj)
      return false;
  }
  const float4 p = s.leaf->p[threadIdx.x & 31], d = s.leaf->d[threadIdx.x & 31];
  const int r = tri_test32(p.x, p.y, p.z, d.x, d.y, d.z, p.w, a, b, c);
  if (r == 2) {
    ++rechecks;
    const float* q = pts + 3 * (int64_t)s.vj;
    return tri_recheck(p.x, p.y, p.z, q[0], q[1], q[2], a, b, c);
  }
  return r == 1;
}

// Warp-packet any-hit traversal. Every lane carries its own segment; the warp
// walks one path through the BVH: a child is visited when any still-active
// lane's segment overlaps its box (ballot), node records are fetched at a
// warp-uniform address (one broadcast transaction), and a lane retires at its
// first hit. The stack is per warp and lives in registers: entry k is held by
// lane k mod 32, in the first register for k < 32 and the second above, so a
// push is a select and a pop one shuffle (no shared memory, no warp barrier).
// Lanes retire only at leaf tests, so the warp checks for an early exit only
// after those. Returns this lane's hit flag; `visits` grows by the node
// records fetched. `status_bits` collects stack-overflow / iteration-overrun
// conditions (the lane is then reported as hit and the call fails on the
// host).
template <bool WIDE>
static __device__ __forceinline__ bool packet_hits(const float4* __restrict__ nodes, const float4* __restrict__ tris,
                                                   int nt, const Seg& s, const float* __restrict__ pts, bool active,
                                                   unsigned& rechecks, unsigned& status_bits, unsigned& visits,
                                                   unsigned& tri_tests) {
  static_assert(kStack == 64, "two stack registers per lane");
  const unsigned full = 0xffffffffu;
  bool hit = false;
  if (nt <= 0) return false;
  if (!__ballot_sync(full, active)) return false;
  const int lane = threadIdx.x & 31;
  int stk0 = 0, stk1 = 0;
  int node = 0, sp = 0;
  const int max_iter = 4 * nt + 64;
  for (int it = 0; it < max_iter; ++it) {
    const float4* nd = nodes + 4 * node;
    const float4 n0 = __ldg(nd), n1 = __ldg(nd + 1), n2 = __ldg(nd + 2);
    const int2 lr = __ldg(reinterpret_cast<const int2*>(nd + 3));
    const int l = lr.x, r = lr.y;
    bool hl, hr;
    if (WIDE) {
      const float4 o = s.leaf->p[threadIdx.x & 31];
      const float3 p = make_float3(o.x, o.y, o.z);
      hl = active && box_hit_wide(s, p, n0.x, n0.y, n0.z, n0.w, n1.x, n1.y);
      hr = active && box_hit_wide(s, p, n1.z, n1.w, n2.x, n2.y, n2.z, n2.w);
    } else {
      hl = active && box_hit(s, n0.x, n0.y, n0.z, n0.w, n1.x, n1.y);
      hr = active && box_hit(s, n1.z, n1.w, n2.x, n2.y, n2.z, n2.w);
    }
    const unsigned bl = __ballot_sync(full, hl);
    const unsigned br = __ballot_sync(full, hr);
    int next = -1;
    // (all of these are the same in every lane)
    const bool leaf_l = bl && l < 0, leaf_r = br && r < 0, leaf = leaf_l || leaf_r;
    if (leaf) {
      // (one copy of the triangle test: two would cost registers)
#pragma unroll 1
      for (int k = leaf_l ? 0 : 1; k < (leaf_r ? 2 : 1); ++k) {
        if (active && (k ? hr : hl)) {
          ++tri_tests;
          if (leaf_hit(tris, ~(k ? r : l), s, pts, rechecks)) {
            hit = true;
            active = false;
          }
        }
      }
    }
    if (bl && l >= 0) next = l;
    if (br && r >= 0) {
      if (next < 0) {
        next = r;
      } else {
        if (sp >= kStack) {
          visits += it + 1;
          status_bits |= kStatusStackOverflow;
          return true;
        }
        if (sp < 32) {
          stk0 = lane == sp ? r : stk0;
        } else {
          stk1 = lane == sp - 32 ? r : stk1;
        }
        ++sp;
      }
    }
    if (leaf && !__ballot_sync(full, active)) {
      visits += it + 1;
      return hit;
    }
    if (next < 0) {
      if (sp == 0) {
        visits += it + 1;
        return hit;
      }
      --sp;
      next = __shfl_sync(full, sp < 32 ? stk0 : stk1, sp & 31);
    }
    node = next;
  }
  visits += max_iter;
  status_bits |= kStatusTraversalOverrun;
  return true;
}

static __device__ __noinline__ bool packet_hits_wide(const float4* __restrict__ nodes,
                                                     const float4* __restrict__ tris, int nt, Seg s,
                                                     const float* __restrict__ pts, bool active, unsigned* counts) {
  return packet_hits<true>(nodes, tris, nt, s, pts, active, counts[0], counts[1], counts[2], counts[3]);
}

// What a tile is traced against: [0] the cage, [1] the part.
struct TileMesh {
  const float4* nodes[2];
  const float4* tris[2];
  int32_t nt[2];
  const float* amax[2];  // the meshes' largest |coordinate|
};

inline TileMesh tile_mesh(const visacd_ctx* ctx, const visacd_bvh* part, const visacd_bvh* cage) {
  TileMesh m;
  const visacd_bvh* b[2] = {cage, part};
  for (int k = 0; k < 2; ++k) {
    m.nodes[k] = b[k]->nodes;
    m.tris[k] = b[k]->tris;
    m.nt[k] = b[k]->nt;
    m.amax[k] = bvh_amax(ctx, b[k]);
  }
  return m;
}

// A warp's totals of a launch, in shared memory (in registers they would be
// spilled inside the traversal).
enum { kSumPairs, kSumEdges, kSumSelf, kSumCage, kSumDegenerate, kSumRechecks, kSumVisits, kSumTests, kSums };

// The warp's segments (pts[i] -> pts[j], i < j, on active lanes) against the
// cage, then those that leave it against the part. Few segments leave the
// cage (most vertex pairs of a part are interior chords, which cross neither
// surface), so the second test runs for few. Bit 0: hits the cage; bit 1: hits
// the part as well (1 alone: an edge). leaf, sum: the warp's.
static __device__ __forceinline__ unsigned trace_tile(const TileMesh& M, const float* __restrict__ pts, uint32_t i,
                                                      uint32_t j, float3 p, float3 q, bool active,
                                                      SegLeaf* leaf, unsigned long long* sum,
                                                      unsigned& status_bits) {
  Seg s;
  const float amax[2] = {*M.amax[0], *M.amax[1]}, least = seg_least(amax[0], amax[1]);
  make_seg(s, p, q, (int)i, (int)j, least, leaf);
  unsigned h = 0, rechecks = 0, visits = 0, tests = 0;
  const bool holds[2] = {!active || box_test_holds(p, q, amax[0], least),
                         !active || box_test_holds(p, q, amax[1], least)};
#pragma unroll 1
  for (int k = 0; k < 2; ++k) {
    s.exclude = k == 1;
    bool hit;
    if (__all_sync(0xffffffffu, k ? holds[1] : holds[0])) {
      hit = packet_hits<false>(k ? M.nodes[1] : M.nodes[0], k ? M.tris[1] : M.tris[0], k ? M.nt[1] : M.nt[0], s, pts,
                               active, rechecks, status_bits, visits, tests);
    } else {
      unsigned counts[4] = {0, 0, 0, 0};
      hit = packet_hits_wide(k ? M.nodes[1] : M.nodes[0], k ? M.tris[1] : M.tris[0], k ? M.nt[1] : M.nt[0], s, pts,
                             active, counts);
      rechecks += counts[0];
      status_bits |= counts[1];
      visits += counts[2];
      tests += counts[3];
    }
    active = active && hit;
    if (active) h |= 1u << k;
    if (!__any_sync(0xffffffffu, active)) break;
  }
  const unsigned cage = __ballot_sync(0xffffffffu, h & 1u), self = __ballot_sync(0xffffffffu, h & 2u);
  rechecks = __reduce_add_sync(0xffffffffu, rechecks);
  tests = __reduce_add_sync(0xffffffffu, tests);
  if ((threadIdx.x & 31) == 0) {
    sum[kSumEdges] += __popc(cage & ~self);
    sum[kSumSelf] += __popc(self);
    sum[kSumCage] += __popc(cage);
    sum[kSumRechecks] += rechecks;
    sum[kSumVisits] += visits;
    sum[kSumTests] += tests;
  }
  return h;
}

__device__ __forceinline__ int64_t row_start(int64_t i, int64_t n) {
  return i * (2 * n - i - 1) / 2;
}

// Morton order of n device points into perm (vis.cu); synchronizes.
int vis_morton_order(visacd_ctx* ctx, const float* d_pts, int32_t n, uint32_t* perm);

}  // namespace vgpu
