// Device-resident linear BVH shared by the builder and the visibility kernel.
#pragma once

#include <string.h>

#include "common.cuh"

// Node record (64 bytes, 4 x float4): centre c and half extents e of both
// children's boxes, then the children.
//   [0] L.c.x L.c.y L.c.z L.e.x
//   [1] L.e.y L.e.z R.c.x R.c.y
//   [2] R.c.z R.e.x R.e.y R.e.z
//   [3] left  right  (int bits; >= 0 internal node, < 0 leaf ~sorted_triangle)
// Leaf triangle record (48 bytes, 3 x float4): vertex xyz + vertex index bits.
struct visacd_bvh {
  int device = 0;
  int32_t nt = 0;
  int32_t nv = 0;
  int32_t depth = 0;         // the tree's depth, or a bound of it (depth_exact)
  bool depth_exact = false;
  // Bounds of the triangles' vertices (min xyz, max xyz), on the host once
  // bvh_head() has read them (builds in one launch leave them on the device).
  bool head_read = false;
  float tri_bounds[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  void* head = nullptr;      // device BvhHead, part of the nodes' allocation
  float4* nodes = nullptr;
  float4* tris = nullptr;
  visacd_ctx* ctx = nullptr;       // owning context (null once it is destroyed)
  cudaStream_t stream = nullptr;   // the owner's stream (stream-ordered allocations)
  // Free-space grid (freegrid.cu), built on first use for a large visibility
  // call when this BVH is the cage: lb per cell, x fastest.
  bool free_built = false;
  float* free_lb = nullptr;
  cudaArray_t free_arr = nullptr;            // the same values as a 3D texture
  cudaTextureObject_t free_tex = 0;          // (point sampling, border 0)
  float fg_ox = 0.f, fg_oy = 0.f, fg_oz = 0.f, fg_h = 0.f, fg_inv_h = 0.f, fg_margin = 0.f;
  int32_t fg_nx = 0, fg_ny = 0, fg_nz = 0;
};

namespace vgpu {

#ifdef __CUDACC__
// Centre and half extent of [lo, hi] along an axis: c - e and c + e enclose it (e
// rounded up). An infinite side (a vertex that is not finite) opens the axis both
// ways: its own centre would be infinite, and c - e or c + e a NaN.
__device__ __forceinline__ void box_axis(float lo, float hi, float& c, float& e) {
  c = 0.5f * lo + 0.5f * hi;
  e = fmaxf(__fsub_ru(hi, c), __fsub_ru(c, lo));
  if (!(e < INFINITY)) {
    c = 0.f;
    e = INFINITY;
  }
}

// The record of a node whose children's boxes are (lo xyz, hi xyz).
__device__ __forceinline__ void node_record(float4* __restrict__ nodes, int64_t i, const float* l, const float* r,
                                            int left, int right) {
  float lc[3], le[3], rc[3], re[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    box_axis(l[a], l[3 + a], lc[a], le[a]);
    box_axis(r[a], r[3 + a], rc[a], re[a]);
  }
  nodes[4 * i + 0] = make_float4(lc[0], lc[1], lc[2], le[0]);
  nodes[4 * i + 1] = make_float4(le[1], le[2], rc[0], rc[1]);
  nodes[4 * i + 2] = make_float4(rc[2], re[0], re[1], re[2]);
  nodes[4 * i + 3] = make_float4(__int_as_float(left), __int_as_float(right), 0.f, 0.f);
}
#endif

// Device address of a mesh's largest |coordinate| (for a mesh without
// triangles a word that is never needed).
inline const float* bvh_amax(const visacd_ctx* ctx, const visacd_bvh* b) {
  return b->head ? reinterpret_cast<const float*>(b->head) + 6 : reinterpret_cast<const float*>(ctx->d_status);
}

int bvh_build(visacd_ctx* ctx, const float* verts, int32_t nv, const uint32_t* tris, int32_t nt,
              int device_ptrs, visacd_bvh** out);
// Frees a BVH's device memory when its context goes away (the handle itself
// stays valid until visacd_bvh_destroy, and is rejected by queries).
void bvh_detach(visacd_bvh* b);
// Makes `depth` the tree's exact depth (waits for the stream; once per BVH).
int bvh_depth(visacd_bvh* b);
// Reads the BVH's head to the host (waits for the stream; once per BVH).
int bvh_head(visacd_ctx* ctx, visacd_bvh* b);
// A build may still be running on its context's stream: a call on another
// stream waits for that one first, in the way its own context waits.
int bvh_settle(visacd_ctx* ctx, const visacd_bvh* b);
// Builds the BVH's free-space grid (once; a BVH whose grid would not be
// usable keeps none), its resolution sized for a call over `pairs` pairs. Uses the context's counter slot and pinned staging
// buffer (waits for the stream first), so it runs before a call takes them.
// Asynchronous after one small read-back.
int free_grid_build(visacd_ctx* ctx, visacd_bvh* b, int64_t pairs);

}  // namespace vgpu
