// Morton orders of triangles and points in one launch per batch of jobs, one
// thread-block cluster per job (order.cu).
#pragma once

#include "common.cuh"

namespace vgpu {

// What a BVH build leaves beside its nodes for the host (read when needed).
struct BvhHead {
  float tb[6];   // bounds of the triangles' vertices: min xyz, max xyz
  float amax;    // largest |vertex coordinate|
  unsigned bad;  // a triangle references a vertex out of range
};

// Primitives of one job: a BVH build of 32,768, 65,536 and 131,072 triangles takes
// 91, 112 and 167 us of kernels here and 249, 243 and 298 as separate launches (the
// grid-wide sort, hierarchy and fit), which spread larger sorts over more SMs than
// a cluster has.
constexpr int kOrderMax = 131072;
constexpr int kOrderMaxJobs = 12;  // jobs of one launch (kernel parameter space)

struct OrderJob {
  const float* verts;    // vertices (triangle jobs) or the points themselves
  const uint32_t* tris;  // null: a point job
  int32_t nv, n;         // vertices, primitives
  int32_t bits;          // Morton bits per axis (at most 10)
  uint32_t *k0, *v0;     // sorted keys and primitive ids
  uint32_t *k1, *v1;     // scratch of the same size
  float* cent;           // scratch: 3 n (triangle jobs)
  uint32_t* hist;        // scratch: 2 x cluster x 256
  float* part;           // scratch: cluster x 16
  // Triangle jobs: the leaves in order and the box tables of order_box.
  BvhHead* head;
  float4* nodes;                   // 4 (n - 1)
  float4* leaves;                  // 3 n
  float *box, *pre, *suf;          // 6 n: leaf boxes; unions from / to the ends of each run of 32 leaves
  float *bpre, *bsuf;              // 6 per run: unions from / to the ends of each group of 32 runs
  float* group;                    // 6 per group: its union
  // Point jobs with a mask: the new points in order and every point's rank.
  const uint8_t* is_new;
  uint32_t* rows;
  int32_t* rank;
};

// Scratch bytes of a job of n primitives, and its pointers carved from `base`
// (256-byte aligned pieces); k0 / v0 included.
size_t order_scratch(int64_t n, bool tris);
void order_carve(OrderJob& j, char* base);

// Enqueues the jobs (each at most kOrderMax primitives, at least one).
int order_run(visacd_ctx* ctx, const OrderJob* jobs, int n_jobs);

// Karras hierarchies and node records of finished triangle jobs (OrderJob::nodes).
int order_nodes(visacd_ctx* ctx, const OrderJob* jobs, int n_jobs);

// A one-launch build of a BVH over device input (1 to kOrderMax triangles): its
// memory and its job, for order_run and order_nodes. The handle is registered
// with the context; `scratch` holds order_scratch(nt, true) bytes.
int bvh_prepare(visacd_ctx* ctx, const float* dv, int32_t nv, const uint32_t* dt, int32_t nt, char* scratch,
                visacd_bvh** out, OrderJob& job);

}  // namespace vgpu
