// Morton order of triangles or points, and the tables a BVH is read off from,
// in one launch: the steps of the build that need the whole input (bounds, then
// four passes of a stable LSD radix sort) run inside one thread-block cluster,
// whose hardware barrier takes the place of a launch boundary.
//
// What bounds it is latency, not data (a part of 15,000 triangles is 1 MB): as
// separate launches the same steps took 8 (up to 32,768 triangles) to 20
// launches plus a read-back the host waited for, and the sort ran on one SM.
// A cluster of 8 CTAs cuts the sort's serial chain by 8 and needs no spin
// barrier; a single CTA serves up to kOrderSmall primitives and ranks the keys
// by counting up to kOrderRank (no passes).
//
// The sort is stable on exactly the Morton bits and starts from index order, so
// the order is that of radix_sort_u64 on the same codes.
//
// The tree's boxes are unions over runs of consecutive leaves (Karras' nodes
// are ranges of the sorted order). Instead of a bottom-up pass (an atomic
// arrival chain of one L2 round trip per level) every box is put together from
// precomputed unions: within runs of 32 leaves and groups of 32 runs, from the
// left and from the right (order_box). Unions of boxes are minima and maxima,
// so the boxes equal the bottom-up ones.
#include "bvh.cuh"
#include "order.cuh"

namespace vgpu {

namespace {

constexpr int kOrderThreads = 1024;
constexpr int kOrderWarps = kOrderThreads / 32;
constexpr int kOrderCluster = 8;
// Primitives one CTA serves (a build of 1,472 triangles 54 us, with the cluster 57;
// of 2,048 64 and 63), and of those the ones ranked by counting instead of sorted
// (400: 33 us, sorted 41; 512: 37 and 43; 688: 46, sorted 45; 1,024: 68 and 49).
constexpr int kOrderSmall = 2048;
constexpr int kOrderRank = 512;

struct OrderArgs {
  OrderJob job[kOrderMaxJobs];
};

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned cluster_size() {
  unsigned r;
  asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(r));
  return r;
}
// Barrier over the cluster's threads; orders their global accesses as well.
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ uint32_t spread10(uint32_t x) {
  x &= 0x3ffu;
  x = (x | (x << 16)) & 0x030000ffu;
  x = (x | (x << 8)) & 0x0300f00fu;
  x = (x | (x << 4)) & 0x030c30c3u;
  x = (x | (x << 2)) & 0x09249249u;
  return x;
}

__device__ __forceinline__ void box_union(float (&b)[6], const float* __restrict__ o) {
  const float2 a = *reinterpret_cast<const float2*>(o), c = *reinterpret_cast<const float2*>(o + 2),
               d = *reinterpret_cast<const float2*>(o + 4);
  b[0] = fminf(b[0], a.x);
  b[1] = fminf(b[1], a.y);
  b[2] = fminf(b[2], c.x);
  b[3] = fmaxf(b[3], c.y);
  b[4] = fmaxf(b[4], d.x);
  b[5] = fmaxf(b[5], d.y);
}
__device__ __forceinline__ void box_store(float* __restrict__ o, const float (&b)[6]) {
  *reinterpret_cast<float2*>(o) = make_float2(b[0], b[1]);
  *reinterpret_cast<float2*>(o + 2) = make_float2(b[2], b[3]);
  *reinterpret_cast<float2*>(o + 4) = make_float2(b[4], b[5]);
}
// Inclusive unions over the warp's lanes from lane 0 up / from lane 31 down.
__device__ __forceinline__ void warp_unions(const float (&b)[6], float (&pre)[6], float (&suf)[6]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int a = 0; a < 6; ++a) pre[a] = suf[a] = b[a];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
    for (int a = 0; a < 6; ++a) {
      const float x = __shfl_up_sync(0xffffffffu, pre[a], o), y = __shfl_down_sync(0xffffffffu, suf[a], o);
      if (lane >= o) pre[a] = a < 3 ? fminf(pre[a], x) : fmaxf(pre[a], x);
      if (lane + o < 32) suf[a] = a < 3 ? fminf(suf[a], y) : fmaxf(suf[a], y);
    }
  }
}

// Group g of 1024 leaves in order, by a block of 1024 threads: the leaf
// records, their boxes and the tables of unions; one run of 32 per warp.
__device__ __forceinline__ void order_leaves(const OrderJob& J, int g, float amax, float (&sum)[kOrderWarps][6]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, i = 1024 * g + (int)threadIdx.x;
  const float pad = amax * 1.9073486e-6f + 1e-30f;  // 2^-19 * max|coord|
  float b[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  if (i < J.n) {
    const uint32_t t = __ldcg(&J.v0[i]);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const uint32_t id = J.tris[3 * (int64_t)t + k];
      const uint32_t vi = id < (uint32_t)J.nv ? id : 0u;
      const float x = J.verts[3 * (int64_t)vi], y = J.verts[3 * (int64_t)vi + 1], z = J.verts[3 * (int64_t)vi + 2];
      J.leaves[3 * (int64_t)i + k] = make_float4(x, y, z, __int_as_float((int)id));
      b[0] = fminf(b[0], x);
      b[1] = fminf(b[1], y);
      b[2] = fminf(b[2], z);
      b[3] = fmaxf(b[3], x);
      b[4] = fmaxf(b[4], y);
      b[5] = fmaxf(b[5], z);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      b[a] -= pad;
      b[3 + a] += pad;
    }
    box_store(J.box + 6 * (int64_t)i, b);
  }
  float pre[6], suf[6];
  warp_unions(b, pre, suf);
  if (i < J.n) {
    box_store(J.pre + 6 * (int64_t)i, pre);
    box_store(J.suf + 6 * (int64_t)i, suf);
  }
  __syncthreads();  // the sums of a previous group are read
  if (lane == 31) {
#pragma unroll
    for (int a = 0; a < 6; ++a) sum[warp][a] = pre[a];
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int a = 0; a < 6; ++a) b[a] = sum[lane][a];
    warp_unions(b, pre, suf);
    const int r = 32 * g + lane;
    if (32 * r < J.n) {
      box_store(J.bpre + 6 * (int64_t)r, pre);
      box_store(J.bsuf + 6 * (int64_t)r, suf);
    }
    if (lane == 31) box_store(J.group + 6 * (int64_t)g, pre);
  }
}

// The leaves of a job a cluster sorted: one block per group (inside the
// cluster the groups would run one after another, 6.6 us each).
// blockIdx.y: the job.
__global__ void __launch_bounds__(kOrderThreads) order_leaves_kernel(const __grid_constant__ OrderArgs A) {
  __shared__ float sum[kOrderWarps][6];
  const OrderJob& J = A.job[blockIdx.y];
  if ((int)blockIdx.x * 1024 < J.n && J.n > kOrderSmall) order_leaves(J, (int)blockIdx.x, J.head->amax, sum);
}

__global__ void __launch_bounds__(kOrderThreads) order_kernel(const __grid_constant__ OrderArgs A) {
  __shared__ __align__(16) uint32_t cnt[kOrderWarps][256];
  __shared__ float red[kOrderWarps][14];
  __shared__ float sum[kOrderWarps][6];
  __shared__ float bnd[14];
  __shared__ uint32_t wsum[kOrderWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int C = (int)cluster_size(), rank = (int)cluster_rank();
  const OrderJob& J = A.job[blockIdx.x / C];
  const int n = J.n;
  const bool is_tri = J.tris != nullptr;
  const int chunk = (n + C - 1) / C;
  const int c0 = min(n, rank * chunk), c1 = min(n, c0 + chunk);
  // ---- bounds of the primitives' centres (finite ones), of the triangles'
  // vertices, the largest |coordinate|, bad indices.
  float s[14];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    s[a] = s[6 + a] = INFINITY;
    s[3 + a] = s[9 + a] = -INFINITY;
  }
  s[12] = s[13] = 0.f;
  if (is_tri) {
    const int64_t m = 3LL * J.nv, step = (int64_t)C * kOrderThreads;
    for (int64_t i = (int64_t)rank * kOrderThreads + tid; i < m; i += 4 * step) {
      float x[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) x[q] = i + q * step < m ? fabsf(J.verts[i + q * step]) : 0.f;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (x[q] < INFINITY) s[12] = fmaxf(s[12], x[q]);
    }
  }
#pragma unroll 2
  for (int i = c0 + tid; i < c1; i += kOrderThreads) {
    float c[3];
    if (is_tri) {
      const uint32_t id[3] = {J.tris[3 * (int64_t)i], J.tris[3 * (int64_t)i + 1], J.tris[3 * (int64_t)i + 2]};
      const bool bad = id[0] >= (uint32_t)J.nv || id[1] >= (uint32_t)J.nv || id[2] >= (uint32_t)J.nv;
      if (bad) s[13] = 1.f;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        float v[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          // (out-of-range indices read vertex 0; the build then fails)
          v[k] = J.verts[3 * (int64_t)(id[k] < (uint32_t)J.nv ? id[k] : 0u) + a];
          s[6 + a] = fminf(s[6 + a], v[k]);
          s[9 + a] = fmaxf(s[9 + a], v[k]);
        }
        c[a] = bad ? 0.f : (v[0] + v[1] + v[2]) * (1.0f / 3.0f);
        J.cent[3 * (int64_t)i + a] = c[a];
      }
      if (bad) continue;
    } else {
#pragma unroll
      for (int a = 0; a < 3; ++a) c[a] = J.verts[3 * (int64_t)i + a];
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      if (fabsf(c[a]) < INFINITY) {
        s[a] = fminf(s[a], c[a]);
        s[3 + a] = fmaxf(s[3 + a], c[a]);
      }
    }
  }
#pragma unroll
  for (int q = 0; q < 14; ++q) {
    const bool mn = q < 3 || (q >= 6 && q < 9);
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const float y = __shfl_xor_sync(0xffffffffu, s[q], o);
      s[q] = mn ? fminf(s[q], y) : fmaxf(s[q], y);
    }
    if (lane == 0) red[warp][q] = s[q];
  }
  __syncthreads();
  if (tid < 14) {
    const bool mn = tid < 3 || (tid >= 6 && tid < 9);
    float x = red[0][tid];
    for (int w = 1; w < kOrderWarps; ++w) x = mn ? fminf(x, red[w][tid]) : fmaxf(x, red[w][tid]);
    J.part[16 * rank + tid] = x;
  }
  cluster_barrier();
  if (tid < 14) {
    const bool mn = tid < 3 || (tid >= 6 && tid < 9);
    float x = __ldcg(&J.part[tid]);
    for (int r = 1; r < C; ++r) {
      const float y = __ldcg(&J.part[16 * r + tid]);
      x = mn ? fminf(x, y) : fmaxf(x, y);
    }
    bnd[tid] = x;
  }
  __syncthreads();
  if (is_tri && rank == 0) {
    if (tid < 6) J.head->tb[tid] = bnd[6 + tid];
    if (tid == 6) J.head->amax = bnd[12];
    if (tid == 7) J.head->bad = bnd[13] > 0.f ? 1u : 0u;
  }
  // ---- Morton codes of this CTA's chunk, in index order.
  const int passes = (3 * J.bits + 7) / 8;
  uint32_t *ks = passes & 1 ? J.k1 : J.k0, *vs = passes & 1 ? J.v1 : J.v0;
  uint32_t *kd = passes & 1 ? J.k0 : J.k1, *vd = passes & 1 ? J.v0 : J.v1;
  {
    float lo[3], sc[3];
    const float top = (float)((1u << J.bits) - 1u);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      lo[a] = bnd[a];
      const float ext = bnd[3 + a] - lo[a];
      sc[a] = ext > 0.f ? top / ext : 0.f;
    }
    const float* src = is_tri ? J.cent : J.verts;
    for (int i = c0 + tid; i < c1; i += kOrderThreads) {
      uint32_t q[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const float x = (src[3 * (int64_t)i + a] - lo[a]) * sc[a];
        q[a] = (uint32_t)fminf(fmaxf(x, 0.f), top);  // NaN -> 0
      }
      ks[i] = (spread10(q[0]) << 2) | (spread10(q[1]) << 1) | spread10(q[2]);
      vs[i] = (uint32_t)i;
    }
  }
  __syncthreads();
  const int run = (c1 - c0 + kOrderWarps - 1) / kOrderWarps;
  const int b0 = min(c1, c0 + warp * run), b1 = min(c1, b0 + run);
  const unsigned lt = (1u << lane) - 1u;
  if (n <= kOrderRank) {
    // ---- small jobs: every key's rank is the number of keys before it in
    // (key, index) order, counted over the keys in shared memory.
    uint32_t* sk = &cnt[0][0];
    const int pad = (n + 3) & ~3;
    const uint32_t own = tid < n ? __ldcg(&ks[tid]) : 0xffffffffu;
    if (tid < pad) sk[tid] = own;
    __syncthreads();
    if (32 * warp < n) {
      int rk = 0;
      for (int j = 0; j < pad; j += 4) {
        // (the padding keys are above every key)
        const uint4 o = *reinterpret_cast<const uint4*>(sk + j);
        rk += (o.x < own || (o.x == own && j < tid)) + (o.y < own || (o.y == own && j + 1 < tid)) +
              (o.z < own || (o.z == own && j + 2 < tid)) + (o.w < own || (o.w == own && j + 3 < tid));
      }
      // (every key was read before the barrier: source and destination may be
      // the same buffer)
      if (tid < n) {
        J.k0[rk] = own;
        J.v0[rk] = (uint32_t)tid;
      }
    }
    vs = J.v0;
    __syncthreads();
  } else {
    // ---- stable LSD passes: warp w owns a contiguous run of the CTA's chunk,
    // kept in registers over a pass when it fits (up to 65536 primitives).
    constexpr int kHold = 8;
    uint32_t* my = cnt[warp];
    for (int p = 0; p < passes; ++p) {
      const int shift = 8 * p;
      uint32_t* hist = J.hist + (size_t)(p & 1) * C * 256;
      const bool hold = run <= 32 * kHold;
      uint32_t hk[kHold], hv[kHold];
      if (hold) {
#pragma unroll
        for (int q = 0; q < kHold; ++q) {
          const int i = b0 + 32 * q + lane;
          hk[q] = i < b1 ? __ldcg(&ks[i]) : 0u;
          hv[q] = i < b1 ? __ldcg(&vs[i]) : 0u;
        }
      }
      for (int d = lane; d < 256; d += 32) my[d] = 0;
      __syncwarp();
      if (hold) {
#pragma unroll
        for (int q = 0; q < kHold; ++q)
          if (b0 + 32 * q + lane < b1) atomicAdd(&my[(hk[q] >> shift) & 255u], 1u);
      } else {
        for (int i = b0 + lane; i < b1; i += 32) atomicAdd(&my[(__ldcg(&ks[i]) >> shift) & 255u], 1u);
      }
      __syncthreads();
      // Digit d's count over the warps: four threads a digit, eight warps each.
      const int d = tid >> 2, w0 = (tid & 3) * 8;
      uint32_t part = 0;
#pragma unroll
      for (int w = 0; w < 8; ++w) part += cnt[w0 + w][d];
      uint32_t upto = part;  // inclusive over the four
      {
        const uint32_t y = __shfl_up_sync(0xffffffffu, upto, 1, 4);
        if ((tid & 3) >= 1) upto += y;
        const uint32_t z = __shfl_up_sync(0xffffffffu, upto, 2, 4);
        if ((tid & 3) >= 2) upto += z;
      }
      const uint32_t tot = __shfl_sync(0xffffffffu, upto, 3, 4);
      uint32_t all = tot, before = 0;
      if (C > 1) {
        if ((tid & 3) == 0) hist[rank * 256 + d] = tot;
        cluster_barrier();
        // Counts of this digit in all CTAs: two ranks a thread of the four.
        all = 0;
        for (int r = tid & 3; r < C; r += 4) {
          const uint32_t h = __ldcg(&hist[r * 256 + d]);
          all += h;
          if (r < rank) before += h;
        }
        all += __shfl_xor_sync(0xffffffffu, all, 1);
        all += __shfl_xor_sync(0xffffffffu, all, 2);
        before += __shfl_xor_sync(0xffffffffu, before, 1);
        before += __shfl_xor_sync(0xffffffffu, before, 2);
      }
      // Exclusive prefix over the digits (a digit's four threads hold the same).
      uint32_t x = (tid & 3) == 0 ? all : 0u;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (lane == 31) wsum[warp] = x;
      x = __shfl_sync(0xffffffffu, x, lane & ~3);  // through the digit's first thread
      __syncthreads();
      uint32_t first = lane < warp ? wsum[lane] : 0u;
#pragma unroll
      for (int o = 16; o; o >>= 1) first += __shfl_xor_sync(0xffffffffu, first, o);
      uint32_t at = first + x - all + before + upto - part;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        const uint32_t c = cnt[w0 + w][d];
        cnt[w0 + w][d] = at;
        at += c;
      }
      __syncthreads();
      auto place = [&](bool valid, uint32_t k, uint32_t v) {
        const uint32_t digit = valid ? (k >> shift) & 255u : 0xffffffffu;
        const unsigned peers = __match_any_sync(0xffffffffu, digit);
        if (valid) {
          const uint32_t pos = my[digit] + __popc(peers & lt);
          kd[pos] = k;
          vd[pos] = v;
        }
        __syncwarp();
        if (valid && (peers & lt) == 0) my[digit] += __popc(peers);
        __syncwarp();
      };
      if (hold) {
#pragma unroll
        for (int q = 0; q < kHold; ++q)
          if (b0 + 32 * q < b1) place(b0 + 32 * q + lane < b1, hk[q], hv[q]);
      } else {
        for (int base = b0; base < b1; base += 32) {
          const int i = base + lane;
          place(i < b1, i < b1 ? __ldcg(&ks[i]) : 0u, i < b1 ? __ldcg(&vs[i]) : 0u);
        }
      }
      if (C > 1) cluster_barrier();
      else __syncthreads();
      uint32_t* t = ks;
      ks = kd;
      kd = t;
      t = vs;
      vs = vd;
      vd = t;
    }
  }
  if (is_tri) {
    if (C == 1)
      for (int g = 0; 1024 * g < n; ++g) order_leaves(J, g, bnd[12], sum);
  } else if (J.is_new) {
    // ---- the new points in order (rows), and every point's rank among them.
    int c = 0;
    for (int i = b0 + lane; i < b1; i += 32) c += J.is_new[__ldcg(&vs[i])] != 0;
#pragma unroll
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (lane == 0) wsum[warp] = (uint32_t)c;
    __syncthreads();
    uint32_t own = 0, at = 0;
    for (int w = 0; w < kOrderWarps; ++w) {
      if (w < warp) at += wsum[w];
      own += wsum[w];
    }
    if (C > 1) {
      uint32_t* hist = J.hist;
      if (tid == 0) hist[rank * 256] = own;
      cluster_barrier();
      for (int r = 0; r < rank; ++r) at += __ldcg(&hist[r * 256]);
    }
    for (int base = b0; base < b1; base += 32) {
      const int i = base + lane;
      const uint32_t v = i < b1 ? __ldcg(&vs[i]) : 0u;
      const bool nw = i < b1 && J.is_new[v] != 0;
      const unsigned m = __ballot_sync(0xffffffffu, nw);
      if (nw) {
        const uint32_t k = at + __popc(m & lt);
        J.rows[k] = v;
        J.rank[v] = (int32_t)k;
      } else if (i < b1) {
        J.rank[v] = 0x7fffffff;
      }
      at += __popc(m);
    }
  }
}

// Union of the leaf boxes lo..hi (in order) from the tables.
__device__ __forceinline__ void order_box(const OrderJob& J, int lo, int hi, float (&b)[6]) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    b[a] = INFINITY;
    b[3 + a] = -INFINITY;
  }
  const int rl = lo >> 5, rh = hi >> 5;
  if (rl == rh) {
    if ((lo & 31) == 0) {
      box_union(b, J.pre + 6 * (int64_t)hi);
    } else if ((hi & 31) == 31 || hi == J.n - 1) {
      box_union(b, J.suf + 6 * (int64_t)lo);
    } else {
      for (int i = lo; i <= hi; ++i) box_union(b, J.box + 6 * (int64_t)i);
    }
    return;
  }
  box_union(b, J.suf + 6 * (int64_t)lo);
  box_union(b, J.pre + 6 * (int64_t)hi);
  const int r0 = rl + 1, r1 = rh - 1;  // whole runs in between
  if (r0 > r1) return;
  const int gl = r0 >> 5, gh = r1 >> 5;
  if (gl == gh) {
    if ((r0 & 31) == 0) {
      box_union(b, J.bpre + 6 * (int64_t)r1);
    } else if ((r1 & 31) == 31) {
      box_union(b, J.bsuf + 6 * (int64_t)r0);
    } else {
      for (int r = r0; r <= r1; ++r) box_union(b, J.pre + 6 * (int64_t)(32 * r + 31));
    }
    return;
  }
  box_union(b, J.bsuf + 6 * (int64_t)r0);
  box_union(b, J.bpre + 6 * (int64_t)r1);
  for (int g = gl + 1; g < gh; ++g) box_union(b, J.group + 6 * (int64_t)g);
}

// Common-prefix length of sorted keys i and j (ties broken by position).
__device__ __forceinline__ int key_delta(const uint32_t* __restrict__ k, int n, int i, int j) {
  if (j < 0 || j >= n) return -1;
  const uint32_t a = k[i], b = k[j];
  if (a == b) return 32 + __clz((unsigned)(i ^ j));
  return __clz(a ^ b);
}

// Internal node i of Karras (2012): its range from the common-prefix lengths,
// its split, both children's boxes and the traversal record, one thread each.
// blockIdx.y: the job.
__global__ void __launch_bounds__(128) order_nodes_kernel(const __grid_constant__ OrderArgs A) {
  const OrderJob& J = A.job[blockIdx.y];
  float4* __restrict__ nodes = J.nodes;
  const int n = J.n;
  const uint32_t* __restrict__ keys = J.k0;
  if (n == 1) {  // one internal node whose two children are that leaf
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      float b[6];
      order_box(J, 0, 0, b);
      node_record(nodes, 0, b, b, ~0, ~0);
    }
    return;
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n - 1; i += gridDim.x * blockDim.x) {
    const int d = (key_delta(keys, n, i, i + 1) - key_delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
    const int dmin = key_delta(keys, n, i, i - d);
    int lmax = 2;
    while (key_delta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
      if (key_delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = key_delta(keys, n, i, j);
    int s = 0, t = l;
    do {
      t = (t + 1) >> 1;
      if (key_delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    const int gamma = i + s * d + min(d, 0);
    const int lo = min(i, j), hi = max(i, j);
    float lb[6], rb[6];
    order_box(J, lo, gamma, lb);
    order_box(J, gamma + 1, hi, rb);
    node_record(nodes, i, lb, rb, lo == gamma ? ~gamma : gamma, hi == gamma + 1 ? ~(gamma + 1) : gamma + 1);
  }
}

inline size_t al256(size_t b) { return (b + 255) & ~size_t(255); }

}  // namespace

// The pieces of a job's scratch, in order.
static size_t order_layout(int64_t n, bool tris, size_t (&o)[15]) {
  const size_t runs = (size_t)((n + 31) / 32), groups = (size_t)((n + 1023) / 1024), N = (size_t)n;
  const size_t bytes[15] = {N * 4, N * 4, N * 4, N * 4, tris ? N * 12 : 0, (size_t)2 * kOrderCluster * 256 * 4,
                            (size_t)kOrderCluster * 16 * 4, 0, 0, tris ? N * 24 : 0, tris ? N * 24 : 0,
                            tris ? N * 24 : 0, tris ? runs * 24 : 0, tris ? runs * 24 : 0, tris ? groups * 24 : 0};
  size_t at = 0;
  for (int k = 0; k < 15; ++k) {
    o[k] = at;
    at += al256(bytes[k]);
  }
  return at;
}

size_t order_scratch(int64_t n, bool tris) {
  size_t o[15];
  return order_layout(n, tris, o);
}

void order_carve(OrderJob& j, char* base) {
  size_t o[15];
  order_layout(j.n, j.tris != nullptr, o);
  j.k0 = reinterpret_cast<uint32_t*>(base + o[0]);
  j.v0 = reinterpret_cast<uint32_t*>(base + o[1]);
  j.k1 = reinterpret_cast<uint32_t*>(base + o[2]);
  j.v1 = reinterpret_cast<uint32_t*>(base + o[3]);
  j.cent = reinterpret_cast<float*>(base + o[4]);
  j.hist = reinterpret_cast<uint32_t*>(base + o[5]);
  j.part = reinterpret_cast<float*>(base + o[6]);
  j.box = reinterpret_cast<float*>(base + o[9]);
  j.pre = reinterpret_cast<float*>(base + o[10]);
  j.suf = reinterpret_cast<float*>(base + o[11]);
  j.bpre = reinterpret_cast<float*>(base + o[12]);
  j.bsuf = reinterpret_cast<float*>(base + o[13]);
  j.group = reinterpret_cast<float*>(base + o[14]);
}

int order_run(visacd_ctx* ctx, const OrderJob* jobs, int n_jobs) {
  for (int at = 0; at < n_jobs;) {
    // Jobs of one cluster size share a launch.
    OrderArgs a;
    int m = 0;
    const bool small = jobs[at].n <= kOrderSmall;
    while (at < n_jobs && m < kOrderMaxJobs && (jobs[at].n <= kOrderSmall) == small) a.job[m++] = jobs[at++];
    const int C = small ? 1 : kOrderCluster;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(m * C));
    cfg.blockDim = dim3(kOrderThreads);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaEvent_t ev = nullptr;
    timing_begin(ctx, kKSortScatter, &ev);
    VCUDA(cudaLaunchKernelEx(&cfg, order_kernel, a));
    VTRY(after_launch(ctx, "order_kernel"));
    VTRY(timing_end(ctx, kKSortScatter, ev));
  }
  return VISACD_OK;
}

int order_nodes(visacd_ctx* ctx, const OrderJob* jobs, int n_jobs) {
  OrderArgs a;
  int most = 0;
  for (int k = 0; k < n_jobs; ++k) {
    a.job[k] = jobs[k];
    most = std::max(most, jobs[k].n);
  }
  if (most > kOrderSmall)
    VLAUNCH(ctx, kKNodeLayout, dim3((unsigned)((most + 1023) / 1024), (unsigned)n_jobs), kOrderThreads, 0,
            order_leaves_kernel, a);
  VLAUNCH(ctx, kKKarras, dim3(grid_for(most > 1 ? most - 1 : 1, 128, 32LL * ctx->sm_count), (unsigned)n_jobs), 128, 0,
          order_nodes_kernel, a);
  return VISACD_OK;
}

}  // namespace vgpu
