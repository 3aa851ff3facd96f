// small.cu — the whole build of a small mesh (2 .. kSmallMaxTri triangles) by one
// block in one launch: centroids and their AABB, fit transform, Morton codes,
// the stable sort, Karras branches and the boxes, all on chip.
//
// Why.  Below a few thousand triangles the build is a chain of latencies: the
// cooperative front's barriers and four passes, the topology and six refit
// kernels, and the gaps between ten launches, of which each phase works for a
// microsecond or two.  One block does the same work without leaving its SM.
// Back-to-back builds (displaced tori), us:
//   triangles      18    60   242   968  1250  1984  3960
//   many kernels   36    36    37    41    44    48    53
//   one block     6.2   6.5   7.9    16    26    29    56
// (From 2,700 triangles on the two are within 3 us, where one launch instead of
// nine still decides: each costs a caller without a captured graph 2 us or more.)
// What bounds it from there on is one SM's instruction issue, in the sort first;
// at 4,096 triangles (two heaps of boxes, 213 KB) the shared memory is full too.
//
// Values and order of operations are those of the kernels it stands in for:
// - centroids, NaN-aware min / max, fit transform and codes as k_centroid_aabb
//   and k_morton_tri (transform_homogeneous, morton_code3);
// - the sort is a bitonic network over (code << 32 | triangle), whose order is the
//   stable order of the codes; the keys stay in registers and cross threads by
//   shuffles, through shared memory only for strides above a warp;
// - branches by topology_node on the sorted codes in shared memory;
// - boxes by range queries on a heap of the sorted leaf boxes in shared memory (a
//   branch's box is the leftmost extreme of its leaves, see build.cu).  With a NaN
//   in a leaf box the branches are merged in tree order instead, as the climb does.
#include <atomic>

#include "dm_device.cuh"
#include "dm_internal.h"
#include "dm_lbvh.cuh"

namespace dm {
namespace {

struct SharedCodes {
  const uint32_t* p;
  __device__ __forceinline__ uint32_t operator()(uint32_t i) const { return p[i]; }
};

struct SmallArgs {
  uint32_t num_tri, num_vtx, size;  // size: keys sorted and heap leaves, a power of two >= num_tri
  const uint32_t* tri2vtx;
  const float* vtx2xyz;
  uint32_t* bvhnodes;
  float* aabb;
  float* transform_out;                                           // optional, as are
  uint32_t *tri2morton_out, *idx2tri_out, *idx2morton_out, *other_end_out;  // these
  uint32_t* status;
};

__device__ __forceinline__ unsigned long long shfl_xor64(unsigned long long v, int mask) {
  return __shfl_xor_sync(0xffffffffu, v, mask);
}

// Ascending bitonic sort of size = kE * blockDim.x keys, kE consecutive ones per
// thread; `sh` holds size keys.
template <int kE>
__device__ __forceinline__ void bitonic_sort(unsigned long long (&key)[kE], uint32_t size, unsigned long long* sh) {
  const uint32_t p0 = threadIdx.x * kE;
#pragma unroll 1
  for (uint32_t k = 2; k <= size; k <<= 1) {
#pragma unroll 1
    for (uint32_t j = k >> 1; j >= static_cast<uint32_t>(kE); j >>= 1) {
      const bool cross = j >= 32u * kE;
      if (cross) {
#pragma unroll
        for (int e = 0; e < kE; ++e) sh[p0 + e] = key[e];
        __syncthreads();
      }
#pragma unroll
      for (int e = 0; e < kE; ++e) {
        const uint32_t p = p0 + e;
        const unsigned long long other = cross ? sh[p ^ j] : shfl_xor64(key[e], static_cast<int>(j / kE));
        const bool want_min = ((p & j) == 0u) == ((p & k) == 0u);
        key[e] = (other < key[e]) == want_min ? other : key[e];
      }
      if (cross) __syncthreads();
    }
#pragma unroll
    for (int j = kE / 2; j >= 1; j >>= 1) {
      if (k >= 2u * j) {
#pragma unroll
        for (int e = 0; e < kE; ++e) {
          if ((e & j) == 0) {
            const bool up = ((p0 + e) & k) == 0u;
            const unsigned long long a = key[e], b = key[e ^ j];
            const bool swap = (b < a) == up;
            key[e] = swap ? b : a;
            key[e ^ j] = swap ? a : b;
          }
        }
      }
    }
  }
}

template <int kE>
__global__ void __launch_bounds__(1024, 1) k_build_small(SmallArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Box* tree = reinterpret_cast<Box*>(smem_raw);  // 2 * size boxes: heap node h, leaf i at size + i
  uint32_t* other_end = reinterpret_cast<uint32_t*>(tree + 2 * a.size);  // size words
  // before the leaf boxes are known, the same room holds the sort's keys, then
  // the sorted codes and triangles
  unsigned long long* sh_keys = reinterpret_cast<unsigned long long*>(smem_raw);
  uint32_t* codes = reinterpret_cast<uint32_t*>(smem_raw);
  uint32_t* tris = codes + a.size;
  __shared__ float sh_mm[32][6];
  __shared__ float m[16];
  const uint32_t T = a.num_tri, tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;

  // centroids and their AABB: NaN is ignored, every comparison with it is false
  float3 c[kE];
  float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int e = 0; e < kE; ++e) {
    const uint32_t i = tid * kE + e;
    c[e] = make_float3(0.f, 0.f, 0.f);
    if (i >= T) continue;
    c[e] = tri_centroid(a.tri2vtx, a.num_vtx, a.vtx2xyz, i, a.status);
    const float cc[3] = {c[e].x, c[e].y, c[e].z};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (cc[d] < lo[d]) lo[d] = cc[d];
      const float h = __fadd_rn(cc[d], 0.0f);
      if (h > hi[d]) hi[d] = h;
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float l = __shfl_down_sync(0xffffffffu, lo[d], off), h = __shfl_down_sync(0xffffffffu, hi[d], off);
      if (l < lo[d]) lo[d] = l;
      if (h > hi[d]) hi[d] = h;
    }
  }
  if (lane == 0) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      sh_mm[warp][d] = lo[d];
      sh_mm[warp][3 + d] = hi[d];
    }
  }
  __syncthreads();
  // The fit transform (vtx2xyz.rs:19-37 on the centroids, Mat44/torch.py:120-140):
  // a component is NaN iff the first centroid's is.
  if (tid == 0) {
    for (uint32_t w = 1; w < blockDim.x / 32; ++w) {
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        if (sh_mm[w][d] < lo[d]) lo[d] = sh_mm[w][d];
        if (sh_mm[w][3 + d] > hi[d]) hi[d] = sh_mm[w][3 + d];
      }
    }
    const float c0[3] = {c[0].x, c[0].y, c[0].z};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (c0[d] != c0[d]) lo[d] = hi[d] = c0[d];
    }
    float ext = __fsub_rn(hi[0], lo[0]);
    const float ey = __fsub_rn(hi[1], lo[1]), ez = __fsub_rn(hi[2], lo[2]);
    if (ey > ext) ext = ey;
    if (ez > ext) ext = ez;
    const float s = __fdiv_rn(1.0f, ext);
#pragma unroll
    for (int k = 0; k < 16; ++k) m[k] = 0.0f;
    m[0] = m[5] = m[10] = s;
    m[15] = 1.0f;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float mid = __fmul_rn(__fadd_rn(lo[d], hi[d]), 0.5f);
      m[12 + d] = __fadd_rn(__fmul_rn(-mid, s), 0.5f);
    }
    if (a.transform_out) {
#pragma unroll
      for (int k = 0; k < 16; ++k) a.transform_out[k] = m[k];
    }
  }
  __syncthreads();

  // codes, sorted with their triangles
  unsigned long long key[kE];
#pragma unroll
  for (int e = 0; e < kE; ++e) {
    const uint32_t i = tid * kE + e;
    key[e] = ~0ull;  // past the mesh: after every key
    if (i >= T) continue;
    const float3 q = transform_homogeneous(m, c[e].x, c[e].y, c[e].z);
    const uint32_t code = morton_code3(q.x, q.y, q.z);
    if (a.tri2morton_out) a.tri2morton_out[i] = code;
    key[e] = static_cast<unsigned long long>(code) << 32 | i;
  }
  bitonic_sort<kE>(key, a.size, sh_keys);
#pragma unroll
  for (int e = 0; e < kE; ++e) {
    const uint32_t i = tid * kE + e;
    const uint32_t code = static_cast<uint32_t>(key[e] >> 32), tri = static_cast<uint32_t>(key[e]);
    codes[i] = code;
    tris[i] = tri;
    if (i >= T) continue;
    if (a.idx2morton_out) a.idx2morton_out[i] = code;
    if (a.idx2tri_out) a.idx2tri_out[i] = tri;
  }
  __syncthreads();

  // branches (neighbouring threads take neighbouring branches)
  for (uint32_t ib = tid; ib + 1 < T; ib += blockDim.x) {
    topology_node(T, SharedCodes{codes}, SharedCodes{tris}, a.bvhnodes, ib, other_end);
    if (a.other_end_out) a.other_end_out[ib] = other_end[ib];
  }
  uint32_t tri[kE];  // of the leaves tid, tid + blockDim.x, ..
#pragma unroll
  for (int e = 0; e < kE; ++e) tri[e] = tris[tid + e * blockDim.x];
  __syncthreads();

  // leaf boxes and the heap over them
  bool nan = false;
#pragma unroll
  for (int e = 0; e < kE; ++e) {
    const uint32_t i = tid + e * blockDim.x;
    Box b{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}};
    if (i < T) {
      tri_centroid_box(a.tri2vtx, a.num_vtx, a.vtx2xyz, tri[e], a.status, &b);
      box_store(a.aabb + 6ull * (T - 1 + i), b);
#pragma unroll
      for (int d = 0; d < 3; ++d) nan = nan || b.lo[d] != b.lo[d] || b.hi[d] != b.hi[d];
    }
    tree[a.size + i] = b;
  }
  if (__syncthreads_or(nan)) {
    // Tree order: the second child to arrive at a branch merges the two.  The
    // heap's inner part holds the branches' boxes, the arrivals take the place
    // of other_end.
    for (uint32_t i = tid; i < a.size; i += blockDim.x) other_end[i] = 0u;
    __syncthreads();
    for (uint32_t i = tid; i < T; i += blockDim.x) {
      uint32_t node = a.bvhnodes[3ull * (T - 1 + i)];
      // a branch has two children, so this climbs at most T - 1 branches
      for (uint32_t guard = 0; node < T - 1 && guard < T; ++guard) {
        __threadfence_block();
        if (atomicAdd(&other_end[node], 1u) == 0u) break;
        __threadfence_block();
        const uint32_t c0 = a.bvhnodes[3ull * node + 1], c1 = a.bvhnodes[3ull * node + 2];
        const Box b = box_union(tree[c0 < T - 1 ? c0 : a.size + c0 - (T - 1)],
                                tree[c1 < T - 1 ? c1 : a.size + c1 - (T - 1)]);
        tree[node] = b;
        box_store(a.aabb + 6ull * node, b);
        node = a.bvhnodes[3ull * node];
      }
    }
    return;
  }
  for (uint32_t half = a.size / 2; half > 0; half >>= 1) {
    for (uint32_t h = half + tid; h < 2 * half; h += blockDim.x) tree[h] = box_union(tree[2 * h], tree[2 * h + 1]);
    __syncthreads();
  }
  for (uint32_t ib = tid; ib + 1 < T; ib += blockDim.x) {
    const uint32_t o = other_end[ib];
    uint32_t l = (ib < o ? ib : o) + a.size, r = (ib < o ? o : ib) + a.size + 1;
    Box L{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}}, R = L;
    while (l < r) {
      if (l & 1u) L = box_union(L, tree[l++]);
      if (r & 1u) R = box_union(tree[--r], R);
      l >>= 1;
      r >>= 1;
    }
    box_store(a.aabb + 6ull * ib, box_union(L, R));
  }
}

inline size_t small_smem(uint32_t size) { return size * (2 * sizeof(Box) + sizeof(uint32_t)); }

}  // namespace

bool launch_build_small(cudaStream_t s, uint32_t num_tri, const uint32_t* tri2vtx, uint32_t num_vtx,
                        const float* vtx2xyz, uint32_t* bvhnodes, float* aabb, float* transform_out,
                        uint32_t* tri2morton_out, uint32_t* idx2tri_out, uint32_t* idx2morton_out,
                        uint32_t* other_end_out, uint32_t* status) {
  if (num_tri < 2 || num_tri > kSmallMaxTri) return false;
  uint32_t size = 64;
  while (size < num_tri) size *= 2;
  // the attribute is per device; set once, so that later calls (possibly under
  // stream capture) configure nothing
  static std::atomic<bool> configured[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  if (!configured[dev].load(std::memory_order_acquire)) {
    const int most = static_cast<int>(small_smem(kSmallMaxTri));
    if (cudaFuncSetAttribute(k_build_small<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess ||
        cudaFuncSetAttribute(k_build_small<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess ||
        cudaFuncSetAttribute(k_build_small<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    configured[dev].store(true, std::memory_order_release);
  }
  const SmallArgs a{num_tri, num_vtx,       size,           tri2vtx,     vtx2xyz,        bvhnodes,      aabb,
                    transform_out, tri2morton_out, idx2tri_out, idx2morton_out, other_end_out, status};
  const size_t smem = small_smem(size);
  if (size <= 1024) k_build_small<1><<<1, size, smem, s>>>(a);
  else if (size <= 2048) k_build_small<2><<<1, size / 2, smem, s>>>(a);
  else k_build_small<4><<<1, size / 4, smem, s>>>(a);
  return true;
}

}  // namespace dm
