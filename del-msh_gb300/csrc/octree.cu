// octree.cu — quad/oct-trees from the binary radix tree of sorted, unique
// Morton codes (quad_oct_tree.cu:1-233, CPU quad_oct_tree.rs:1-234,420-451):
//
//   k_brt_depth      per branch: Karras range / split (the LBVH's), branch
//                    links (leaf children encoded num_bnode + i), and the
//                    branch's depth (common prefix of the split pair) in
//                    levels of num_dim bits
//   k_onode_count /  a branch starts an octree node when its depth differs
//   k_onode_scan /   from its parent's; bnode2onode is the exclusive prefix
//   k_onode_write    sum of those flags (three-kernel scan), and idx2bnode
//                    is each leaf's parent branch
//   k_make_tree      per leaf and per node-starting branch: the octree
//                    parent (walk up the binary tree to the branch that
//                    starts a node), the child slot from the Morton digit,
//                    centres and depths
//   k_aggregate      the sum of the leaves below each octree node, combined
//                    on chip before it is added
//
// Everything but k_aggregate is integer work or exact float arithmetic
// (halvings of sums of 0/1), so the outputs are bit-exact; k_aggregate adds
// with atomics, as the reference kernel does.
#include "dm_device.cuh"
#include "dm_internal.h"
#include "dm_lbvh.cuh"

namespace dm {
namespace {

constexpr int kThreads = 256;
constexpr int kScanItems = 8;  // flags per thread in the scan kernels
constexpr uint32_t kScanTile = kThreads * kScanItems;

struct Codes {
  const uint32_t* p;
  __device__ __forceinline__ uint32_t operator()(uint32_t i) const { return __ldg(p + i); }
};

__global__ void __launch_bounds__(kThreads) k_brt_depth(uint32_t num_bnode, const uint32_t* __restrict__ idx2morton,
                                                       uint32_t num_dim, uint32_t max_depth, uint32_t* bnodes,
                                                       uint32_t* bnode2depth) {
  const uint32_t ib = blockIdx.x * kThreads + threadIdx.x;
  if (ib >= num_bnode) return;
  if (ib == 0) bnodes[0] = kUMax;
  uint32_t r0, r1, isplit;
  const Codes c{idx2morton};
  karras_range_split(num_bnode + 1, c, ib, r0, r1, isplit);
  uint32_t* me = bnodes + static_cast<size_t>(ib) * 3;
  if (r0 == isplit) {
    me[1] = num_bnode + isplit;
  } else {
    me[1] = isplit;
    bnodes[static_cast<size_t>(isplit) * 3] = ib;
  }
  if (r1 == isplit + 1) {
    me[2] = num_bnode + isplit + 1;
  } else {
    me[2] = isplit + 1;
    bnodes[static_cast<size_t>(isplit + 1) * 3] = ib;
  }
  const uint32_t delta = static_cast<uint32_t>(__clz(c(isplit) ^ c(isplit + 1)));
  const uint32_t offset = 32u - num_dim * max_depth;
  bnode2depth[ib] = (delta - offset) / num_dim;  // u32 arithmetic, as the CPU code
}

// flag k (k < num_bnode - 1): branch k + 1 starts an octree node
__device__ __forceinline__ uint32_t onode_flag(uint32_t k, uint32_t num_bnode, const uint32_t* __restrict__ bnodes,
                                               const uint32_t* __restrict__ bnode2depth, uint32_t* status) {
  if (k + 1 >= num_bnode) return 0u;
  const uint32_t ib = k + 1, parent = __ldg(bnodes + static_cast<size_t>(ib) * 3);
  if (parent >= num_bnode) {
    raise_status(status, kStatusBadIndex);
    return 0u;
  }
  return __ldg(bnode2depth + ib) != __ldg(bnode2depth + parent) ? 1u : 0u;
}

__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t* sh) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  uint32_t t = 0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kThreads / 32; ++w) t += sh[w];
  return t;  // thread 0
}

// Per tile of kScanTile flags: their sum; also idx2bnode.
__global__ void __launch_bounds__(kThreads) k_onode_count(uint32_t num_bnode, const uint32_t* __restrict__ bnodes,
                                                         const uint32_t* __restrict__ bnode2depth,
                                                         uint32_t* idx2bnode, uint32_t* tile_sums, uint32_t* status) {
  __shared__ uint32_t sh[kThreads / 32];
  const uint32_t base = blockIdx.x * kScanTile;
  uint32_t v = 0;
  for (int q = 0; q < kScanItems; ++q) {
    const uint32_t k = base + q * kThreads + threadIdx.x;
    if (k >= num_bnode) continue;
    v += onode_flag(k, num_bnode, bnodes, bnode2depth, status);
    for (int side = 1; side <= 2; ++side) {
      const uint32_t ch = __ldg(bnodes + static_cast<size_t>(k) * 3 + side);
      if (ch >= num_bnode) {
        const uint32_t idx = ch - num_bnode;
        if (idx <= num_bnode) idx2bnode[idx] = k;
        else raise_status(status, kStatusBadIndex);
      }
    }
  }
  const uint32_t t = block_sum(v, sh);
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = t;
}

// One block: exclusive scan of the tile sums, in place.
__global__ void __launch_bounds__(1024) k_onode_scan(uint32_t num_tiles, uint32_t* tile_sums) {
  __shared__ uint32_t sh[32];
  __shared__ uint32_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (uint32_t b = 0; b < num_tiles; b += 1024) {
    const uint32_t i = b + threadIdx.x;
    const uint32_t v = i < num_tiles ? tile_sums[i] : 0u;
    uint32_t x = v;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
      if (lane >= off) x += y;
    }
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    if (warp == 0) {
      uint32_t w = sh[lane];
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, w, off);
        if (lane >= off) w += y;
      }
      sh[lane] = w;
    }
    __syncthreads();
    const uint32_t excl = carry + (warp > 0 ? sh[warp - 1] : 0u) + x - v;
    if (i < num_tiles) tile_sums[i] = excl;
    __syncthreads();
    if (threadIdx.x == 1023) carry = excl + v;
    __syncthreads();
  }
}

// bnode2onode[i] = sum of flags k < i: the tile's offset plus a scan of the
// tile, kScanItems consecutive flags per thread.
__global__ void __launch_bounds__(kThreads) k_onode_write(uint32_t num_bnode, const uint32_t* __restrict__ bnodes,
                                                         const uint32_t* __restrict__ bnode2depth,
                                                         const uint32_t* __restrict__ tile_offsets,
                                                         uint32_t* bnode2onode, uint32_t* status) {
  __shared__ uint32_t sh[kThreads / 32];
  const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  uint32_t f[kScanItems], sum = 0;
#pragma unroll
  for (int q = 0; q < kScanItems; ++q) {
    f[q] = base + q < num_bnode ? onode_flag(base + q, num_bnode, bnodes, bnode2depth, status) : 0u;
    sum += f[q];
  }
  // exclusive scan of the per-thread sums over the block
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = sum;
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off) x += y;
  }
  if (lane == 31) sh[warp] = x;
  __syncthreads();
  uint32_t before = 0;
  for (int w = 0; w < warp; ++w) before += sh[w];
  uint32_t run = __ldg(tile_offsets + blockIdx.x) + before + x - sum;
#pragma unroll
  for (int q = 0; q < kScanItems; ++q) {
    if (base + q < num_bnode) bnode2onode[base + q] = run;
    run += f[q];
  }
}

// quad_oct_tree.rs:52-63: centre of the cell of `morton` at `depth`.
__device__ __forceinline__ void morton2center(uint32_t morton, uint32_t num_dim, uint32_t depth, uint32_t max_depth,
                                              float center[3]) {
  uint32_t key = morton >> ((max_depth - depth) * num_dim);
  for (uint32_t d = 0; d < num_dim; ++d) center[d] = 0.5f;
  for (uint32_t i = 0; i < depth; ++i)
    for (uint32_t d = 0; d < num_dim; ++d) {
      const uint32_t j = num_dim - d - 1;
      center[j] = __fmul_rn(__fadd_rn(center[j], static_cast<float>(key & 1u)), 0.5f);
      key >>= 1;
    }
}

// The octree parent of binary node `cur`: walk up to the branch that starts
// an octree node (the root, or bnode2onode changes at it).
__device__ __forceinline__ bool onode_parent(uint32_t cur, uint32_t num_bnode, const uint32_t* __restrict__ bnodes,
                                             const uint32_t* __restrict__ bnode2onode,
                                             const uint32_t* __restrict__ bnode2depth, uint32_t& onode,
                                             uint32_t& depth) {
  for (uint32_t guard = 0; guard <= num_bnode; ++guard) {
    if (cur >= num_bnode) return false;
    if (cur == 0 || __ldg(bnode2onode + cur) != __ldg(bnode2onode + cur - 1)) {
      onode = __ldg(bnode2onode + cur);
      depth = __ldg(bnode2depth + cur);
      return true;
    }
    cur = __ldg(bnodes + static_cast<size_t>(cur) * 3);
  }
  return false;
}

// quad_oct_tree.rs:127-233 / quad_oct_tree.cu make_tree_from_binary_radix_tree.
__global__ void __launch_bounds__(kThreads) k_make_tree(uint32_t num_idx, const uint32_t* __restrict__ bnodes,
                                                       const uint32_t* __restrict__ bnode2onode,
                                                       const uint32_t* __restrict__ bnode2depth,
                                                       const uint32_t* __restrict__ idx2bnode,
                                                       const uint32_t* __restrict__ idx2morton, uint32_t num_onode,
                                                       uint32_t max_depth, uint32_t num_dim, uint32_t* onodes,
                                                       uint32_t* onode2depth, float* onode2center,
                                                       uint32_t* idx2onode, float* idx2center, uint32_t* status) {
  const uint32_t i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= num_idx) return;
  const uint32_t num_bnode = num_idx - 1, num_child = 1u << num_dim, nlink = num_child + 1;
  {  // leaf i
    uint32_t op, dp;
    if (!onode_parent(__ldg(idx2bnode + i), num_bnode, bnodes, bnode2onode, bnode2depth, op, dp) || op >= num_onode ||
        dp >= max_depth) {
      raise_status(status, kStatusBadIndex);
    } else {
      const uint32_t key = __ldg(idx2morton + i);
      const uint32_t ic = (key >> ((max_depth - 1 - dp) * num_dim)) & (num_child - 1);
      onodes[static_cast<size_t>(op) * nlink + 1 + ic] = i + num_onode;
      idx2onode[i] = op;
      float center[3];
      morton2center(key, num_dim, max_depth, max_depth, center);
      for (uint32_t d = 0; d < num_dim; ++d) idx2center[static_cast<size_t>(i) * num_dim + d] = center[d];
    }
  }
  if (i + 1 >= num_idx) return;
  const uint32_t ib = i;  // branch i
  if (ib == 0) {
    for (uint32_t d = 0; d < num_dim; ++d) onode2center[d] = 0.5f;
    return;
  }
  if (__ldg(bnode2onode + ib - 1) == __ldg(bnode2onode + ib)) return;  // starts no octree node
  uint32_t op, dp;
  if (!onode_parent(__ldg(bnodes + static_cast<size_t>(ib) * 3), num_bnode, bnodes, bnode2onode, bnode2depth, op,
                    dp) ||
      op >= num_onode || dp >= max_depth) {
    raise_status(status, kStatusBadIndex);
    return;
  }
  const uint32_t morton = __ldg(idx2morton + ib);
  const uint32_t ic = (morton >> ((max_depth - 1 - dp) * num_dim)) & (num_child - 1);
  const uint32_t on = __ldg(bnode2onode + ib);
  if (on >= num_onode) {
    raise_status(status, kStatusBadIndex);
    return;
  }
  onodes[static_cast<size_t>(op) * nlink + 1 + ic] = on;
  onodes[static_cast<size_t>(on) * nlink] = op;
  const uint32_t depth = __ldg(bnode2depth + ib);
  float center[3];
  morton2center(morton, num_dim, depth, max_depth, center);
  for (uint32_t d = 0; d < num_dim; ++d) onode2center[static_cast<size_t>(on) * num_dim + d] = center[d];
  onode2depth[on] = depth;
}

// Aggregation (quad_oct_tree.cu aggregate / quad_oct_tree.rs:420-451).
//
// Adding every leaf to every ancestor with one atomic each makes all leaves
// queue on the root's and the top cells' addresses: 6.14 ms for 1,000,003
// points of 4 values.  Here the sums are combined on chip first.  Each lane
// walks one leaf's path; the lanes of a warp climb together, deepest node
// first, so that all leaves below a node are at it in the same step: they are
// summed with shuffles, one lane adds the sum to the node and goes on alone to
// the parent.  Once a warp is down to one path (a few levels up, for leaves in
// code order) it hands that path to the block, whose 32 warps' paths are
// climbed the same way.  A node thus gets one addition per warp, near the root
// one per block of 1024 leaves: the same sums take 31 us (46 MB of values, links
// and sums at 1.5 TB/s; the paths' dependent loads bound it), and their error
// against binary64 sums went from 8.2e-6 to 3.3e-7.  The order of the leaves
// does not matter for the result, only for how early the paths meet.

// Peers' values summed into the lowest lane of each group (all lanes of
// `members` call it; `peers` are the lanes of the caller's group).  The published
// peer reduction of E. Westphal, "Voting and Shuffling to Optimize Atomic
// Operations" (2015): each lane adds the next peer's value, the odd ranks drop out.
template <int kV>
__device__ __forceinline__ void sum_peers(uint32_t members, uint32_t peers, uint32_t lane, float (&v)[kV]) {
  uint32_t rank = __popc(peers & ((1u << lane) - 1u));
  uint32_t above = peers & (0xfffffffeu << lane);
  while (__any_sync(members, above != 0u)) {
    const uint32_t next = static_cast<uint32_t>(__ffs(above));
    const int from = next ? static_cast<int>(next) - 1 : static_cast<int>(lane);
#pragma unroll
    for (int d = 0; d < kV; ++d) {
      const float x = __shfl_sync(members, v[d], from);
      if (next) v[d] += x;
    }
    above &= __ballot_sync(members, (rank & 1u) == 0u);
    rank >>= 1;
  }
}

// Adds v to out (kVec: as one vector operation, out aligned to it).
template <int kV, bool kVec>
__device__ __forceinline__ void add_values(float* out, const float (&v)[kV]) {
  if constexpr (kVec && kV == 4) {
    atomicAdd(reinterpret_cast<float4*>(out), make_float4(v[0], v[1], v[2], v[3]));
  } else if constexpr (kVec && kV == 2) {
    atomicAdd(reinterpret_cast<float2*>(out), make_float2(v[0], v[1]));
  } else {
#pragma unroll
    for (int d = 0; d < kV; ++d) atomicAdd(out + d, v[d]);
  }
}

// The lanes' paths climbed together: lane at node `on` (kUMax: none), `depth`
// links below the end of its path.  Stops early once a single path is left.
template <int kV, bool kVec>
__device__ __forceinline__ void climb_paths(uint32_t lane, uint32_t num_vdim, uint32_t num_link,
                                            const uint32_t* __restrict__ onodes, float* out, bool stop_at_one,
                                            uint32_t& on, uint32_t& depth, float (&v)[kV]) {
  constexpr uint32_t kAll = 0xffffffffu;
  for (;;) {
    const uint32_t active = __ballot_sync(kAll, on != kUMax);
    if (active == 0u || (stop_at_one && (active & (active - 1u)) == 0u)) return;
    const uint32_t top = __reduce_max_sync(kAll, on != kUMax ? depth + 1u : 0u);
    const bool here = on != kUMax && depth + 1u == top;
    const uint32_t members = __ballot_sync(kAll, here);
    if (here) {
      const uint32_t peers = __match_any_sync(members, on);
      sum_peers<kV>(members, peers, lane, v);
      if (lane == static_cast<uint32_t>(__ffs(peers)) - 1u) {
        add_values<kV, kVec>(out + static_cast<size_t>(on) * num_vdim, v);
        on = depth == 0u ? kUMax : __ldg(onodes + static_cast<size_t>(on) * num_link);
        --depth;  // unused once the path has ended
      } else {
        on = kUMax;
      }
    }
  }
}

constexpr int kAggThreads = 1024;

// Dimensions off .. off + kV - 1 of the values.
template <int kV, bool kVec>
__global__ void __launch_bounds__(kAggThreads) k_aggregate(uint32_t num_idx, uint32_t num_vdim, uint32_t off,
                                                          const float* __restrict__ idx2val,
                                                          const uint32_t* __restrict__ idx2onode, uint32_t num_link,
                                                          const uint32_t* __restrict__ onodes, uint32_t num_onode,
                                                          float* onode2aggval, uint32_t* status) {
  __shared__ uint32_t sh_on[32], sh_depth[32];
  __shared__ float sh_v[32][kV];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t idx = blockIdx.x * kAggThreads + threadIdx.x;
  uint32_t on = idx < num_idx ? __ldg(idx2onode + idx) : kUMax;
  float v[kV];
#pragma unroll
  for (int d = 0; d < kV; ++d) v[d] = 0.0f;
  uint32_t depth = 0;
  if (on != kUMax) {
    const float* val = idx2val + static_cast<size_t>(idx) * num_vdim + off;
    if constexpr (kVec && kV == 4) {
      const float4 x = __ldg(reinterpret_cast<const float4*>(val));
      v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
    } else {
#pragma unroll
      for (int d = 0; d < kV; ++d) v[d] = __ldg(val + d);
    }
    // the links from the leaf's node to the root; a link out of range ends the
    // path, and a walk longer than the tree has nodes (a cycle) drops it
    if (on >= num_onode) {
      raise_status(status, kStatusBadIndex);
      on = kUMax;
    } else {
      for (uint32_t cur = on;;) {
        cur = __ldg(onodes + static_cast<size_t>(cur) * num_link);
        if (cur == kUMax) break;
        if (cur >= num_onode || depth >= num_onode) {
          raise_status(status, kStatusBadIndex);
          if (cur < num_onode) on = kUMax;
          break;
        }
        ++depth;
      }
    }
  }
  float* out = onode2aggval + off;
  climb_paths<kV, kVec>(lane, num_vdim, num_link, onodes, out, true, on, depth, v);
  // what the warp has left: one path or none
  const uint32_t left = __ballot_sync(0xffffffffu, on != kUMax);
  if (left == 0u ? lane == 0u : on != kUMax) {
    sh_on[warp] = on;
    sh_depth[warp] = depth;
#pragma unroll
    for (int d = 0; d < kV; ++d) sh_v[warp][d] = v[d];
  }
  __syncthreads();
  if (warp != 0u) return;
  on = sh_on[lane];
  depth = sh_depth[lane];
#pragma unroll
  for (int d = 0; d < kV; ++d) v[d] = sh_v[lane][d];
  climb_paths<kV, kVec>(lane, num_vdim, num_link, onodes, out, false, on, depth, v);
}

template <int kV>
void launch_aggregate_dims(cudaStream_t s, uint32_t num_idx, uint32_t num_vdim, uint32_t off, const float* idx2val,
                           const uint32_t* idx2onode, uint32_t num_link, const uint32_t* onodes, uint32_t num_onode,
                           float* out, uint32_t* status) {
  const uint32_t grid = (num_idx + kAggThreads - 1) / kAggThreads;
  const uintptr_t at = reinterpret_cast<uintptr_t>(idx2val + off) | reinterpret_cast<uintptr_t>(out + off);
  // rows of whole, aligned vectors are read and added as vectors
  const bool vec = (kV == 2 || kV == 4) && num_vdim % kV == 0 && at % (kV * sizeof(float)) == 0;
  if (vec)
    k_aggregate<kV, true><<<grid, kAggThreads, 0, s>>>(num_idx, num_vdim, off, idx2val, idx2onode, num_link, onodes,
                                                       num_onode, out, status);
  else
    k_aggregate<kV, false><<<grid, kAggThreads, 0, s>>>(num_idx, num_vdim, off, idx2val, idx2onode, num_link, onodes,
                                                        num_onode, out, status);
}

inline uint32_t grid_of(uint32_t n) { return (n + kThreads - 1) / kThreads; }

}  // namespace

size_t octree_scratch_bytes(uint32_t num_idx) {
  const uint32_t num_bnode = num_idx > 0 ? num_idx - 1 : 0;
  return (static_cast<size_t>((num_bnode + kScanTile - 1) / kScanTile) + 1) * 4 + 256;
}

void launch_octree_brt(cudaStream_t s, uint32_t num_idx, const uint32_t* idx2morton, uint32_t num_dim,
                       uint32_t max_depth, uint32_t* bnodes, uint32_t* bnode2depth, uint32_t* bnode2onode,
                       uint32_t* idx2bnode, uint32_t* tile_sums, uint32_t* status) {
  const uint32_t num_bnode = num_idx - 1;
  if (num_bnode == 0) return;
  const uint32_t tiles = (num_bnode + kScanTile - 1) / kScanTile;
  k_brt_depth<<<grid_of(num_bnode), kThreads, 0, s>>>(num_bnode, idx2morton, num_dim, max_depth, bnodes,
                                                       bnode2depth);
  k_onode_count<<<tiles, kThreads, 0, s>>>(num_bnode, bnodes, bnode2depth, idx2bnode, tile_sums, status);
  k_onode_scan<<<1, 1024, 0, s>>>(tiles, tile_sums);
  k_onode_write<<<tiles, kThreads, 0, s>>>(num_bnode, bnodes, bnode2depth, tile_sums, bnode2onode, status);
}

void launch_octree_make(cudaStream_t s, uint32_t num_idx, const uint32_t* bnodes, const uint32_t* bnode2onode,
                        const uint32_t* bnode2depth, const uint32_t* idx2bnode, const uint32_t* idx2morton,
                        uint32_t num_onode, uint32_t max_depth, uint32_t num_dim, uint32_t* onodes,
                        uint32_t* onode2depth, float* onode2center, uint32_t* idx2onode, float* idx2center,
                        uint32_t* status) {
  if (num_idx == 0) return;
  k_make_tree<<<grid_of(num_idx), kThreads, 0, s>>>(num_idx, bnodes, bnode2onode, bnode2depth, idx2bnode, idx2morton,
                                                     num_onode, max_depth, num_dim, onodes, onode2depth, onode2center,
                                                     idx2onode, idx2center, status);
}

void launch_octree_aggregate(cudaStream_t s, uint32_t num_idx, uint32_t num_vdim, const float* idx2val,
                             const uint32_t* idx2onode, uint32_t num_link, const uint32_t* onodes, uint32_t num_onode,
                             float* onode2aggval, uint32_t* status) {
  if (num_idx == 0 || num_vdim == 0) return;
  for (uint32_t off = 0; off < num_vdim; off += 4) {
    const uint32_t left = num_vdim - off;
    if (left >= 4)
      launch_aggregate_dims<4>(s, num_idx, num_vdim, off, idx2val, idx2onode, num_link, onodes, num_onode,
                               onode2aggval, status);
    else if (left == 3)
      launch_aggregate_dims<3>(s, num_idx, num_vdim, off, idx2val, idx2onode, num_link, onodes, num_onode,
                               onode2aggval, status);
    else if (left == 2)
      launch_aggregate_dims<2>(s, num_idx, num_vdim, off, idx2val, idx2onode, num_link, onodes, num_onode,
                               onode2aggval, status);
    else
      launch_aggregate_dims<1>(s, num_idx, num_vdim, off, idx2val, idx2onode, num_link, onodes, num_onode,
                               onode2aggval, status);
  }
}

}  // namespace dm
