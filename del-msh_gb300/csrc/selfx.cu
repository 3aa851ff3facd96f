// selfx.cu — self-intersection of a triangle mesh through its BVH
// (trimesh3_intersection.rs:1-179: search_with_bvh_inside_branch and
// search_with_bvh_between_branches).  The recursion inside(root) visits, at
// every branch n, between(left(n), right(n)) and recurses; so the pairs are
// exactly the union over branches n of between(left(n), right(n)).  Warps
// take start pairs and search them 32 node pairs at a time from a stack in
// shared memory, in rounds: a warp that still has pairs when the round's start
// pairs have run out hands them to the next round, so that the few large
// subtree pairs near the root spread over all warps instead of one.
// Every unordered pair of leaves meets at exactly one branch (their
// lowest common ancestor), with the triangle of the left subtree first, as
// in the recursion; only the order of the output list differs.
//
// Triangle pairs (trimesh3_intersection.rs:10-79): no shared vertex -> the
// segment where the two triangles cross; one shared vertex -> the segment
// from the shared vertex to where an opposite edge pierces the other
// triangle; two shared vertices -> none (three -> none here; the reference
// panics).  The segment formulas of del-geo-core are restated:
// - tri/tri: each triangle's crossing segment with the other's plane (edge
//   crossings v_i + (v_j - v_i) d_i / (d_i - d_j), plus vertices on the
//   plane), both projected on the planes' common direction n_a x n_b, and
//   their overlap [max of starts, min of ends], reported when of non-zero
//   length; coplanar pairs are not reported;
// - shared vertex: Moller-Trumbore of the opposite edge of one triangle (as
//   a segment, 0 <= t <= 1) against the other, first (q1, q2) against the
//   first triangle, then (p1, p2) against the second.
#include "dm_device.cuh"
#include "dm_internal.h"

namespace dm {
namespace {

constexpr int kThreads = 128;

__device__ __forceinline__ float3 lerp_cross(float3 vi, float3 vj, float di, float dj) {
  const float s = __fdiv_rn(di, __fsub_rn(di, dj));
  return make_float3(__fadd_rn(vi.x, __fmul_rn(__fsub_rn(vj.x, vi.x), s)),
                     __fadd_rn(vi.y, __fmul_rn(__fsub_rn(vj.y, vi.y), s)),
                     __fadd_rn(vi.z, __fmul_rn(__fsub_rn(vj.z, vi.z), s)));
}

// The segment where triangle v crosses the plane with signed distances d.
__device__ __forceinline__ bool plane_segment(const float3 v[3], const float d[3], float3& s0, float3& s1) {
  float3 pts[4];
  int n = 0;
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (d[k] == 0.0f) pts[n++] = v[k];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int i = k, j = (k + 1) % 3;
    if ((d[i] > 0.0f && d[j] < 0.0f) || (d[i] < 0.0f && d[j] > 0.0f)) pts[n++] = lerp_cross(v[i], v[j], d[i], d[j]);
  }
  if (n < 2) return false;
  s0 = pts[0];
  s1 = pts[1];
  return true;
}

__device__ __forceinline__ bool tri_tri_segment(const float3 a[3], const float3 b[3], float3& p0, float3& p1) {
  const float3 nb = cross3(sub3(b[1], b[0]), sub3(b[2], b[0]));
  const float db = -dot3(nb, b[0]);
  float da[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) da[k] = __fadd_rn(dot3(nb, a[k]), db);
  if ((da[0] > 0.0f && da[1] > 0.0f && da[2] > 0.0f) || (da[0] < 0.0f && da[1] < 0.0f && da[2] < 0.0f)) return false;
  if (da[0] == 0.0f && da[1] == 0.0f && da[2] == 0.0f) return false;
  const float3 na = cross3(sub3(a[1], a[0]), sub3(a[2], a[0]));
  const float dA = -dot3(na, a[0]);
  float dbv[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) dbv[k] = __fadd_rn(dot3(na, b[k]), dA);
  if ((dbv[0] > 0.0f && dbv[1] > 0.0f && dbv[2] > 0.0f) || (dbv[0] < 0.0f && dbv[1] < 0.0f && dbv[2] < 0.0f))
    return false;
  float3 sa0, sa1, sb0, sb1;
  if (!plane_segment(a, da, sa0, sa1) || !plane_segment(b, dbv, sb0, sb1)) return false;
  const float3 D = cross3(na, nb);
  float ta0 = dot3(D, sa0), ta1 = dot3(D, sa1), tb0 = dot3(D, sb0), tb1 = dot3(D, sb1);
  if (ta1 < ta0) {
    const float3 t = sa0;
    sa0 = sa1;
    sa1 = t;
    const float x = ta0;
    ta0 = ta1;
    ta1 = x;
  }
  if (tb1 < tb0) {
    const float3 t = sb0;
    sb0 = sb1;
    sb1 = t;
    const float x = tb0;
    tb0 = tb1;
    tb1 = x;
  }
  const float lo = ta0 >= tb0 ? ta0 : tb0, hi = ta1 <= tb1 ? ta1 : tb1;
  if (!(lo < hi)) return false;
  p0 = ta0 >= tb0 ? sa0 : sb0;
  p1 = ta1 <= tb1 ? sa1 : sb1;
  return true;
}

// Segment (e0, e1) against triangle (t0, t1, t2): Moller-Trumbore with
// 0 <= t <= 1, inclusive edges.
__device__ __forceinline__ bool edge_tri(float3 e0, float3 e1, float3 t0, float3 t1, float3 t2, float3& x) {
  float t, u, v;
  const float3 dir = sub3(e1, e0);
  if (!tri_ray(t0, t1, t2, e0, dir, t, u, v) || !(t <= 1.0f)) return false;
  x = make_float3(__fadd_rn(e0.x, __fmul_rn(t, dir.x)), __fadd_rn(e0.y, __fmul_rn(t, dir.y)),
                  __fadd_rn(e0.z, __fmul_rn(t, dir.z)));
  return true;
}

__device__ __forceinline__ bool tri_pair(const MeshView& m, uint32_t it, uint32_t jt, float3& p0, float3& p1,
                                         uint32_t* status) {
  if (it == jt) return false;
  if (it >= m.num_tri || jt >= m.num_tri) {
    raise_status(status, kStatusBadIndex);
    return false;
  }
  uint32_t vi[3], vj[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    vi[k] = __ldg(m.tri2vtx + static_cast<size_t>(it) * 3 + k);
    vj[k] = __ldg(m.tri2vtx + static_cast<size_t>(jt) * 3 + k);
    if (vi[k] >= m.num_vtx || vj[k] >= m.num_vtx) {
      raise_status(status, kStatusBadIndex);
      return false;
    }
  }
  bool ci[3], cj[3];
  int shared = 0, si = 0, sj = 0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    ci[k] = vi[k] == vj[0] || vi[k] == vj[1] || vi[k] == vj[2];
    cj[k] = vj[k] == vi[0] || vj[k] == vi[1] || vj[k] == vi[2];
    shared += ci[k] ? 1 : 0;
  }
  if (shared >= 2) return false;
  float3 a[3], b[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    a[k] = load_vtx(m.vtx2xyz, vi[k]);
    b[k] = load_vtx(m.vtx2xyz, vj[k]);
  }
  if (shared == 0) return tri_tri_segment(a, b, p0, p1);
  si = ci[0] ? 0 : (ci[1] ? 1 : 2);
  sj = cj[0] ? 0 : (cj[1] ? 1 : 2);
  const float3 s = a[si], pa = a[(si + 1) % 3], pb = a[(si + 2) % 3];
  const float3 qa = b[(sj + 1) % 3], qb = b[(sj + 2) % 3];
  float3 x;
  if (edge_tri(qa, qb, s, pa, pb, x) || edge_tri(pa, pb, s, qa, qb, x)) {
    p0 = s;
    p1 = x;
    return true;
  }
  return false;
}

struct Box6 {
  float2 a, b, c;  // lo.x lo.y | lo.z hi.x | hi.y hi.z
};

// kVec: the box array is 8-byte aligned, as boxes of 24 bytes then are.
template <bool kVec>
__device__ __forceinline__ Box6 load_box(const float* aabb, uint32_t n) {
  const float* f = aabb + static_cast<size_t>(n) * 6;
  if constexpr (kVec) {
    const float2* p = reinterpret_cast<const float2*>(f);
    return Box6{__ldg(p), __ldg(p + 1), __ldg(p + 2)};
  } else {
    return Box6{make_float2(__ldg(f), __ldg(f + 1)), make_float2(__ldg(f + 2), __ldg(f + 3)),
                make_float2(__ldg(f + 4), __ldg(f + 5))};
  }
}

__device__ __forceinline__ bool overlap6(const Box6& p, const Box6& q) {
  return p.a.x <= q.b.y && q.a.x <= p.b.y && p.a.y <= q.c.x && q.a.y <= p.c.x && p.b.x <= q.c.y && q.b.x <= p.c.y;
}

__device__ __forceinline__ void report_pair(const MeshView& m, uint32_t a0, uint32_t b0, uint32_t capacity,
                                            uint32_t* pairs, float* segments, uint32_t* count, uint32_t* status) {
  float3 p0, p1;
  if (!tri_pair(m, a0, b0, p0, p1, status)) return;
  const uint32_t slot = atomicAdd(count, 1u);
  if (slot >= capacity) return;
  pairs[static_cast<size_t>(slot) * 2] = a0;
  pairs[static_cast<size_t>(slot) * 2 + 1] = b0;
  float* sg = segments + static_cast<size_t>(slot) * 6;
  sg[0] = p0.x;
  sg[1] = p0.y;
  sg[2] = p0.z;
  sg[3] = p1.x;
  sg[4] = p1.y;
  sg[5] = p1.z;
}

// One warp searches with one stack of node pairs in shared memory: each step
// pops up to 32 pairs, one per lane, and pushes the child pairs whose boxes
// overlap.  A pair of leaves goes to a small buffer, tested 32 at a time, so
// that the long triangle test never runs for a few lanes.  What bounds it is
// the dependent round trips of a step (records, then boxes), hidden by the 32
// resident warps per SM.  A search by single threads, each with a stack of its
// own in local memory, ran eight rounds of 500 us whose ends were a few long
// threads: 4.24 ms for two crossing tori of 260,084 triangles in all, against
// 0.33 ms for the four rounds here.
constexpr uint32_t kWarpsPerBlock = kThreads / 32;
constexpr uint32_t kPairStack = 704;   // node pairs on a warp's stack (784 cost two crossing tori 2%)
constexpr uint32_t kWideStack = 512;   // of them while pairs are popped several at a time
constexpr uint32_t kLeafBuffer = 64;   // leaf pairs waiting for their test
// Every so many steps a warp looks whether the round's start pairs are all
// given out; if so warps are running idle, and it hands its own pairs to the
// next round, where they are dealt out anew.  The subtree pairs near the root,
// which hold most of the work, are split this way.  The whole query with its Python
// side took 1.49, 1.18, 1.03 and 1.08 ms for 8, 16, 32 and 64 steps.
constexpr uint32_t kRoundSteps = 32;

// Looks without handing over after which a warp counts its pairs for all, and
// after which it hands over although others are still busy: a search that does
// not end shows in the one or in the number of rounds.  (Every warp adding its
// count once a round cost two crossing tori 18 us of 380.)
constexpr uint32_t kCountLooks = 64, kAloneLooks = 2048;

// A warp whose next list is full goes on alone, and must not run out of stack:
// popping 32 pairs whose boxes all overlap pushes up to 128.  From then on it pops
// a twelfth of what is left below kWideStack, 1 at the least, which settles at
// some 10 pairs a step where everything overlaps everything (a host model of the
// stack; a third of what is left settles at 2).  The 192 entries above kWideStack
// hold 64 levels of a search by single pairs, each of which leaves three behind.
constexpr uint32_t kNarrowPart = 12;
static_assert((kPairStack - kWideStack) / 3 >= 64, "levels of a search by single pairs");

// A round's start pairs are `start[0 .. *num_start)`, or without a list the
// children (left(n), right(n)) of every branch n.
struct RoundList {
  const uint2* start;
  const uint32_t* num_start;
  uint32_t* take;      // start pairs given out
  uint2* next;         // the next round's list
  uint32_t* num_next;
  uint32_t next_cap;
  // pairs popped by searches that go on for long, and how many there can be: a
  // tree has each pair of nodes once, so a search beyond that does not end (a cycle)
  unsigned long long* popped;
  unsigned long long most;
};

// Moves the `k` bottom pairs of the stack, those with the most below them, to the
// next round's list: all of them while the list is less than half full, else none,
// or with `some` a small part of what is free, so that every warp that is still
// busy at the end of a round finds room for its largest pairs, look after look
// (131,072 triangles whose boxes all overlap, 8.6e9 pairs of leaves: 14.8 s with
// whole stacks or nothing up to the end of the list, as the last warps of a round
// then search on alone, and 0.43 s so).  Returns how many.
__device__ __forceinline__ uint32_t hand_over(const RoundList& rl, uint2* stack, uint32_t& sp, uint32_t k, bool some,
                                              uint32_t lane) {
  uint32_t at = 0, got = 0;
  if (lane == 0) {
    // a reservation that would pass the end is refused by compare-and-swap, so
    // that the list has no unwritten holes (a bounded number of attempts)
    const uint32_t half = rl.next_cap / 2;
    uint32_t cur = *reinterpret_cast<volatile uint32_t*>(rl.num_next);
    for (int attempt = 0; attempt < 64; ++attempt) {
      uint32_t n = k;
      if (cur > half || k > half - cur)
        n = some ? min(min(k, (rl.next_cap - cur + 65535u) / 65536u), rl.next_cap - cur) : 0u;
      if (n == 0) break;
      const uint32_t seen = atomicCAS(rl.num_next, cur, cur + n);
      if (seen == cur) {
        at = cur;
        got = n;
        break;
      }
      cur = seen;
    }
  }
  at = __shfl_sync(0xffffffffu, at, 0);
  got = __shfl_sync(0xffffffffu, got, 0);
  if (got == 0) return 0;
  for (uint32_t q = lane; q < got; q += 32) rl.next[at + q] = stack[q];
  __syncwarp();
  // the rest moves down, 32 pairs at a time (each read before it is overwritten)
  for (uint32_t q = got; q < sp; q += 32) {
    const uint2 v = q + lane < sp ? stack[q + lane] : make_uint2(0, 0);
    __syncwarp();
    if (q + lane < sp) stack[q + lane - got] = v;
    __syncwarp();
  }
  sp -= got;
  return got;
}

template <bool kVec>
__global__ void __launch_bounds__(kThreads, 8) k_selfx_round(MeshView m, RoundList rl, uint32_t capacity,
                                                            uint32_t* pairs, float* segments, uint32_t* count,
                                                            uint32_t* status) {
  __shared__ uint2 sh_stack[kWarpsPerBlock][kPairStack];
  __shared__ uint2 sh_leaf[kWarpsPerBlock][kLeafBuffer];
  constexpr uint32_t kAll = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
  uint2* stack = sh_stack[warp];
  uint2* leaf = sh_leaf[warp];
  const uint32_t num_node = 2 * m.num_tri - 1;
  const uint32_t num_start = rl.start ? *rl.num_start : m.num_tri - 1;
  // start pairs are dealt out a few at a time (8 against 32: 0.95 against 1.03 ms,
  // as fewer warps end with much left), and one by one when there are few
  const uint32_t chunk = min(8u, max(1u, num_start / (gridDim.x * kWarpsPerBlock)));
  uint32_t sp = 0, nleaf = 0, steps = 0, alone = 0, popped = 0;
  bool bad = __any_sync(kAll, *reinterpret_cast<volatile unsigned long long*>(rl.popped) > rl.most);
  bool more = num_start > 0 && !bad, full = false;  // full: the next list had no room
  for (;;) {
    bool live = false;  // this lane holds a pair of branches, or of a branch and a leaf
    uint32_t a = 0, b = 0, a0 = 0, a1 = 0, b0 = 0, b1 = 0;
    if (more && sp < chunk) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(rl.take, chunk);
      base = __shfl_sync(kAll, base, 0);
      if (base >= num_start || base + chunk < base) {
        more = false;
        continue;
      }
      bool mine = lane < chunk && base + lane < num_start;
      if (mine) {
        if (rl.start) {
          const uint2 pr = rl.start[base + lane];
          a = pr.x;
          b = pr.y;
        } else {
          a = __ldg(m.bvhnodes + static_cast<size_t>(base + lane) * 3 + 1);
          b = __ldg(m.bvhnodes + static_cast<size_t>(base + lane) * 3 + 2);
        }
        if (a >= num_node || b >= num_node) {
          bad = true;
          mine = false;
        }
      }
      const bool keep = mine && overlap6(load_box<kVec>(m.aabb, a), load_box<kVec>(m.aabb, b));
      const uint32_t mask = __ballot_sync(kAll, keep);
      if (keep) stack[sp + __popc(mask & lt)] = make_uint2(a, b);
      sp += __popc(mask);  // sp < chunk <= 32 before, so there is room
      __syncwarp();
      continue;
    }
    if (sp == 0) break;
    if (steps >= kRoundSteps) {
      steps = 0;
      // while start pairs are left no warp is idle, and there is nothing to
      // split; a search of this length without an end (a tree with a cycle,
      // for which the rounds are the bound) is handed over all the same
      uint32_t taken = 0;
      bool endless = false;
      if (lane == 0) taken = *reinterpret_cast<volatile uint32_t*>(rl.take);
      if (alone >= kCountLooks) {
        if (lane == 0) endless = atomicAdd(rl.popped, static_cast<unsigned long long>(popped)) + popped > rl.most;
        popped = 0;
        if (__any_sync(kAll, endless)) {
          bad = true;
          break;
        }
      }
      taken = __shfl_sync(kAll, taken, 0);
      if ((taken >= num_start || alone >= kAloneLooks) && hand_over(rl, stack, sp, sp, true, lane) != 0) {
        alone = popped = 0;
        full = full && sp + 96 > kWideStack;
        continue;
      }
      ++alone;
    }
    ++steps;
    // a popped pair leaves room for at most four, so 32 are popped only while the
    // stack takes their children; before that its older half is handed on
    if (sp + 96 > kWideStack && !full) full = hand_over(rl, stack, sp, sp / 2, false, lane) == 0;
    const uint32_t narrow = sp < kWideStack ? max(1u, (kWideStack - sp) / kNarrowPart) : 1u;
    const uint32_t k = min(full ? min(32u, narrow) : 32u, sp);
    popped += k;
    if (lane < k) {
      const uint2 pr = stack[sp - 1 - lane];
      a = pr.x;
      b = pr.y;
      const uint32_t* ra = m.bvhnodes + static_cast<size_t>(a) * 3;
      const uint32_t* rb = m.bvhnodes + static_cast<size_t>(b) * 3;
      a0 = __ldg(ra + 1);
      a1 = __ldg(ra + 2);
      b0 = __ldg(rb + 1);
      b1 = __ldg(rb + 2);
      live = true;
    }
    sp -= k;
    __syncwarp();
    const bool la = a1 == kUMax, lb = b1 == kUMax;
    const uint32_t lmask = __ballot_sync(kAll, live && la && lb);
    if (live && la && lb) {
      leaf[nleaf + __popc(lmask & lt)] = make_uint2(a0, b0);
      live = false;
    }
    nleaf += __popc(lmask);  // at most 31 before this step
    // the two (or one) nodes on each side and the overlaps among them
    bool push[4] = {false, false, false, false};
    const uint32_t xa[2] = {la ? a : a0, a1}, xb[2] = {lb ? b : b0, b1};
    if (live) {
      if (xa[0] >= num_node || xb[0] >= num_node || (!la && a1 >= num_node) || (!lb && b1 >= num_node)) {
        bad = true;
        live = false;
      }
    }
    if (live) {
      const Box6 p0 = load_box<kVec>(m.aabb, xa[0]), q0 = load_box<kVec>(m.aabb, xb[0]);
      const Box6 p1 = la ? p0 : load_box<kVec>(m.aabb, a1), q1 = lb ? q0 : load_box<kVec>(m.aabb, b1);
      push[0] = overlap6(p0, q0);
      push[1] = !la && overlap6(p1, q0);
      push[2] = !lb && overlap6(p0, q1);
      push[3] = !la && !lb && overlap6(p1, q1);
    }
    if (sp + 4 * k > kPairStack) {  // a search by single pairs; beyond 64 levels of it
      uint32_t total = 0;
#pragma unroll
      for (int c = 0; c < 4; ++c) total += __popc(__ballot_sync(kAll, push[c]));
      if (sp + total > kPairStack) {
        if (lane == 0) raise_status(status, kStatusStackOverflow);
        sp = 0;
        push[0] = push[1] = push[2] = push[3] = false;
      }
    }
    // pushed in reverse of the recursion's order
#pragma unroll
    for (int c = 3; c >= 0; --c) {
      const uint32_t mask = __ballot_sync(kAll, push[c]);
      if (push[c]) stack[sp + __popc(mask & lt)] = make_uint2(xa[c & 1], xb[c >> 1]);
      sp += __popc(mask);
    }
    __syncwarp();
    if (nleaf >= 32) {
      nleaf -= 32;
      const uint2 pr = leaf[nleaf + lane];
      report_pair(m, pr.x, pr.y, capacity, pairs, segments, count, status);
      __syncwarp();
    }
  }
  if (lane < nleaf) {
    const uint2 pr = leaf[lane];
    report_pair(m, pr.x, pr.y, capacity, pairs, segments, count, status);
  }
  if (bad) raise_status(status, kStatusBadIndex);
}

}  // namespace

namespace {

// The rounds have run out with pairs left.
__global__ void k_selfx_unfinished(uint32_t* status) { raise_status(status, kStatusStackOverflow); }

constexpr uint32_t kRounds = 64;       // rounds between two clearings of the counters
constexpr size_t kHeaderBytes = 1024;  // [start pairs given out, length of the list] per round, pairs popped

int round_grid() {
  static int cached[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (cached[dev] == 0) {
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_selfx_round<true>, kThreads, 0);
    cached[dev] = (sms > 0 ? sms : 152) * (per_sm > 0 ? per_sm : 1);
  }
  return cached[dev];
}

}  // namespace

size_t self_intersection_scratch_bytes(uint32_t num_tri) {
  const uint64_t cap = num_tri < (1u << 20) ? (1u << 20) : num_tri;  // start pairs per round
  return kHeaderBytes + 2 * cap * sizeof(uint2);
}

int launch_self_intersection(cudaStream_t s, const MeshView& m, uint32_t capacity, uint32_t* pairs, float* segments,
                             uint32_t* count, void* scratch, size_t scratch_bytes, uint32_t* status) {
  if (m.num_tri < 2) return 0;
  uint32_t* counters = static_cast<uint32_t*>(scratch);  // 2 * kRounds words and the last list's length
  static_assert((2 * kRounds + 2) * sizeof(uint32_t) <= kHeaderBytes - 8, "counters");
  const uint64_t cap = (scratch_bytes - kHeaderBytes) / (2 * sizeof(uint2));
  uint2* list[2] = {reinterpret_cast<uint2*>(static_cast<char*>(scratch) + kHeaderBytes), nullptr};
  list[1] = list[0] + cap;
  int full = round_grid();
  const uint32_t need = (m.num_tri - 1 + kThreads - 1) / kThreads;
  if (cudaMemsetAsync(counters, 0, kHeaderBytes, s) != cudaSuccess) return -1;
  // Rounds until no warp hands work on.  Each round either finishes its warps'
  // work or splits it, so there are few, but a search down a chain of n links by
  // itself (n equal codes) takes n / kRoundSteps of them; the bound is for trees
  // with cycles.  The length of a round's list stays on the device: kAhead rounds
  // are launched between two looks at it, an empty one costs 2 us and a look 15.
  constexpr uint32_t kAhead = 4;
  const uint32_t max_round = 4000 + m.num_tri / 16 / kAhead * kAhead;
  static_assert(4000 % kAhead == 0, "the last round is looked at");
  for (uint32_t round = 0; round < max_round; ++round) {
    const uint32_t r = round % kRounds;
    if (r == 0 && round > 0) {  // the list's length moves to the front, the rest is cleared
      if (cudaMemcpyAsync(counters + 1, counters + 2 * kRounds + 1, sizeof(uint32_t), cudaMemcpyDeviceToDevice, s) !=
              cudaSuccess ||
          cudaMemsetAsync(counters + 2, 0, 2 * kRounds * sizeof(uint32_t), s) != cudaSuccess ||
          cudaMemsetAsync(counters, 0, 4, s) != cudaSuccess)
        return -1;
    }
    RoundList rl;
    rl.take = counters + 2 * r;
    rl.start = round == 0 ? nullptr : list[(round + 1) & 1];
    rl.num_start = counters + 2 * r + 1;
    rl.next = list[round & 1];
    rl.num_next = counters + 2 * (r + 1) + 1;
    rl.next_cap = static_cast<uint32_t>(cap < 0x7fffffffu ? cap : 0x7fffffffu);
    rl.popped = reinterpret_cast<unsigned long long*>(static_cast<char*>(scratch) + kHeaderBytes - 8);
    rl.most = 2ull * m.num_tri * m.num_tri;
    // the first round of a small mesh has no more warps than start pairs
    const int grid = round == 0 && need < static_cast<uint32_t>(full) ? static_cast<int>(need) : full;
    if (reinterpret_cast<uintptr_t>(m.aabb) % 8 == 0)
      k_selfx_round<true><<<grid, kThreads, 0, s>>>(m, rl, capacity, pairs, segments, count, status);
    else
      k_selfx_round<false><<<grid, kThreads, 0, s>>>(m, rl, capacity, pairs, segments, count, status);
    if (round % kAhead == kAhead - 1) {
      uint32_t n = 0;
      if (cudaMemcpyAsync(&n, rl.num_next, sizeof(uint32_t), cudaMemcpyDeviceToHost, s) != cudaSuccess) return -1;
      if (cudaStreamSynchronize(s) != cudaSuccess) return -1;
      if (n == 0) return 0;
    }
  }
  k_selfx_unfinished<<<1, 1, 0, s>>>(status);
  return 0;
}

}  // namespace dm
