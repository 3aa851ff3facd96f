// dm_traverse.cuh — closest-hit traversal of an LBVH in del-msh's layout
// (bvhnodes u32[(2T-1)*3] = [parent, left, right], bvhnode2aabb f32[(2T-1)*6]),
// shared by the single-mesh cast (cast.cu) and the batched cast (batch.cu).
//
// The result is, bit for bit, del-msh-cpu's recursive near-first search
// (search_bvh3.rs:103-221): at a branch the child with the smaller
// (t_enter, t_exit) tuple is searched first; the far child is skipped when the
// near result exists and the far box is missed or entered beyond it; and of
// two results the far one wins unless the near one is strictly closer.
//
// Iterative form.  Call R(n) the recursive result of node n.  "Pick" (keep
// the later of two results unless the earlier is strictly closer) is
// associative, so a run of picks is the last closest result in visit order.
// Only a branch whose two child boxes are both hit and whose near child is a
// branch needs a frame: it holds the far child, its slab entry, and the result
// accumulated so far at the enclosing level ("saved"), and the accumulator
// restarts empty, so that when the near subtree is finished the accumulator
// equals R(near) exactly — the value the far-child test of
// search_bvh3.rs:168-189 needs.  When only one child box is hit, R(n) is that
// child's result and the descent continues without a frame; a leaf near child
// is resolved inline; a far child that must be searched continues in the
// enclosing level after folding R(near) into "saved".
//
// Link chains.  A "link" branch i has the leaf i (node T-1+i) as left child
// and branch i+1 as right child; a run of k equal Morton codes is a chain of
// k-1 links.  When a link's near child is branch i+1 and both boxes are hit,
// its frame is (far = leaf i, enter, saved); along a descent through
// consecutive links every frame after the first has saved = none, so the
// whole run is kept as one chain frame (first link s, last link t, saved of
// s) and unwound leaf by leaf (t, t-1, ..., s), recomputing each far leaf's
// slab entry.  The stack then grows with the number of runs, not their
// length, and the decisions are exactly those of the uncompressed frames.
//
// Execution.  The traversal is split into phases (entering a branch, testing
// a triangle, popping frames) run by persistent warps: a lane whose ray is
// finished takes the next ray index from a global counter (one atomic per
// warp), so lanes stay busy while long rays finish, and the rarer phases
// wait until several lanes need them (k_cast_persistent).  Frames live in a
// kCastStack-entry on-chip (local) stack.  A second kernel (k_cast_tail) finishes
// what the warps hand over: long rays, parked with their stacks and searched by
// several lanes each (split tier); rays that overflowed the stack or are about to
// enter a long chain, re-cast from scratch by teams of warps that fold chains
// (team tier); and the rare ray whose frames outgrow a team's slice of the global
// pool, re-cast with stacks carved from the whole pool, at last with capacity
// num_tri, which no tree can exceed.  The latter two keep the top 64 frames of
// each stack in an on-chip ring (RingStack) and only its bottom in the pool.
// Duplicate Morton codes produce long chains (a run of k equal codes is a chain of
// height k), which is where the team tier is used.
#pragma once
#include "dm_device.cuh"
#include "dm_internal.h"

namespace dm {

struct Hit {
  float t;
  uint32_t id;  // kUMax == none
};

// Keep `b` (the later result) unless `a` is strictly closer; none is the identity.
__device__ __forceinline__ Hit pick(Hit a, Hit b) {
  if (a.id == kUMax) return b;
  if (b.id == kUMax) return a;
  return (a.t < b.t) ? a : b;
}

struct Ray {
  float3 org, dir, inv;
  bool nz;  // no zero direction component: box tests take slab_nz
};

__device__ __forceinline__ Ray make_ray(float3 o, float3 d) {
  Ray r;
  r.org = o;
  r.dir = d;
  r.inv = make_float3(__fdiv_rn(1.0f, d.x), __fdiv_rn(1.0f, d.y), __fdiv_rn(1.0f, d.z));
  r.nz = d.x != 0.0f && d.y != 0.0f && d.z != 0.0f;
  return r;
}

// Leaf test: search_bvh3.rs:117-128 with dis = +inf.  Out-of-range triangle
// or vertex indices count as a miss and are reported through `bad`.
__device__ __forceinline__ bool leaf_hit(const MeshView& m, const Ray& r, uint32_t it, float& t, float& u, float& v,
                                         bool& bad) {
  if (it >= m.num_tri) {
    bad = true;
    return false;
  }
  const uint32_t* tv = m.tri2vtx + static_cast<size_t>(it) * 3;
  const uint32_t i0 = __ldg(tv), i1 = __ldg(tv + 1), i2 = __ldg(tv + 2);
  if (i0 >= m.num_vtx || i1 >= m.num_vtx || i2 >= m.num_vtx) {
    bad = true;
    return false;
  }
  const float3 p0 = load_vtx(m.vtx2xyz, i0);
  const float3 p1 = load_vtx(m.vtx2xyz, i1);
  const float3 p2 = load_vtx(m.vtx2xyz, i2);
  return tri_ray(p0, p1, p2, r.org, r.dir, t, u, v) && t < INFINITY;
}

__device__ __forceinline__ bool node_slab(const MeshView& m, const Ray& r, uint32_t n, float& te, float& tx) {
  const float* box = m.aabb + static_cast<size_t>(n) * 6;
  return r.nz ? slab_nz(box, r.org, r.inv, te, tx) : slab(box, r.org, r.inv, r.dir, te, tx);
}

struct LocalStack {
  uint4* p;
  __device__ __forceinline__ void store(uint32_t i, uint4 v) const { p[i] = v; }
  __device__ __forceinline__ uint4 load(uint32_t i) const { return p[i]; }
};

// A ray's stack for the overflow tiers: frames [*lo, sp) live in an on-chip
// ring of kRing frames, the frames below *lo in the ray's global area.  The
// traversal only ever reads the top frame and writes the top or the next
// slot, so a push past the ring spills the ring's oldest frame, and reading a
// top that has left the ring (the ring is then empty) brings it back.  Deep
// chains thus push and pop at on-chip latency; only their bottoms go to L2.
template <int kRing>
struct RingStack {
  static_assert((kRing & (kRing - 1)) == 0, "ring size is a power of two");
  uint4* ring;   // kRing on-chip frames
  uint4* glob;   // the ray's global frames (capacity: the tier's cap)
  uint32_t* lo;  // first frame held by the ring
  __device__ __forceinline__ void store(uint32_t i, uint4 v) const {
    if (i >= *lo + kRing) {  // a push past the ring: spill its oldest frame
      __stcg(glob + *lo, ring[*lo & (kRing - 1)]);
      ++*lo;
    }
    if (i >= *lo) ring[i & (kRing - 1)] = v;
    else __stcg(glob + i, v);
  }
  __device__ __forceinline__ uint4 load(uint32_t i) const {
    if (i >= *lo) return ring[i & (kRing - 1)];
    const uint4 v = __ldcg(glob + i);
    ring[i & (kRing - 1)] = v;  // i is the top and the ring is empty: i becomes its only frame
    *lo = i;
    return v;
  }
};

constexpr uint32_t kChainBit = 0x80000000u;  // frame.x flag of a chain frame (node ids are < 2^31)
constexpr uint32_t kGivenBits = 0xC0000000u;  // frame.x of a given frame, with the lane that has it (links are < 2^30)

// Per-ray traversal state between phases.
struct Trav {
  uint32_t node;         // node to enter next
  uint32_t left, right;  // its record (bvhnodes[node*3+1], [node*3+2]), fetched ahead
  uint32_t sp;           // frames in use
  uint32_t steps;        // node entries so far (bounded by the node count)
  uint32_t chain_next;   // the link that would extend the top chain frame, or kUMax
  uint32_t leaf_tri;     // triangle of a pending leaf test
  float far_enter;       // slab entry of the far child that follows a near leaf
  bool leaf_far;         // a far child (node/left/right) follows the pending leaf
  Hit best;              // accumulator of the current level
};

__device__ __forceinline__ void load_record(const uint32_t* __restrict__ bn, uint32_t n, uint32_t& left,
                                            uint32_t& right) {
  left = __ldg(bn + static_cast<size_t>(n) * 3 + 1);
  right = __ldg(bn + static_cast<size_t>(n) * 3 + 2);
}

enum StepResult : int { kStepContinue = 0, kStepDone = 1, kStepOverflow = 2 };

// What a ray does next.  A step of the recursion is split into phases so
// that the lanes of a warp can run each phase together: entering a branch
// (kLaneInner), testing one triangle (kLaneLeaf), and popping frames until a
// far child is to be searched or the ray is finished (kLaneAscend).
enum LaneState : int {
  kLaneIdle = 0,
  kLaneInner = 1,
  kLaneLeaf = 2,
  kLaneAscend = 3,
  kLaneOverflow = 4,  // the on-chip stack is full: the ray is re-cast by a deeper tier
  kLaneDone = 5,      // s.best is the ray's result
  kLaneJoin = 6,      // its next frame was given to another lane, whose result it needs
  kLaneHelped = 7,    // a given frame's result is in s.best
  kLaneParked = 8,    // waits to be parked for the split tier
};

// Chain links: branch j whose left child is leaf j and right child branch
// j + 1 (runs of equal Morton codes build long runs of them).  The team tier
// folds runs of at least kFoldMin links instead of walking them.
constexpr uint32_t kFoldMin = 8;

__device__ __forceinline__ bool is_link(const MeshView& m, uint32_t node, uint32_t left, uint32_t right) {
  return left == m.num_tri - 1 + node && right == node + 1;
}

// Whether a run of at least kFoldMin links starts at branch `node` (its
// record: left, right); the other records are loaded together.
__device__ __forceinline__ bool long_chain_at(const MeshView& m, uint32_t node, uint32_t left, uint32_t right) {
  if (!is_link(m, node, left, right) || node + kFoldMin > m.num_tri - 1) return false;
  bool all = true;
#pragma unroll
  for (uint32_t k = 1; k < kFoldMin; ++k) {
    uint32_t l, r;
    load_record(m.bvhnodes, node + k, l, r);
    all = all && is_link(m, node + k, l, r);
  }
  return all;
}

// Starts a ray: a miss of the root box finishes it immediately.
__device__ __forceinline__ bool trav_begin(const MeshView& m, const Ray& r, Trav& s) {
  s.node = 0;
  s.sp = 0;
  s.steps = 0;
  s.chain_next = kUMax;
  s.leaf_tri = kUMax;
  s.far_enter = 0.f;
  s.leaf_far = false;
  s.best = Hit{INFINITY, kUMax};
  load_record(m.bvhnodes, 0, s.left, s.right);
  float te, tx;
  return node_slab(m, r, 0, te, tx);
}

// Entering node s.node.  A leaf (reached as the root or as a far child)
// becomes a pending test.  A branch tests both child boxes; the records of
// both children are fetched together with their boxes, so descending costs
// one dependent memory round trip per level.  A near leaf becomes a pending
// test with the far child (if its box is hit) parked in s.node/left/right.
// A malformed tree (child index out of range, or more node entries than the
// tree has nodes) finishes the ray and sets `bad`.
template <typename StackT>
__device__ __forceinline__ int phase_inner(const MeshView& m, const Ray& r, StackT stack, uint32_t cap, Trav& s,
                                           bool& bad) {
  const uint32_t* __restrict__ bn = m.bvhnodes;
  const uint32_t num_node = 2 * m.num_tri - 1;
  ++s.steps;
  if (s.right == kUMax) {
    s.leaf_tri = s.left;
    s.leaf_far = false;
    return kLaneLeaf;
  }
  const uint32_t node = s.node, left = s.left, right = s.right;
  if (max(left, right) >= num_node || s.steps > num_node + 1) {
    bad = true;
    return kLaneDone;
  }
  uint32_t ll, lr, rl, rr;
  load_record(bn, left, ll, lr);
  load_record(bn, right, rl, rr);
  float l0 = 0.f, l1 = 0.f, r0 = 0.f, r1 = 0.f;
  const bool hl = node_slab(m, r, left, l0, l1);
  const bool hr = node_slab(m, r, right, r0, r1);
  const bool both = hl && hr;
  const bool near_left = both ? tuple_lt(l0, l1, r0, r1) : hl;
  const uint32_t nn = near_left ? left : right, nf = near_left ? right : left;
  const uint32_t n_l = near_left ? ll : rl, n_r = near_left ? lr : rr;
  const float far_enter = near_left ? r0 : l0;
  const bool near_leaf = n_r == kUMax;  // the near child is a leaf holding triangle n_l
  if (both && !near_leaf) {
    const bool link = !near_left && left == m.num_tri - 1 + node && right == node + 1;
    if (link && node == s.chain_next && s.best.id == kUMax) {
      // extend the chain frame on top: its last link becomes `node`
      const uint4 f = stack.load(s.sp - 1);
      stack.store(s.sp - 1, make_uint4(f.x, node, f.z, f.w));
    } else {
      if (s.sp >= cap) return kLaneOverflow;
      stack.store(s.sp++, make_uint4(link ? kChainBit | node : nf, link ? node : __float_as_uint(far_enter),
                                     __float_as_uint(s.best.t), s.best.id));
    }
    s.chain_next = link ? node + 1 : kUMax;
    s.best = Hit{INFINITY, kUMax};
  }
  // without a far child R(node) == R(near): no pending decision, no frame.
  // What the next phase does not read may be written all the same: the three
  // outcomes then differ by selects and not by branches.
  s.leaf_tri = n_l;
  s.leaf_far = both;
  s.far_enter = far_enter;
  s.node = near_leaf ? nf : nn;
  s.left = near_leaf ? (near_left ? rl : ll) : n_l;
  s.right = near_leaf ? (near_left ? rr : lr) : n_r;
  return hl || hr ? (near_leaf ? kLaneLeaf : kLaneInner) : kLaneAscend;
}

// The pending triangle test.  After a near leaf the far child is searched
// unless the leaf was hit before the far box is entered (search_bvh3.rs:168-189).
__device__ __forceinline__ int phase_leaf(const MeshView& m, const Ray& r, Trav& s, bool& bad) {
  float t, u, v;
  const bool h = leaf_hit(m, r, s.leaf_tri, t, u, v, bad);
  if (h) s.best = pick(s.best, Hit{t, s.leaf_tri});
  if (!s.leaf_far || (h && s.far_enter > t)) return kLaneAscend;
  return kLaneInner;
}

// A frame kind that only the team tier pushes (see ChainFold); elsewhere none.
struct NoFold {
  __device__ __forceinline__ int operator()(const uint4&, Trav&) const { return 0; }
};

// Pops frames until a far child is to be searched (kLaneInner) or the stack
// is empty (kLaneDone).  `fold` consumes the frames of its own kind (1), or
// reports a malformed one (2).  The `given` bottom frames are in the hands of
// other lanes: once the others are popped the lane is at a join (kLaneJoin).
template <typename StackT, typename Fold = NoFold>
__device__ __forceinline__ int phase_ascend(const MeshView& m, const Ray& r, StackT stack, Trav& s, bool& bad,
                                            const Fold& fold = Fold{}, uint32_t given = 0) {
  const uint32_t num_node = 2 * m.num_tri - 1;
  s.chain_next = kUMax;
  while (s.sp > given) {
    const uint4 f = stack.load(s.sp - 1);
    const int folded = fold(f, s);
    if (folded == 1) continue;
    if (folded == 2) {
      bad = true;
      return kLaneDone;
    }
    const Hit saved{__uint_as_float(f.z), f.w};
    uint32_t far;
    float far_enter;
    bool pop = true;
    if (f.x & kChainBit) {
      // level j = f.y of a chain frame: far child = leaf j, saved = none
      // unless j is the chain's first link
      const uint32_t first = f.x & ~kChainBit, j = f.y;
      far = m.num_tri - 1 + j;
      if (far >= num_node) {
        bad = true;
        return kLaneDone;
      }
      float te = 0.f, tx = 0.f;
      node_slab(m, r, far, te, tx);  // hit when the frame was pushed; same value again
      far_enter = te;
      pop = j == first;
      if (pop) --s.sp;
      else stack.store(s.sp - 1, make_uint4(f.x, j - 1, f.z, f.w));
    } else {
      --s.sp;
      far = f.x;
      far_enter = __uint_as_float(f.y);
    }
    // The far test sees R(near) alone (search_bvh3.rs:168-189); only then is
    // the enclosing level's result folded in.  Deciding on the folded value
    // instead agrees only while every hit lies at or beyond its box's entry
    // t, which rounding does not guarantee (a triangle on a box face).
    const bool skip = (s.best.id != kUMax) && far_enter > s.best.t;
    if (pop) s.best = pick(saved, s.best);
    if (!skip) {
      s.node = far;
      if (s.node >= num_node) {
        bad = true;
        return kLaneDone;
      }
      load_record(m.bvhnodes, s.node, s.left, s.right);
      return kLaneInner;
    }
  }
  return given == 0 ? kLaneDone : kLaneJoin;
}

// One node entry and everything up to the next one (the phases back to
// back), for one ray at a time.  On kStepDone the ray's result is s.best.
template <typename StackT>
__device__ __forceinline__ int trav_step(const MeshView& m, const Ray& r, StackT stack, uint32_t cap, Trav& s,
                                         bool& bad) {
  int st = phase_inner(m, r, stack, cap, s, bad);
  if (st == kLaneLeaf) st = phase_leaf(m, r, s, bad);
  if (st == kLaneAscend) st = phase_ascend(m, r, stack, s, bad);
  return st == kLaneInner ? kStepContinue : (st == kLaneOverflow ? kStepOverflow : kStepDone);
}

// Barycentrics of a final hit (recomputed once per ray when asked for).
__device__ __forceinline__ void hit_bc(const MeshView& m, const Ray& r, const Hit& h, float bc[3]) {
  bc[0] = bc[1] = bc[2] = 0.0f;
  if (h.id == kUMax) return;
  float t, u, v;
  bool bad = false;
  if (leaf_hit(m, r, h.id, t, u, v, bad)) {
    bc[0] = __fsub_rn(__fsub_rn(1.0f, u), v);
    bc[1] = u;
    bc[2] = v;
  }
}

constexpr int kCastThreads = 128;
// Node entries per iteration of the persistent loop.  Measured on GB300
// (2M-triangle torus 1920x1080 cast / 4096-mesh batched cast): 1 step 0.528 / 4.94 ms, 2 steps
// 0.480 / 4.61, 3 steps 0.466 / 4.54, 4 steps 0.469 / 5.33, 6 steps 0.561 / 6.20.
constexpr int kInnerSteps = 3;
// Of the split tier's loop (2M torus 1920 x 1080 / 641 x 479 on a 66k torus, parked at 64 entries): 1 step 542 /
// 153 us, 2 steps 514 / 154, 3 steps 513 / 156.
constexpr int kTailSteps = 2;
constexpr int kDeepRing = 64;  // on-chip frames per ray of the overflow tiers

// A Job maps a work index to (mesh, ray, output slot):
//   uint32_t num_work;                              work indices are 0..num_work-1
//   __device__ void prepare(float* smem) const;    once per block, before __syncthreads
//   __device__ bool fetch(uint32_t w, const float* smem, MeshView& m, Ray& r, uint32_t& out) const;
//                                                   false: w is padding, nothing to do
//   __device__ void share(MeshView& m, int from) const;
//                                                   m becomes that of lane `from` (all lanes call it)
//   __device__ void write(uint32_t out, const MeshView& m, const Ray& r, const Hit& h) const;
//   kRefillHalves                                   halves of cast_refill_min at which a warp takes rays
//   kCastRegs                                       registers a thread of the persistent cast

// Thresholds of the phased loop: a phase runs when at least this many lanes
// of the warp wait for it, or when nothing else can run.
struct PhaseMins {
  uint32_t refill, leaf, ascend;
  uint32_t long_steps;  // node entries after which a ray at a long chain goes to the team tier
  uint32_t park_steps;  // node entries after which a ray is parked for the split tier
  uint32_t share;       // rays a warp takes at a time, at most
};

struct Parked {
  uint4* rays;  // per ray: {work, node, left, right}, {sp, steps, best}, the frames
  uint32_t* count;
  uint32_t capacity, stride;
  __device__ __forceinline__ uint32_t work(uint32_t i) const { return rays[static_cast<size_t>(i) * stride].x; }
  // The first of a block's list of rays that the split tier hands over (linked by
  // their second word), or kUMax; by many threads of the block at a time.
  __device__ __forceinline__ uint32_t take_handed(uint32_t* head) const {
    uint32_t i = *reinterpret_cast<volatile uint32_t*>(head);
    while (i != kUMax) {
      const uint32_t seen = atomicCAS(head, i, rays[static_cast<size_t>(i) * stride + 1].x);
      if (seen == i) break;
      i = seen;
    }
    return i;
  }
};

// Persistent warps with per-lane ray refill, run in phases.  Each lane holds
// one ray in a LaneState; per iteration the warp enters up to kInnerSteps
// nodes in every lane that is at a branch, then runs the triangle tests, then the ascents,
// then takes new rays for its idle lanes.  The triangle test, the ascent and
// the refill each happen about once per ray but in some lane nearly every
// iteration, so running them whenever any lane needs one leaves most lanes
// idle through them; waiting until `mins` lanes need one runs each for more
// lanes at once, while the others go on entering nodes.  Every lane still makes
// the same decisions in the same order, so results do not depend on the
// thresholds.  Rays overflowing the on-chip stack, and rays past mins.long_steps
// node entries at a long chain once the warp's work is exhausted, go to ovf_list
// (their work index) for the team tier.  kThreads threads per block and kStack
// on-chip frames per ray are tuning choices (Tuning).  The register bound is the
// job's: the cast waits for loads most of all (a third of its stalls), and 56
// registers keep 36 warps resident where 64 keep 32.  For the batch that pays,
// 64 / 56 / 48 registers: 1220 / 1173 / 1195 us; one mesh's cast spills more and
// is also held by single rays: 2M triangles at 1920 x 1080 431 / 440 / 446 us,
// 16,384 rays 136 / 143 / 144 us.
// With kPark the loop after the work has run out is a second copy of the phases:
// with one loop for both, the parking code cost the first one 100 bytes of spills
// (batched cast 1.26 -> 1.48 ms).  Without it, for a GPU that is busy with other
// requests' kernels (see launch_tiers), one loop does both: with two, a server's
// capacity was 6,220 requests/s, with one it is 7,270 (512 meshes, 8 in flight).
template <typename Job, int kThreads, int kStack, bool kPark>
__global__ void __launch_bounds__(kThreads, 65536 / (Job::kCastRegs * kThreads)) k_cast_persistent(Job job, uint32_t* work_counter,
                                                                                 uint32_t* ovf_list,
                                                                                 uint32_t* ovf_count,
                                                                                 uint32_t* status, PhaseMins mins,
                                                                                 Parked parked) {
  __shared__ float smem[64];
  job.prepare(smem);
  pdl_wait();  // k_cast_begin
  __syncthreads();
  constexpr uint32_t kAll = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t lt_mask = (1u << lane) - 1u;
  uint4 frames[kStack];
  LocalStack stack{frames};
  MeshView m{};
  Ray r{};
  Trav s{};
  uint32_t out = 0, work = kUMax;
  int state = kLaneIdle;
  bool exhausted = false, bad = false;
  for (;;) {
    // refill idle lanes with consecutive work indices
    const uint32_t idle = __ballot_sync(kAll, state == kLaneIdle);
    if (idle != 0u && !exhausted && (idle == kAll || static_cast<uint32_t>(__popc(idle)) >= mins.refill)) {
      const uint32_t take = min(static_cast<uint32_t>(__popc(idle)), mins.share);
      uint32_t base = 0;
      if (lane == static_cast<uint32_t>(__ffs(idle) - 1)) base = atomicAdd(work_counter, take);
      base = __shfl_sync(kAll, base, __ffs(idle) - 1);
      if (base + take >= job.num_work) exhausted = true;  // warp-uniform: no work after this
      const uint32_t rank = __popc(idle & lt_mask);
      if (state == kLaneIdle && rank < take) {
        const uint32_t w = base + rank;
        if (w < job.num_work && job.fetch(w, smem, m, r, out)) {
          work = w;
          if (trav_begin(m, r, s)) state = kLaneInner;
          else job.write(out, m, r, s.best);
        }
      }
    }
    if (kPark && exhausted) break;
    if (__all_sync(kAll, state == kLaneIdle)) {
      if (exhausted) break;
      continue;
    }
    const uint32_t leaf_min = exhausted ? 1u : mins.leaf, ascend_min = exhausted ? 1u : mins.ascend;
    // Up to kInnerSteps node entries per iteration: the warp's votes and
    // phase decisions are paid once for several entries, and a lane that
    // leaves the inner phase early waits for the others' entries.
#pragma unroll
    for (int k = 0; k < kInnerSteps; ++k)
      if (state == kLaneInner) state = phase_inner(m, r, stack, kStack, s, bad);
    uint32_t inner = __ballot_sync(kAll, state == kLaneInner);
    const uint32_t leaf = __ballot_sync(kAll, state == kLaneLeaf);
    if (leaf != 0u && (inner == 0u || static_cast<uint32_t>(__popc(leaf)) >= leaf_min)) {
      if (state == kLaneLeaf) state = phase_leaf(m, r, s, bad);
      inner = __ballot_sync(kAll, state == kLaneInner);
    }
    const uint32_t asc = __ballot_sync(kAll, state == kLaneAscend);
    if (asc != 0u && (inner == 0u || static_cast<uint32_t>(__popc(asc)) >= ascend_min)) {
      if (state == kLaneAscend) state = phase_ascend(m, r, stack, s, bad);
    }
    if (!kPark && exhausted && state == kLaneInner && s.steps > mins.long_steps &&
        long_chain_at(m, s.node, s.left, s.right))
      state = kLaneOverflow;
    if (state == kLaneDone) {
      job.write(out, m, r, s.best);
      state = kLaneIdle;
    } else if (state == kLaneOverflow) {
      ovf_list[atomicAdd(ovf_count, 1u)] = work;
      state = kLaneIdle;
    }
  }
  if constexpr (!kPark) {
    if (bad) raise_status(status, kStatusBadIndex);
    return;
  }
  // The warp has no more rays to take: a waiting lane would only lengthen its
  // longest ray, so every phase runs whenever a lane needs it.  A ray past the
  // step budget that is about to enter a long chain would hold the kernel's end:
  // it is handed to the team tier, which folds chains many links at a time.  One
  // that goes on for long stops here and is parked for the split tier.
  uint32_t park_steps = mins.park_steps;
  for (;;) {
    while (__any_sync(kAll, state == kLaneInner || state == kLaneLeaf || state == kLaneAscend)) {
#pragma unroll
      for (int k = 0; k < kInnerSteps; ++k)
        if (state == kLaneInner) state = phase_inner(m, r, stack, kStack, s, bad);
      if (state == kLaneLeaf) state = phase_leaf(m, r, s, bad);
      if (state == kLaneAscend) state = phase_ascend(m, r, stack, s, bad);
      if (state == kLaneInner && s.steps > mins.long_steps && long_chain_at(m, s.node, s.left, s.right))
        state = kLaneOverflow;
      if (state == kLaneInner && s.steps > park_steps) state = kLaneParked;
      if (state == kLaneDone) {
        job.write(out, m, r, s.best);
        state = kLaneIdle;
      } else if (state == kLaneOverflow) {
        ovf_list[atomicAdd(ovf_count, 1u)] = work;
        state = kLaneIdle;
      }
    }
    if (!__any_sync(kAll, state == kLaneParked)) break;
    if (state == kLaneParked) {
      const uint32_t at = atomicAdd(parked.count, 1u);
      if (at < parked.capacity) {
        uint4* to = parked.rays + static_cast<size_t>(at) * parked.stride;
        to[0] = make_uint4(work, s.node, s.left, s.right);
        to[1] = make_uint4(s.sp, s.steps, __float_as_uint(s.best.t), s.best.id);
        for (uint32_t k = 0; k < s.sp; ++k) to[2 + k] = frames[k];
        state = kLaneIdle;
      } else {
        state = kLaneInner;  // no room: it goes on here
      }
    }
    park_steps = kUMax;
  }
  if (bad) raise_status(status, kStatusBadIndex);
}

// ------------------------------------------------------------ team tier
// Rays that overflowed the persistent cast's stack, or that were about to
// enter a long chain past its step budget once their warp had no more rays to
// take, one team of warps each.  Every lane of a team runs the same serial
// traversal on the same state (the same loads, the same decisions), except at a
// chain: a run of links, branches j whose left child is leaf j and right child
// branch j + 1 (runs of equal Morton codes build them).  The recursion's result
// over a chain c0..c1 is a fold from its far end: with x = F(c1 + 1), for j = c1
// down to c0
//   x <- g_j(x):  neither child box hit: none;  only leaf j's box: h_j (its hit);
//                 only branch j+1's box: x;  both, the leaf nearer: h_j if h_j
//                 is a hit before branch j+1's entry, else pick(h_j, x);  both,
//                 the branch nearer: x if x is a hit before leaf j's entry,
//                 else pick(x, h_j)
// (the rules of phase_inner / phase_leaf / phase_ascend).  So the team pushes
// a fold frame, searches the tail c1 + 1 on its own, and on popping the frame
// tests kFoldLinks links per warp and round, all loads in flight together, and
// applies those that change the result in order.  Most change nothing: a link
// whose branch box is hit and whose leaf holds no hit leaves x as it is.
// On the duplicate-heavy soup 96% of the long rays' node entries are links.
//
// The kernel ends with its longest ray (26,600 links in 17 chains and 100 other
// steps, of 1,048,576 rays in a soup of 4,194,304 triangles), and a round is a
// few dependent trips to DRAM whatever it holds, so what counts is the number
// of rounds.  That soup's cast, three draws: 2.1-3.3 ms with a warp per ray, 32
// links per round and every link shuffled through; 1.06 ms with 128 links and
// only the links that matter; 0.54-0.68 ms with teams of 4 warps that take their
// rays from a counter (0.59-0.69 ms with fixed shares; teams of 8 warps
// 0.71-0.84 ms and of 16 1.08-1.23 ms, fewer of which are resident).  2 links
// per lane or 4 to 16 prefetched groups give the same within 3%.
constexpr uint32_t kWarpAll = 0xffffffffu;
constexpr uint32_t kTeamThreads = 128;
constexpr uint32_t kTeamWarps = kTeamThreads / 32;
constexpr uint32_t kFoldBatch = 2;  // links per lane and round
constexpr uint32_t kFoldLinks = 32 * kFoldBatch;

// A warp's part of a round: the leaves to test and their hits, then the links
// to apply.  Two of the latter, so that a round does not wait for the team to
// finish the one before.
struct FoldShared {
  float t[kFoldLinks];
  uint32_t id[kFoldLinks];
  uint8_t todo[kFoldLinks];
  struct Op {
    float t, enter;
    uint32_t id, flags;
  } op[2][kFoldLinks];
  uint32_t num_op[2];
  uint32_t cut[2];    // the first link to apply does not look at x
  uint32_t first[2];  // chain_last: the first record of the warp's that is no link
};

// The warps that cast one ray together: the whole block, or a warp alone (known when
// compiled: one function for both took 5% longer for a soup's build and cast).  The
// two sides of FoldShared are used in turn over all chains of a ray, so that a warp
// writes a side again only after a meeting of the team that the others reach when
// they have read it.
template <bool kSolo>
struct Team {
  static constexpr uint32_t warps = kSolo ? 1u : kTeamWarps;
  FoldShared* sh;  // the team's first warp's
  uint32_t rank, lane;
  mutable uint32_t scan_side, fold_side;
  __device__ __forceinline__ void sync() const {
    if constexpr (kSolo) __syncwarp();
    else __syncthreads();
  }
};

// The last link of the chain starting at link c0 (the same in every lane of the
// team), 256 records per warp and round (8 per lane).
template <bool kSolo>
__device__ __forceinline__ uint32_t chain_last(const MeshView& m, uint32_t c0, const Team<kSolo>& tm) {
  const uint32_t num_branch = m.num_tri - 1;
  uint32_t last = c0;
  for (;;) {
    const uint32_t side = tm.scan_side;
    tm.scan_side ^= 1u;
    // lane l of warp w checks links last + 1 + 256 w + 8 l and the 7 after it
    const uint32_t base = last + 1 + 256 * tm.rank + 8 * tm.lane;
    bool ok[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      ok[q] = false;
      if (base + q < num_branch) {
        uint32_t l, r;
        load_record(m.bvhnodes, base + q, l, r);
        ok[q] = is_link(m, base + q, l, r);
      }
    }
    uint32_t first_bad = 8;
#pragma unroll
    for (int q = 7; q >= 0; --q)
      if (!ok[q]) first_bad = q;
    const uint32_t fail = __ballot_sync(kWarpAll, first_bad < 8);
    uint32_t mine = 256;  // links of this warp's before the first other record
    if (fail != 0u) {
      const uint32_t l0 = static_cast<uint32_t>(__ffs(fail)) - 1u;
      mine = 8 * l0 + __shfl_sync(kWarpAll, first_bad, l0);
    }
    if constexpr (kSolo) {
      if (mine < 256) return last + mine;
    } else {
      if (tm.lane == 0) tm.sh[tm.rank].first[side] = mine;
      __syncthreads();
      for (uint32_t w = 0; w < tm.warps; ++w) {
        const uint32_t f = tm.sh[w].first[side];
        if (f < 256) return last + 256 * w + f;
      }
    }
    last += 256 * tm.warps;
  }
}

// This warp's n links hi, hi - 1, .. (1 to kFoldLinks of them): tests them and
// leaves those to be applied, in order, in sh.op[side].
__device__ __forceinline__ void test_links(const MeshView& m, const Ray& r, uint32_t hi, uint32_t n, uint32_t lane,
                                           FoldShared& sh, uint32_t side, bool& bad) {
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t flags[kFoldBatch];  // 1: leaf box hit, 2: branch box hit, 4: the leaf is the near child
  float far_enter[kFoldBatch];
  uint32_t ntodo = 0;
#pragma unroll
  for (uint32_t q = 0; q < kFoldBatch; ++q) {
    // past the last link, that one is tested again and ignored
    const uint32_t i = lane + 32 * q, j = hi - (i < n ? i : n - 1);
    float a0 = 0.f, a1 = 0.f, b0 = 0.f, b1 = 0.f;
    const bool ha = node_slab(m, r, m.num_tri - 1 + j, a0, a1);
    const bool hb = node_slab(m, r, j + 1, b0, b1);
    const bool near_leaf = (ha && hb) ? tuple_lt(a0, a1, b0, b1) : ha;
    flags[q] = (ha ? 1u : 0u) | (hb ? 2u : 0u) | (near_leaf ? 4u : 0u);
    far_enter[q] = near_leaf ? b0 : a0;
  }
#pragma unroll
  for (uint32_t q = 0; q < kFoldBatch; ++q) {
    const uint32_t i = lane + 32 * q;
    const bool test = i < n && (flags[q] & 1u);
    const uint32_t mask = __ballot_sync(kWarpAll, test);
    if (test) sh.todo[ntodo + __popc(mask & lt)] = static_cast<uint8_t>(i);
    ntodo += __popc(mask);
  }
  __syncwarp();
  for (uint32_t c = lane; c < ntodo; c += 32) {
    const uint32_t i = sh.todo[c], leaf = m.num_tri - 1 + (hi - i);
    const uint32_t tri = __ldg(m.bvhnodes + static_cast<size_t>(leaf) * 3 + 1);
    float t, u, v;
    const bool h = leaf_hit(m, r, tri, t, u, v, bad);
    sh.t[i] = h ? t : INFINITY;
    sh.id[i] = h ? tri : kUMax;
  }
  __syncwarp();
  uint32_t num = 0, has_cut = 0;
#pragma unroll
  for (uint32_t q = 0; q < kFoldBatch; ++q) {
    const uint32_t i = lane + 32 * q;
    Hit h{INFINITY, kUMax};
    if (i < n && (flags[q] & 1u)) h = Hit{sh.t[i], sh.id[i]};
    const uint32_t cut = __ballot_sync(kWarpAll, i < n && !(flags[q] & 2u));  // links that do not look at x
    uint32_t todo = __ballot_sync(kWarpAll, i < n && (flags[q] & 2u) && h.id != kUMax) | cut;
    if (cut != 0u) {  // what comes before the last of them is lost
      __syncwarp();  // their entries are written over (a ballot orders no memory)
      todo &= 0xffffffffu << (31 - __clz(cut));
      num = 0;
      has_cut = 1;
    }
    if (todo >> lane & 1u)
      sh.op[side][num + __popc(todo & lt)] = FoldShared::Op{h.t, far_enter[q], h.id, flags[q]};
    num += __popc(todo);
  }
  if (lane == 0) {
    sh.num_op[side] = num;
    sh.cut[side] = has_cut;
  }
}

// The links of a round applied to x, the warps' parts from the far end on.
template <bool kSolo>
__device__ __forceinline__ Hit apply_links(const Team<kSolo>& tm, uint32_t side, Hit x) {
  uint32_t w0 = 0;
  for (uint32_t w = 1; w < tm.warps; ++w)
    if (tm.sh[w].cut[side]) w0 = w;
  for (uint32_t w = w0; w < tm.warps; ++w) {
    const uint32_t num = tm.sh[w].num_op[side];
    for (uint32_t k = 0; k < num; ++k) {
      const FoldShared::Op o = tm.sh[w].op[side][k];
      const Hit h{o.t, o.id};
      if ((o.flags & 2u) == 0u) x = h;  // the leaf's hit, or none
      else if (o.flags & 4u) x = o.enter > h.t ? h : pick(h, x);
      else x = (x.id != kUMax && o.enter > x.t) ? x : pick(x, h);
    }
  }
  return x;
}

// phase_inner, except that a branch starting a chain of at least kFoldMin
// links pushes a fold frame {c0 | bit, c1 | bit, saved} and searches the
// chain's tail (if its box is hit) with a fresh result.
template <typename StackT, bool kSolo>
__device__ __forceinline__ int phase_inner_team(const MeshView& m, const Ray& r, StackT stack, uint32_t cap, Trav& s,
                                                bool& bad, const Team<kSolo>& tm) {
  if (s.right != kUMax && is_link(m, s.node, s.left, s.right)) {
    const uint32_t c0 = s.node, c1 = chain_last(m, c0, tm);
    if (c1 - c0 + 1 >= kFoldMin) {
      s.steps += 2 * (c1 - c0 + 1);  // its branches and leaves
      if (s.steps > 2 * m.num_tri) {
        bad = true;
        return kLaneDone;
      }
      if (s.sp >= cap) return kLaneOverflow;
      stack.store(s.sp++, make_uint4(kChainBit | c0, kChainBit | c1, __float_as_uint(s.best.t), s.best.id));
      s.best = Hit{INFINITY, kUMax};
      s.chain_next = kUMax;
      const uint32_t tail = c1 + 1;
      float te, tx;
      if (!node_slab(m, r, tail, te, tx)) return kLaneAscend;  // the fold ignores the tail
      s.node = tail;
      load_record(m.bvhnodes, tail, s.left, s.right);
      return kLaneInner;
    }
  }
  return phase_inner(m, r, stack, cap, s, bad);
}

constexpr uint32_t kChainPrefetch = 8;  // groups of 32 links per warp prefetched ahead of the fold

// Fold frames {c0 | bit, c1 | bit, saved}: the tail's result (the current
// one) is folded through the chain, and the chain's result into `saved`.
template <bool kSolo>
struct ChainFold {
  const MeshView& m;
  const Ray& r;
  const Team<kSolo>& tm;
  bool* bad;
  __device__ __forceinline__ int operator()(const uint4& f, Trav& s) const {
    if (!((f.x & kChainBit) && (f.y & kChainBit))) return 0;
    const uint32_t c0 = f.x & ~kChainBit, c1 = f.y & ~kChainBit;
    if (c0 > c1 || c1 + 1 >= 2 * m.num_tri - 1) return 2;
    Hit x = s.best;
    const uint32_t nb = m.num_tri - 1, total = c1 - c0 + 1, round = kFoldLinks * tm.warps;
    for (uint32_t done = 0; done < total; done += round) {
      const uint32_t side = tm.fold_side;
      tm.fold_side ^= 1u;
      // the warp's links of the next rounds (lane k: one link of each group)
      // toward L2 while this round's are tested: a long chain's tree does not
      // fit L2
#pragma unroll
      for (uint32_t d = 0; d < kChainPrefetch; ++d) {
        const uint32_t i = done + (1 + d / kFoldBatch) * round + tm.rank * kFoldLinks + 32 * (d % kFoldBatch) + tm.lane;
        if (i < total) {
          const uint64_t j = c1 - i;
          asm volatile("prefetch.global.L2 [%0];" ::"l"(m.bvhnodes + 3 * (nb + j)));
          asm volatile("prefetch.global.L2 [%0];" ::"l"(m.aabb + 6 * (nb + j)));
          asm volatile("prefetch.global.L2 [%0];" ::"l"(m.aabb + 6 * (j + 1)));
        }
      }
      const uint32_t from = done + tm.rank * kFoldLinks;
      if (from < total) {
        test_links(m, r, c1 - from, total - from < kFoldLinks ? total - from : kFoldLinks, tm.lane, tm.sh[tm.rank],
                   side, *bad);
      } else if (tm.lane == 0) {
        tm.sh[tm.rank].num_op[side] = 0;
        tm.sh[tm.rank].cut[side] = 0;
      }
      tm.sync();
      x = apply_links(tm, side, x);
    }
    --s.sp;
    s.best = pick(Hit{__uint_as_float(f.z), f.w}, x);
    return 1;
  }
};

template <typename StackT, bool kSolo>
__device__ __forceinline__ int trav_step_team(const MeshView& m, const Ray& r, StackT stack, uint32_t cap, Trav& s,
                                              bool& bad, const Team<kSolo>& tm) {
  int st = phase_inner_team(m, r, stack, cap, s, bad, tm);
  if (st == kLaneLeaf) st = phase_leaf(m, r, s, bad);
  if (st == kLaneAscend) st = phase_ascend(m, r, stack, s, bad, ChainFold<kSolo>{m, r, tm, &bad});
  return st == kLaneInner ? kStepContinue : (st == kLaneOverflow ? kStepOverflow : kStepDone);
}

// Rays that outlast the rest.  When the work runs out, a cast is as long as its
// longest ray from there on, and long rays come in bundles: neighbouring pixels
// graze the same silhouette, so one warp holds many and the others run empty.
// The persistent cast therefore parks rays past park_steps node entries, stack
// and all, and this kernel deals them out again, as few per warp as it can, and
// lets the lanes that hold none help: F(n) of a frame's far child depends on
// nothing outside n, so a lane may search it for another.  A lane gives away its
// frames from the bottom, the largest subtrees first.  Popping a given frame, it
// joins: it drops the helper if the recursion skips the far child (nearer result
// than the far box), else it waits for the helper's result and picks it after
// its own, which is what searching the far child would have done, as pick is
// associative.  Results are therefore the same bits; only subtrees that are
// skipped after all are searched in vain.
// What bounds it: a node entry is about 1,250 cycles (two of them and a leaf test
// or a pop per iteration), and the helpers' ramp.  Measured (cast alone, start ->
// with parking, 3% of which are the branches saved in phase_inner): 2M torus
// 1920 x 1080 (longest ray 504 entries) 613 -> 421 us; 512 x 512 of a deformed
// 502k torus (338) 334 -> 237 us; 641 x 479 of a 66k torus (207) 198 -> 162 us;
// 16,384 rays on a jittered 200k sphere (209) 195 -> 131 us.  Casts with no long
// rays keep their time (4.2M rays on 1,024 small meshes, at most 100 entries:
// 1.26 -> 1.23 ms).
// A ray that runs into a long chain or out of stack is linked into the block's
// own list (`handed`: the first by parked index, and how many; the next one in its
// second word) and cast by the block's team or teams afterwards.
template <typename Job, int kStack>
__device__ __forceinline__ void cast_split(const Job& job, const float* smem, const Parked& parked, uint32_t num,
                                           uint32_t* take, uint2* sh_deal, uint32_t* handed, uint32_t long_steps,
                                           uint32_t* status) {
  constexpr uint32_t kAll = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t lt_mask = (1u << lane) - 1u;
  const uint32_t warps = gridDim.x * (blockDim.x / 32);
  const uint32_t share = min(32u, (num + warps - 1) / warps);  // rays per warp at a time
  uint4 frames[kStack];
  LocalStack stack{frames};
  MeshView m{};
  Ray r{};
  Trav s{};
  uint32_t out = 0, slot = kUMax;
  int state = kLaneIdle;
  bool bad = false;
  uint32_t given = 0, parent = kUMax;  // frames given to other lanes; the lane this one helps
  // Every iteration enters a node, tests a leaf, pops a frame or joins for some
  // lane, and each happens at most once per node of a well-formed tree.
  uint32_t rounds_left = 0;
  for (;;) {
    const uint32_t idle = __ballot_sync(kAll, state == kLaneIdle);
    if (idle == kAll) {  // the next parked rays
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(take, share);
      base = __shfl_sync(kAll, base, 0);
      if (base >= num) break;
      if (lane < share && base + lane < num) {
        const uint4* from = parked.rays + static_cast<size_t>(base + lane) * parked.stride;
        const uint4 a = from[0], b = from[1];
        slot = base + lane;
        if (job.fetch(a.x, smem, m, r, out)) {
          s = Trav{};
          s.node = a.y;
          s.left = a.z;
          s.right = a.w;
          s.sp = b.x;
          s.steps = b.y;
          s.chain_next = kUMax;
          s.best = Hit{__uint_as_float(b.z), b.w};
          for (uint32_t k = 0; k < s.sp; ++k) frames[k] = from[2 + k];
          parent = kUMax;
          given = 0;
          state = kLaneInner;
        }
      }
      rounds_left = __reduce_max_sync(kAll, min(m.num_tri, 1u << 28)) * 8u + 1024u;
      continue;
    }
    if (rounds_left-- == 0u) {
      if (state != kLaneIdle && parent == kUMax) job.write(out, m, r, Hit{INFINITY, kUMax});
      bad = true;
      state = kLaneIdle;
      continue;
    }
    if (idle != 0u) {
      // lanes with a frame to give: the bottom one not yet given
      uint32_t far = kUMax;
      const bool busy = state == kLaneInner || state == kLaneLeaf || state == kLaneAscend;
      if (busy && s.sp > given + (state == kLaneAscend ? 1u : 0u)) far = frames[given].x;
      // in a malformed tree nothing is split, so that the step budget bounds all work
      const uint32_t any_bad = __ballot_sync(kAll, bad);
      const bool can = any_bad == 0u && !(far & kChainBit);
      const uint32_t givers = __ballot_sync(kAll, can);
      const uint32_t n = min(__popc(idle), __popc(givers));
      if (n != 0u) {
        const uint32_t rank_g = __popc(givers & lt_mask), rank_i = __popc(idle & lt_mask);
        const bool gives = can && rank_g < n, takes = state == kLaneIdle && rank_i < n;
        uint2* deal = sh_deal + (threadIdx.x & ~31u);
        if (gives) deal[rank_g].x = lane;
        if (takes) deal[rank_i].y = lane;
        __syncwarp();
        const uint32_t from = takes ? deal[rank_i].x : lane;
        const uint32_t node = __shfl_sync(kAll, far, from);
        r.org = make_float3(__shfl_sync(kAll, r.org.x, from), __shfl_sync(kAll, r.org.y, from),
                            __shfl_sync(kAll, r.org.z, from));
        r.dir = make_float3(__shfl_sync(kAll, r.dir.x, from), __shfl_sync(kAll, r.dir.y, from),
                            __shfl_sync(kAll, r.dir.z, from));
        r.inv = make_float3(__shfl_sync(kAll, r.inv.x, from), __shfl_sync(kAll, r.inv.y, from),
                            __shfl_sync(kAll, r.inv.z, from));
        r.nz = __shfl_sync(kAll, r.nz ? 1 : 0, from) != 0;
        job.share(m, static_cast<int>(from));
        const uint32_t steps = __shfl_sync(kAll, s.steps, from);
        if (gives) {
          frames[given].x = kGivenBits | deal[rank_g].y;
          ++given;
        }
        if (takes) {
          parent = from;
          given = 0;
          s.node = node;
          s.sp = 0;
          s.steps = steps;
          s.chain_next = kUMax;
          s.leaf_far = false;
          s.best = Hit{INFINITY, kUMax};
          state = kLaneInner;
          if (node >= 2 * m.num_tri - 1) {
            bad = true;
            state = kLaneHelped;
          } else {
            load_record(m.bvhnodes, node, s.left, s.right);
          }
        }
        __syncwarp();
      }
    }
#pragma unroll
    for (int k = 0; k < kTailSteps; ++k)
      if (state == kLaneInner) state = phase_inner(m, r, stack, kStack, s, bad);
    if (state == kLaneLeaf) state = phase_leaf(m, r, s, bad);
    if (state == kLaneAscend) state = phase_ascend(m, r, stack, s, bad, NoFold{}, given);
    // A ray past the step budget that is about to enter a long chain would
    // hold the kernel's end: it is handed to the team tier, which folds chains
    // many links at a time.
    if (state == kLaneInner && s.steps > long_steps && long_chain_at(m, s.node, s.left, s.right))
      state = kLaneOverflow;
    if (state == kLaneDone) {
      if (parent == kUMax) {
        job.write(out, m, r, s.best);
        state = kLaneIdle;
      } else {
        state = kLaneHelped;
      }
    }
    uint32_t drop = 0;  // lanes whose result is no longer needed
    if (__any_sync(kAll, state == kLaneJoin)) {
      uint4 f = make_uint4(0, 0, 0, 0);
      if (state == kLaneJoin) f = frames[s.sp - 1];
      const uint32_t helper = f.x & 31u;
      const int h_state = __shfl_sync(kAll, state, helper);
      const Hit h_best{__shfl_sync(kAll, s.best.t, helper), __shfl_sync(kAll, s.best.id, helper)};
      const bool skip = s.best.id != kUMax && __uint_as_float(f.y) > s.best.t;
      const bool pop = state == kLaneJoin && (skip || h_state == kLaneHelped);
      drop = __reduce_or_sync(kAll, pop ? 1u << helper : 0u);
      if (pop) {
        s.best = pick(Hit{__uint_as_float(f.z), f.w}, s.best);
        if (!skip) s.best = pick(s.best, h_best);
        --s.sp;
        --given;
        state = kLaneAscend;
      }
    }
    if (__any_sync(kAll, state == kLaneOverflow)) {
      // the whole ray goes, whichever of its lanes ran into it
      uint32_t over = __ballot_sync(kAll, state == kLaneOverflow);
      for (;;) {
        const bool up = (over >> lane & 1u) && parent != kUMax;
        const uint32_t more = over | __reduce_or_sync(kAll, up ? 1u << (parent & 31u) : 0u);
        if (more == over) break;
        over = more;
      }
      if ((over >> lane & 1u) && parent == kUMax) {
        parked.rays[static_cast<size_t>(slot) * parked.stride + 1].x = atomicExch(handed, slot);
        atomicAdd(handed + 1, 1u);
      }
      drop |= over;
    }
    if (drop != 0u) {  // and with a lane all that help it
      for (;;) {
        const bool down = state != kLaneIdle && parent != kUMax && (drop >> (parent & 31u) & 1u);
        const uint32_t more = drop | __ballot_sync(kAll, down);
        if (more == drop) break;
        drop = more;
      }
      if (drop >> lane & 1u) {
        state = kLaneIdle;
        parent = kUMax;
        given = 0;
      }
    }
  }
  if (bad) raise_status(status, kStatusBadIndex);
}

// Rays of the team tier's list linked into lists of those to be cast again: such a
// list is the index of its first ray, or kUMax.
struct RayLinks {
  uint32_t* team_list;  // work indices
  uint32_t* next;       // per entry of team_list
  __device__ __forceinline__ uint32_t work(uint32_t id) const {
    return *reinterpret_cast<const volatile uint32_t*>(team_list + id);
  }
  // By many at a time; read only after all of them.
  __device__ __forceinline__ void push(uint32_t* head, uint32_t id) const { next[id] = atomicExch(head, id); }
  // For a ray that was parked, and so is in no list yet: `id` is a free entry.
  __device__ __forceinline__ uint32_t append(uint32_t id, uint32_t w) const {
    team_list[id] = w;
    return id;
  }
  // By the threads of one block at a time; no ray is pushed meanwhile.
  __device__ __forceinline__ uint32_t pop(uint32_t* head) const {
    uint32_t id = *reinterpret_cast<volatile uint32_t*>(head);
    while (id != kUMax) {
      const uint32_t seen = atomicCAS(head, id, *reinterpret_cast<volatile uint32_t*>(next + id));
      if (seen == id) break;
      id = seen;
    }
    return id;
  }
};

// Re-casts a list of rays by one block, a thread per ray, with stacks of `cap`
// frames (of pool_frames, if that is less) carved from pool[0 .. pool_frames) and
// more[0 .. more_frames).
template <typename Job>
__device__ __noinline__ void cast_deep(const Job& job, const float* smem, const RayLinks& links, uint32_t* list,
                                       uint4* pool, uint64_t pool_frames, uint4* more, uint64_t more_frames,
                                       uint64_t cap, uint32_t* status) {
  if (cap > pool_frames) cap = pool_frames;
  const uint64_t slot = threadIdx.x, here = pool_frames / cap;
  const bool has_stack = slot < here + more_frames / cap;
  uint4 ring[kDeepRing];
  uint32_t lo = 0;
  const RingStack<kDeepRing> st{ring, slot < here ? pool + slot * cap : more + (slot - here) * cap, &lo};
  bool bad = false;
  for (;;) {
    // a warp's lanes start together: on their own they would stay apart, each of
    // them with the loads of a step to itself
    const uint32_t id = has_stack ? links.pop(list) : kUMax;
    if (!__any_sync(kWarpAll, id != kUMax)) break;
    MeshView m{};
    Ray r{};
    uint32_t out = 0;
    if (id == kUMax || !job.fetch(links.work(id), smem, m, r, out)) continue;
    lo = 0;
    Trav s{};
    int rc = kStepDone;
    if (trav_begin(m, r, s)) {
      do {
        rc = trav_step(m, r, st, static_cast<uint32_t>(cap), s, bad);
      } while (rc == kStepContinue);
    }
    if (rc == kStepDone) {
      job.write(out, m, r, s.best);
    } else {
      raise_status(status, kStatusStackOverflow);
      job.write(out, m, r, Hit{INFINITY, kUMax});
    }
  }
  if (bad) raise_status(status, kStatusBadIndex);
}

// Ray `id` of the list cast by a team.  Every lane keeps the same stack (the ring in
// its own local memory, the spilled frames at the same addresses of its warp's slice
// of the pool); a ray whose frames outgrow the slice is linked into `over`.  All of the
// team meet between two rays.
template <bool kSolo, typename Job>
__device__ __noinline__ void cast_team(const Job& job, const float* smem, uint32_t w, const Team<kSolo>& tm, uint4* slice,
                                       uint32_t cap, uint32_t id, uint32_t* next, uint32_t* over, bool& bad) {
  uint4 ring[kDeepRing];
  uint32_t lo = 0;
  const RingStack<kDeepRing> st{ring, slice, &lo};
  MeshView m{};
  Ray r{};
  uint32_t out = 0;
  if (!job.fetch(w, smem, m, r, out)) return;
  Trav s{};
  int rc = kStepDone;
  if (trav_begin(m, r, s)) {
    do {
      rc = trav_step_team(m, r, st, cap, s, bad, tm);
    } while (rc == kStepContinue);
  }
  if (tm.rank == 0 && tm.lane == 0) {
    if (rc == kStepDone) job.write(out, m, r, s.best);
    else next[id] = atomicExch(over, id);
  }
}

// The lists and counters of the tiers after the persistent cast.
struct TailArgs {
  Parked parked;          // rays for the split tier, in the first half of the pool
  uint32_t* parked_take;  // of them given out
  RayLinks links;
  const uint32_t* team_count;
  uint32_t* team_take;
  uint32_t* team_more;   // parked rays appended to team_list
  uint32_t* deep;        // of all blocks, then per group: the rays whose frames outgrew a team's slice
  uint32_t* done;        // of all blocks, then per group: those that have finished
  uint4* pool;
  uint64_t pool_frames, slice_frames, group_frames;  // of all, of a team's warp, of a group
  uint32_t max_tri, long_steps;
  uint32_t* status;
};

// All tiers after the persistent cast in one launch: the split tier, then the
// team tier, then what outgrew a team's slice (some 570 frames and 64 more): trees
// that are not of Morton codes, whose chains are folded.  The last block to finish
// of each group of blocks casts the group's such rays, with stacks that are sure to
// do, carved from the group's share of the pool; for trees so large that all groups
// hold fewer stacks than one block has threads, the last block of all casts them,
// with the whole pool.  With a kernel for each tier, an image without such rays paid
// three more launches: 6 us each of a server's dispatcher thread.
//
// A team is a whole block while the rays are few, kTeamRays per block or
// fewer: then the longest ray sets the kernel's end.  With more, their number
// does, and each warp takes rays of its own.
// Blocks a multiprocessor of the tail kernel: 6 (80 registers, 80 bytes of spills)
// let the split tier of large images hold more rays at once than 4 (124
// registers) and cost the others nothing; 2M triangles at 1920 x 1080 with 4, 5,
// 6, 8: 431, 432, 407, 416 us, 16,384 rays 135, 130, 132, 138 us, 512 x 512 of
// 502 thousand triangles 212, 213, 213, 220 us, a soup's rays 657, 642, 655,
// 709 us.
constexpr uint32_t kTailBlocks = 6;
constexpr uint32_t kTeamRays = 8;
// Groups of blocks with a list of deep rays each.  Combs whose every level is a
// frame, 4,096 rays, by the last block of all / by groups: 1,200 levels 77 / 5.0 ms,
// 3,000 levels 143 / 16 ms.  (65,536 rays: 802 / 56 and 1,846 / 196 ms.)
constexpr uint32_t kDeepGroups = 24;
static_assert((7 + 2 * (1 + kDeepGroups)) * sizeof(uint32_t) <= kCastCounterBytes, "counters");
template <typename Job, int kStack>
__global__ void __launch_bounds__(kTeamThreads, kTailBlocks) k_cast_tail(Job job, TailArgs a) {
  __shared__ float smem[64];
  __shared__ FoldShared sh[kTeamWarps];
  __shared__ uint2 sh_deal[kTeamThreads];
  __shared__ uint32_t sh_take, sh_handed[2];
  job.prepare(smem);
  if (threadIdx.x == 0) {
    sh_handed[0] = kUMax;
    sh_handed[1] = 0u;
  }
  pdl_wait();
  __syncthreads();
  const uint32_t parked = min(*a.parked.count, a.parked.capacity), num = *a.team_count;
  if (parked == 0 && num == 0) return;
  if (parked != 0) {
    cast_split<Job, kStack>(job, smem, a.parked, parked, a.parked_take, sh_deal, sh_handed, a.long_steps, a.status);
    __syncthreads();
  }
  const uint32_t group = blockIdx.x % kDeepGroups;
  const uint64_t half = a.pool_frames / 2, room = a.group_frames;  // a group's slices lie together
  const uint32_t need = max(a.max_tri, 2u);  // no tree needs more frames than it has leaves
  const bool grouped = room >= 6ull * need;  // 24 times 6: more than the threads of a block
  uint32_t* const deep = a.deep + (grouped ? 1 + group : 0);
  const RayLinks links = a.links;
  // the split tier's rays of this block, then those of the list
  for (uint32_t from_list = 0; from_list < 2; ++from_list) {
    if (from_list ? num == 0 : sh_handed[1] == 0) continue;
    const bool solo = from_list ? num > kTeamRays * gridDim.x : sh_handed[1] >= kTeamWarps;
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x & 31u;
    // the teams' stacks lie in the pool's second half: parked rays may still be
    // waiting in the first
    uint4* const slice =
        a.pool + half + group * room + (blockIdx.x / kDeepGroups * kTeamWarps + warp) * a.slice_frames;
    const uint32_t cap = static_cast<uint32_t>(min(a.slice_frames, static_cast<uint64_t>(need)));
    const Team<true> one{sh + warp, 0u, lane, 0u, 0u};
    const Team<false> all{sh, warp, lane, 0u, 0u};
    bool bad = false;
    for (;;) {
      uint32_t id = kUMax;
      if (solo ? lane == 0 : threadIdx.x == 0) {
        id = from_list ? atomicAdd(a.team_take, 1u) : a.parked.take_handed(sh_handed);
        if (from_list) id = id < num ? id : kUMax;
        else if (id != kUMax) id = links.append(num + atomicAdd(a.team_more, 1u), a.parked.work(id));
      }
      if (solo) {
        id = __shfl_sync(kWarpAll, id, 0);
        __syncwarp();
      } else {
        if (threadIdx.x == 0) sh_take = id;
        __syncthreads();
        id = sh_take;
        __syncthreads();
      }
      if (id == kUMax) break;
      if (solo) cast_team<true>(job, smem, links.work(id), one, slice, cap, id, links.next, deep, bad);
      else cast_team<false>(job, smem, links.work(id), all, slice, cap, id, links.next, deep, bad);
    }
    if (bad) raise_status(a.status, kStatusBadIndex);
    __syncthreads();
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) sh_take = atomicAdd(a.done + (grouped ? 1 + group : 0), 1u);
  __syncthreads();
  // the last block of the group, or of all, casts what is left
  if (sh_take != (grouped ? (gridDim.x - 1 - group) / kDeepGroups : gridDim.x - 1)) return;
  __threadfence();
  if (*reinterpret_cast<volatile uint32_t*>(deep) == kUMax) return;
  if (!grouped) {
    cast_deep(job, smem, links, deep, a.pool, a.pool_frames, static_cast<uint4*>(nullptr), 0ull, need, a.status);
  } else {
    // and from the group's part of what the parked rays leave free of the first half
    const uint64_t used = static_cast<uint64_t>(parked) * a.parked.stride, more = (half - used) / kDeepGroups;
    cast_deep(job, smem, links, deep, a.pool + half + group * room, room, a.pool + used + group * more, more, need,
              a.status);
  }
}

// Number of resident blocks of a persistent kernel instantiation on the
// current device.
template <typename Job, int kThreads, int kStack, bool kPark>
inline int persistent_grid() {
  static int cached[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (cached[dev] == 0) {
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cast_persistent<Job, kThreads, kStack, kPark>, kThreads,
                                                  0);
    cached[dev] = (sms > 0 ? sms : 152) * (per_sm > 0 ? per_sm : 1);
  }
  return cached[dev];
}

// Node entries after which a ray is parked: kParkSteps for up to kParkRays rays,
// kParkMore more for each of the first kParkDoublings doublings.  Parked too early,
// rays crowd the split tier; too late, they hold the persistent cast.  Casts in us
// by threshold:
//   16,384 rays on a jittered sphere    24: 136   40: 142   64: 160   96: 185   never: 194
//   641 x 479 on a torus                40: 177   64: 156   80: 159  112: 184   never: 193
//   512 x 512 on a deformed torus       40: 286   64: 251   80: 235  112: 240   never: 324
// and, means over six 2M tori (never: before there was parking)
//   1280 x 720                          94: 385  140: 415  180: 452  220: 473   never: 537
//   1920 x 1080                         80: 532   94: 520  108: 529  150: 529   never: 629
//   2560 x 1440                         88: 690   94: 697  122: 700  150: 704   never: 765
//   3840 x 2160                         88: 1194  94: 1191 108: 1190 150: 1209  never: 1252
// Where no ray goes on for long, the tail's fixed time is not won back: on the
// smoothest two of the six, 1920 x 1080 takes 485 and 497 us against 465 and 467.
constexpr uint32_t kParkSteps = 24, kParkRays = 16384, kParkMore = 14, kParkDoublings = 5;

// In a tree of up to kParkSmallTri triangles no ray goes on for much longer than
// kParkSmallSteps, and the tail costs more than it saves.  Parked from 24 / from 64
// entries: 20,000 rays on 80 triangles 50.5 / 41.4 us, on 200 61.9 / 51.7, on 648
// 70.5 / 64.0; 64 x 64 pixels of 200 triangles 45.6 / 37.5, of 648 49.7 / 41.4.  Beyond
// that the lower threshold wins: 1,000 and 20,000 rays on 1,250 triangles 52.5 / 57.8
// and 79.1 / 85.3, on 2,048 53.7 / 61.9 and 78.3 / 88.5.
constexpr uint32_t kParkSmallTri = 1024, kParkSmallSteps = 64;

inline uint32_t park_steps(uint32_t num_work, uint32_t max_tri) {
  uint32_t doublings = 0;
  for (uint32_t n = num_work; n >= 2 * kParkRays && doublings < kParkDoublings; n >>= 1) ++doublings;
  const uint32_t steps = kParkSteps + kParkMore * doublings;
  return max_tri <= kParkSmallTri && steps < kParkSmallSteps ? kParkSmallSteps : steps;
}

// Zeroes a cast's counters.  A kernel instead of a copy-engine memset, so that
// the persistent cast's blocks are resident when it ends.
static __global__ void k_cast_begin(uint32_t* counters) {
  pdl_wait();
  pdl_launch_dependents();
  if (threadIdx.x < kCastCounterBytes / sizeof(uint32_t))
    counters[threadIdx.x] = threadIdx.x >= 7 && threadIdx.x < 8 + kDeepGroups ? kUMax : 0u;
}

// `busy`: the GPU has other work to do beside this cast (a server with requests
// in flight).  Then the cast's own latency counts for less than the issue slots
// it takes: warps are filled and nothing is parked, as helpers also search
// subtrees that turn out not to be needed.  64 requests in flight at once took
// 4.65 ms so and 5.01 ms with parking.
template <typename Job, int kThreads, int kStack, bool kBusy>
inline void launch_tiers(cudaStream_t s, const Job& job, const CastScratch& sc, uint32_t max_tri, uint32_t* status) {
  int grid = persistent_grid<Job, kThreads, kStack, !kBusy>();
  const uint32_t warps = static_cast<uint32_t>(grid) * (kThreads / 32);
  // few rays are spread over all warps, so that a warp has fewer phases to run
  // one after the other and more lanes to help in the split tier: 16,384 rays by
  // 32, 8, 4, 2 per warp: 135, 126, 131, 134 us.  From about 8 per warp on there
  // is no gain (65,536 rays by 14: 177 against 171 us for build and cast).
  const uint32_t share =
      job.num_work <= 8 * warps && !kBusy ? (job.num_work + warps - 1) / warps : 32u;
  const uint32_t needed = ((job.num_work + share - 1) / share + kThreads / 32 - 1) / (kThreads / 32);
  if (static_cast<uint32_t>(grid) > needed) grid = static_cast<int>(needed);
  const Tuning t = get_tuning();
  // One mesh takes rays as soon as a quarter of a warp is idle; a batch, whose
  // fetch reads a dozen words of tables and a matrix per ray, waits for half as
  // many again.  Threshold 12 and 8: 2M triangles at 1920 x 1080 458 and 438 us,
  // 500 thousand at 512 x 512 243 and 222 us, but the batch 1232 and 1267 us
  // (at 9, 8, 6 for a mesh and 13, 12, 9 for the batch: 437, 438, 441; 1230,
  // 1231, 1253 us).
  const uint32_t refill = min(t.cast_refill_min * Job::kRefillHalves / 2u, 32u);
  const uint32_t park = kBusy ? kUMax : park_steps(job.num_work, max_tri);
  // A ray that would be parked at a long chain goes to the team tier at once.  Parked, it
  // got there only by the split tier's block, behind that block's other rays, and was cast
  // by it alone.  Rays on clustered soups, parked / handed over: 10,000 on 20 thousand
  // triangles 91 / 95 us, on 70 thousand 189 / 163, on 200 thousand 228 / 195, on 1
  // million 310 / 214, on 4 million 472 / 287; 60,000 on 200 thousand 304 / 230, on 4
  // million 640 / 457.  (With the lower bound in the split tier too: 60,000 on 20 and 70
  // thousand 199 and 220 us, 140 and 162 so.)
  const PhaseMins mins{refill, t.cast_leaf_min, t.cast_ascend_min, min(t.cast_long_steps, park), park, share};
  TailArgs a;
  a.parked.rays = static_cast<uint4*>(sc.pool);
  a.parked.count = sc.counters + 5;
  a.parked.stride = kStack + 2;
  const uint64_t room = sc.pool_bytes / 2 / (sizeof(uint4) * a.parked.stride);
  a.parked.capacity = static_cast<uint32_t>(room < (1u << 20) ? room : (1u << 20));
  a.parked_take = sc.counters + 6;
  a.links = RayLinks{sc.list1, sc.list2};
  a.team_count = sc.counters + 1;
  a.team_take = sc.counters + 4;
  a.team_more = sc.counters + 2;
  a.deep = sc.counters + 7;
  a.done = a.deep + 1 + kDeepGroups;
  a.pool = static_cast<uint4*>(sc.pool);
  a.pool_frames = sc.pool_bytes / kFrameBytes;
  a.max_tri = max_tri;
  a.long_steps = t.cast_long_steps;
  a.status = status;
  const uint32_t tail_grid = 152 * kTailBlocks, group_size = (tail_grid + kDeepGroups - 1) / kDeepGroups;
  a.slice_frames = a.pool_frames / 2 / (kDeepGroups * group_size * kTeamWarps);
  a.group_frames = a.slice_frames * group_size * kTeamWarps;
  launch_pdl(k_cast_begin, dim3(1), dim3(64), 0, s, sc.counters);
  launch_pdl(k_cast_persistent<Job, kThreads, kStack, !kBusy>, dim3(grid), dim3(kThreads), 0, s, job, sc.counters, sc.list1,
             sc.counters + 1, status, mins, a.parked);
  launch_pdl(k_cast_tail<Job, kStack>, dim3(tail_grid), dim3(kTeamThreads), 0, s, job, a);
}

// The tiered cast of every work index of `job`: the persistent cast, then one
// kernel for the rays it hands over (k_cast_tail).  sc.counters
// (kCastCounterBytes) are set first: [0] rays taken, [1] rays for the team tier
// (list1), [2] parked rays added to them, [4] rays taken by the team
// tier, [5] rays parked, [6] parked rays taken, from [7] on the lists of rays with
// more frames (linked by list2), of all blocks and of each group, then the blocks
// done likewise.  The first tier's block size and on-chip stack depth come from the
// current Tuning (kCastVariants lists the choices).
template <typename Job, bool kBusy = false>
inline void cast_job(cudaStream_t s, const Job& job, const CastScratch& sc, uint32_t max_tri, uint32_t* status) {
  if (job.num_work == 0) return;
  const Tuning t = get_tuning();
  if (t.cast_threads == 64 && t.cast_stack == 64) launch_tiers<Job, 64, 64, kBusy>(s, job, sc, max_tri, status);
  else if (t.cast_threads == 256 && t.cast_stack == 64) launch_tiers<Job, 256, 64, kBusy>(s, job, sc, max_tri, status);
  else if (t.cast_threads == 128 && t.cast_stack == 32) launch_tiers<Job, 128, 32, kBusy>(s, job, sc, max_tri, status);
  else if (t.cast_threads == 128 && t.cast_stack == 96) launch_tiers<Job, 128, 96, kBusy>(s, job, sc, max_tri, status);
  else launch_tiers<Job, 128, 64, kBusy>(s, job, sc, max_tri, status);
}

}  // namespace dm
