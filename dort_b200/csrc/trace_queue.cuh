// Warp-cooperative traversal of a queue of rays (device only).
//
// One ray per thread inside a persistent warp, as in trace_ray, but the warp
// decides together what its lanes do next, so that divergent rays keep the
// lanes busy:
//   - a lane whose ray is finished takes the queue's next ray as soon as
//     kIdleLanes lanes are idle, instead of waiting for the warp's longest
//     ray;
//   - leaf triangles are not tested in the node step that finds them: a lane
//     holds up to two nodes' worth of them and goes on with its nodes until
//     kTriLanes lanes hold some (or fewer than kMinLanes can go on), and the
//     warp then tests triangles together until fewer than kMinLanes hold any.
// Neither changes a result: the closest hit is the minimum over the triangles
// tested (ties go to the larger index), whatever their order; a later
// triangle test only means that a few more boxes pass against the older t.
//
// Measured on the 1M-triangle soup: a warp's 32 diffuse bounce rays took 59
// node steps with 16.5 lanes active and 115 triangle tests with 3.5 lanes
// active one ray per lane to the end; 37.5 steps with 26 lanes and 34 tests
// with 12 lanes this way (4M such rays: 3.61 ms against 2.47 ms when it came, 2.24
// now; the camera rays of the same scene 1.69 against 1.65, now 1.50 ms).
#pragma once
#include "trace.cuh"

namespace dort_gpu {

constexpr uint32_t kNoItem = 0xffffffffu;
constexpr uint32_t kWarpAll = 0xffffffffu;

// Brings the bytes of [from, to) on their way to the L2 cache, a 128-byte line
// per lane of `lanes` (the first ones).
__device__ __forceinline__ void prefetch_l2(const void* from, const void* to, uint32_t lane) {
  const char* p = static_cast<const char*>(from) + 128u * lane;
  if(p < to) { asm volatile("prefetch.global.L2 [%0];" :: "l"(p)); }
}

// Neighbours (12 to 20, 6 to 10, 3 to 6) measured within 2 % on the soup's
// camera and bounce rays; refilling at 8 idle lanes or more was slower.
constexpr int kTriLanes = 16;
constexpr int kMinLanes = 8;
constexpr int kIdleLanes = 4;

// Entries of a queue that every warp starts with: an equal share of a short
// queue, down to a single entry (a ray alone in its warp is finished
// soonest), 64 of a long one.
__host__ __device__ __forceinline__ uint32_t queue_first(uint32_t count, uint32_t warps) {
  const uint32_t share = count / warps + (count % warps ? 1u : 0u);
  return share < 1u ? 1u : (share > 64u ? 64u : share);
}

// Entries a warp takes at a time after that when `left` are not yet taken:
// half a share towards the queue's end, so that the warps finish together,
// but not so few that the cursor's atomics (about 1 ns each, one address) add
// up: with eighths down to 8 entries the Cornell frame took 3.92 ms instead
// of 3.65.
__device__ __forceinline__ uint32_t queue_next(uint32_t left, uint32_t warps) {
  return min(64u, max(16u, left / (2u * warps)));
}

// Results that wait in shared memory until 32 of them can be worked off by
// the whole warp (a finished ray's follow-up loads would otherwise stall the
// warp for a few lanes).  kSlots entries of kWords words per warp.
template<uint32_t kWords>
struct WarpBuffer {
  static constexpr uint32_t kSlots = 64;
  uint32_t* slots;     // this warp's words
  uint32_t count;      // warp-uniform

  static constexpr size_t bytes(int block) {
    return size_t(block / 32) * kSlots * kWords * sizeof(uint32_t);
  }
  __device__ __forceinline__ static WarpBuffer of_warp(uint32_t* shared) {
    return WarpBuffer{shared + (threadIdx.x >> 5) * kSlots * kWords, 0u};
  }
  // Adds the entry (a, b) of every lane with `want` (b with two words); true
  // when 32 entries are there.
  __device__ __forceinline__ bool push(bool want, uint32_t a, uint32_t b = 0u) {
    const uint32_t mask = __ballot_sync(kWarpAll, want);
    const uint32_t lane = threadIdx.x & 31u;
    if(want) {
      const uint32_t at = count + __popc(mask & ((1u << lane) - 1u));
      slots[at] = a;
      if(kWords > 1) { slots[at + kSlots] = b; }
    }
    count += __popc(mask);
    return count >= 32u;
  }
  // This lane's entry of the 32 (or the last few) oldest; false if none.
  __device__ __forceinline__ bool take(uint32_t& a, uint32_t& b) {
    const uint32_t lane = threadIdx.x & 31u;
    const bool have = lane < count, rest = lane + 32u < count;
    __syncwarp();
    a = slots[lane];
    b = kWords > 1 ? slots[lane + kSlots] : 0u;
    const uint32_t ra = slots[lane + 32u];
    const uint32_t rb = kWords > 1 ? slots[lane + 32u + kSlots] : 0u;
    __syncwarp();
    if(rest) {
      slots[lane] = ra;
      if(kWords > 1) { slots[lane + kSlots] = rb; }
    }
    count = count > 32u ? count - 32u : 0u;
    return have;
  }
};

// The last few rays of a warp (at most kWideRays, in the lanes `busy`), eight
// lanes to a ray: every lane of a group holds its ray's whole state and walks
// the tree in step with the others; lane j tests the box of slot j and the
// triangles of leaf slot j, and votes and shuffles bring the results together.
// A lone ray's steps are chains of dependent instructions; this way a node
// costs some 90 of them instead of 270 and a node's triangles one test or two.
// The results are those of one lane: the same boxes pass, and the closest hit
// is the minimum whatever the order.
constexpr int kWideRays = 4;

template<bool ANY_HIT, bool EXACT_MT, int WT, class Q, class Stack>
__device__ __forceinline__ void trace_wide(Q& q, TravState& s, Stack& stack, uint2 leaf,
                                           uint2 leaf2, uint32_t item, uint32_t busy) {
  const uint32_t lane = threadIdx.x & 31u, slot = lane & 7u, group = lane & 24u;
  // group k takes the k-th busy lane's ray
  uint32_t from = busy;
  for(uint32_t k = 0; k < (lane >> 3); ++k) { from &= from - 1u; }
  const int src = from ? __ffs(from) - 1 : int(lane);
  auto take = [&](auto& v) { v = __shfl_sync(kWarpAll, v, src); };
  take(s.ox); take(s.oy); take(s.oz);
  take(s.dx); take(s.dy); take(s.dz);
  take(s.t_min);
  take(s.ix); take(s.iy); take(s.iz);
  take(s.near4); take(s.near2); take(s.near1);
  take(s.best.t); take(s.best.b1); take(s.best.b2); take(s.best.prim);
  take(s.group.x); take(s.group.y);
  if(WT != kTriMt) {
    take(s.wt.kx); take(s.wt.ky); take(s.wt.kz);
    take(s.wt.sx); take(s.wt.sy); take(s.wt.sz);
  }
  take(leaf.x); take(leaf.y); take(leaf2.x); take(leaf2.y);
  take(item);
  q.take(src);
  if(!from) { item = kNoItem; }
  const int had = s.sp;
  take(s.sp);
  const int deepest = __reduce_max_sync(kWarpAll, had);
  for(int k = 0; k < deepest; ++k) {
    uint2 e = k < had ? stack.pop(k) : make_uint2(0u, 0u);
    take(e.x);
    take(e.y);
    if(k < s.sp) { stack.push(k, e); }
  }
  for(;;) {
    const bool live = item != kNoItem;
    // the pending triangles: first ones, then second ones
    if(__any_sync(kWarpAll, live && !leaf_empty(leaf))) {
      bool hit = false;
#pragma unroll
      for(uint32_t k = 0; k < 2; ++k) {
        uint2 one = make_uint2(leaf.x, leaf.y & (0xffff0000u | (1u << (8u * k + slot))));
        if(live && !leaf_empty(one)) {
          if(trav_tri<ANY_HIT, EXACT_MT, WT>(s, q.scene(), one)) { hit = true; }
        }
      }
      const uint32_t hits = __ballot_sync(kWarpAll, hit);
      if(hits) {
#pragma unroll
        for(int d = 1; d < 8; d <<= 1) {
          Hit o;
          o.t = __shfl_xor_sync(kWarpAll, s.best.t, d);
          o.b1 = __shfl_xor_sync(kWarpAll, s.best.b1, d);
          o.b2 = __shfl_xor_sync(kWarpAll, s.best.b2, d);
          o.prim = __shfl_xor_sync(kWarpAll, s.best.prim, d);
          if(o.prim != kMiss && (s.best.prim == kMiss || o.t < s.best.t ||
                                 (o.t == s.best.t && o.prim > s.best.prim))) {
            s.best = o;
          }
        }
      }
      leaf = leaf2;
      leaf2.y = 0u;
      if(ANY_HIT && ((hits >> group) & 0xffu)) {
        leaf.y = 0u;
        s.group.y = 0u;
        s.sp = 0;
      }
    }
    const bool go = live && group_left(s) && leaf_empty(leaf);
    bool box = false;
    uint32_t child_base = 0, tri_base = 0, masks = 0;
    if(go) {
      const uint4* np = trav_next(s, q.scene());
      uint32_t n0[8], n1[8], n2[8];
      load_32(np, n0);
      load_32(np + 2, n1);
      load_32(np + 4, n2);
      child_base = n0[6];
      tri_base = n0[7];
      masks = n1[0];
      box = slot_hit(n0, n1, n2, slot, s.ox, s.oy, s.oz, s.ix, s.iy, s.iz, s.t_min,
                     fmaf(fabsf(s.best.t), DORT_SLAB_FAR_WIDEN, s.best.t));
    }
    const uint32_t hits = (__ballot_sync(kWarpAll, box) >> group) & 0xffu;
    if(go) { leaf = trav_enter(s, stack, hits, child_base, tri_base, masks); }
    const bool mine = live && !group_left(s) && leaf_empty(leaf);
    if(__any_sync(kWarpAll, mine)) {
      q.done(mine && slot == 0u, item, s);
      if(mine) { item = kNoItem; }
      if(__all_sync(kWarpAll, item == kNoItem)) { return; }
    }
  }
}

// Traces the entries [0, count) of a queue.  Every warp starts with the chunk
// of its own number; `cursor` (zero before) counts the entries taken after
// those, and is left alone by queues that the first chunks cover.
// Q:
//   const TraceScene& scene()               the scene of this lane's ray
//   void load(uint32_t i, TravState& s)     starts the ray of entry i
//   void done(bool mine, uint32_t i, const TravState& s)
//     called by the whole warp; lanes with `mine` have finished entry i (s.best)
//   void take(int src)                      the lane's own state becomes lane src's
//   void ahead(uint32_t first, uint32_t end)   entries the warp will start soon
template<bool ANY_HIT, bool EXACT_MT, int WT, class Q>
__device__ __forceinline__ void trace_queue(Q& q, uint32_t count, uint32_t* cursor) {
  const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  const uint32_t first = queue_first(count, warps);
  // the warp's entries not yet started
  uint32_t next = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * first;
  uint32_t end = min(next + first, count);
  bool more = warps * first < count;   // the cursor may have more
  uint32_t item = kNoItem;        // this lane's entry
  uint32_t idle = kWarpAll;       // lanes without one
  TravState s;
  s.group = make_uint2(0u, 0u);
  s.sp = 0;
  TraceStack stack;
  stack.init();
  uint2 leaf = make_uint2(0u, 0u), leaf2 = make_uint2(0u, 0u);   // triangles to test
  for(;;) {
    if(__popc(idle) >= kIdleLanes) {
      if(next >= end && more) {
        const uint32_t want = queue_next(count - end, warps);
        uint32_t b = 0;
        if(lane == 0) { b = atomicAdd(cursor, want); }
        next = warps * first + __shfl_sync(kWarpAll, b, 0);
        end = min(next + want, count);
        more = next < count;
        q.ahead(next, end);
      }
      if(next < end) {
        const uint32_t at = next + __popc(idle & lt);
        if(item == kNoItem && at < end) {
          item = at;
          q.load(item, s);
        }
        next += __popc(idle);
      } else if(idle == kWarpAll) {
        break;
      }
      if(next >= end && !more) {
        const uint32_t busy = __ballot_sync(kWarpAll, item != kNoItem);
        if(__popc(busy) <= kWideRays) {
          if(busy) {
            trace_wide<ANY_HIT, EXACT_MT, WT>(q, s, stack, leaf, leaf2, item, busy);
          }
          break;
        }
      }
    }
    // node steps; a lane with two nodes' triangles waits
    for(;;) {
      if(group_left(s) && leaf_empty(leaf2)) {
        const uint2 l = trav_node(s, q.scene(), stack);
        if(!leaf_empty(l)) {
          leaf2 = leaf;
          leaf = l;
        }
      }
      const uint32_t tri = __ballot_sync(kWarpAll, !leaf_empty(leaf));
      if(__popc(tri) >= kTriLanes) { break; }
      const uint32_t node = __ballot_sync(kWarpAll, group_left(s) && leaf_empty(leaf2));
      if(__popc(node) < kMinLanes) { break; }
      if(more && __popc(node | tri) <= 32 - kIdleLanes) { break; }
    }
    // triangle tests, one per lane and round
    uint32_t tri;
    do {
      if(!leaf_empty(leaf)) {
        if(trav_tri<ANY_HIT, EXACT_MT, WT>(s, q.scene(), leaf) && ANY_HIT) {
          leaf.y = 0u;
          leaf2.y = 0u;
          s.group.y = 0u;
          s.sp = 0;
        }
        if(leaf_empty(leaf)) {
          leaf = leaf2;
          leaf2.y = 0u;
        }
      }
      tri = __ballot_sync(kWarpAll, !leaf_empty(leaf));
    } while(__popc(tri) >= kMinLanes);
    const bool mine = item != kNoItem && !group_left(s) && leaf_empty(leaf);
    if(__any_sync(kWarpAll, mine)) {
      q.done(mine, item, s);
      if(mine) { item = kNoItem; }
    }
    idle = __ballot_sync(kWarpAll, item == kNoItem);
  }
}

}  // namespace dort_gpu
