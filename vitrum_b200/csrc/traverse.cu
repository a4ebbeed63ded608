// traverse.cu -- closest-hit and any-hit traversal of the 8-wide compressed BVH.
//
// One thread per ray.  Per wide node: five 128-bit read-only loads, the
// eight quantised child slabs tested against [tmin, closest] in the ray's
// octant order, internal-child hits kept as an 8-bit group mask and leaf
// hits as a 32-bit triangle mask (Ylitie et al. 2017 node groups).  The
// group stack is a per-thread local array (L1-cached where touched).  Triangles use
// the reference's watertight f32 test (tri_intersect.cuh); the accepted hit
// is then re-evaluated once in float-float arithmetic for the reported t
// and barycentrics.
//
// Slab conservativeness: with s = 2^e, a child plane at p + q*s is evaluated as
// fma(1 + q/2^15, a, c), a = (2^15*s)*invd and c = (p - o)*invd -+ err - a (the
// byte q becomes the float 1 + q/2^15 by one byte permute, so no conversion or
// subtraction is needed per child).  With u = 2^-24 and invd within 2u of 1/d (rcp.approx), the
// rounding errors are below 4u*|invd|*(|p| + |o|) for (p - o)*invd, 3u of its
// value for the margin, c and the result, 2u*255*s*|invd| for q*s*invd, and
// 2^15*u*s*|invd| + 2u*255*s*|invd| for c's cancelled term and the last
// rounding: under |invd|*(7u*(|p| + |o|) + 0.0021*s).  The near distance is
// lowered and the far distance raised by |invd|*(8u*(|p| + |o|) + 0.00225*s),
// which widens a box by a quarter of a percent of a grid cell.  Where a
// overflows both distances are NaN, which the maxima and minima ignore: that
// axis does not cull.  With the smallest component that set_ray lets through
// this takes a cell above 10^4 (10^4 lengths for directions above unit length,
// 10^16 for those below 1e-12).  A direction that is zero or not finite, which no
// triangle test accepts, is not traced at all.
// Together with outward quantisation this never culls a box the exact ray
// touches.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "bvh_types.h"
#include "traverse.h"
#include "tc_sm100.cuh"
#include "tri_intersect.cuh"

namespace vt {

namespace {

constexpr int kBlock = 128;
// Group-stack entries a ray can use: the launcher passes the tree's bound
// (two per wide level plus a few; 18 for an 8-level tree), capped here; a tree
// that needs more reports kTraceStackOverflow.  A shared-memory stack sized to
// that bound traced 1.9 % slower on the box room and 4 % slower on the
// instanced cloud than this local-memory one (shared memory taken from L1).
constexpr int kMaxStack = 64;
// Breadth-first prefix of the tree below `root` that every CTA copies into
// shared memory at start when staging is on: the root and its children and
// grandchildren of a full 8-wide tree (1 + 8 + 64), 5840 bytes.
constexpr uint32_t kHotNodes = 73;
constexpr long long kStagingWaitCycles = 2000000000LL;  // about a second

__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
// three-input f32 max / min (sm_100)
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
__device__ __forceinline__ float lo32(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi32(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }
// (near, far) t of one axis: bytes `sel` of the near / far words become the floats
// 1 + q / 2^15 (a byte placed in the mantissa), then one packed FMA with (adj, adj) and
// the offsets
__device__ __forceinline__ uint64_t slab2(uint32_t nw, uint32_t fw, uint32_t sel, uint64_t adj2, uint64_t off2) {
  const uint32_t a = __byte_perm(nw, 0x3F800000u, 0x7604u | (sel << 4)),
                 b = __byte_perm(fw, 0x3F800000u, 0x7604u | (sel << 4));
  uint64_t q, t;
  asm("mov.b64 %0, {%1, %2};" : "=l"(q) : "r"(a), "r"(b));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(t) : "l"(q), "l"(adj2), "l"(off2));
  return t;
}

struct Slab {
  float adj, on, of;  // scale, near and far offset for the factor 1 + q / 2^15
};

__device__ __forceinline__ Slab make_slab(float p, float e_bits, float inv, float o) {
  const float s = e_bits;                 // 2^e
  const float org = (p - o) * inv;
  const float err = fabsf(inv) * fmaf(2.25e-3f, s, 4.76837158203125e-7f * (fabsf(p) + fabsf(o)));
  Slab r;
  r.adj = (32768.0f * s) * inv;  // (in this order: 2^15 * inv alone overflows for short directions)
  r.on = (org - err) - r.adj;
  r.of = (org + err) - r.adj;
  return r;
}

// Per-lane ray state of the persistent kernel.
struct LaneRay {
  float tmin, closest;
  float ix, iy, iz;
  uint32_t oct;
  int best;  // triangle record index of the closest hit so far
};

// Per-ray traversal constants for origin o and direction d (world ray, or an
// instance's local ray: d is not renormalised, so t is the same in both).  The
// origin and direction are kept once, in the watertight test's state.  False: the
// direction is zero or not finite, nothing can be hit, and the tree is not entered
// (the slabs of such a ray cull nothing: 26 of them among 262,144 rays through
// 65,536 triangles took 35 ms, the batch without them 0.27).
__device__ __forceinline__ bool set_ray(LaneRay& R, TravRay& wr, float ox, float oy, float oz, float dx, float dy,
                                        float dz) {
  float m;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(fabsf(dx)), "f"(fabsf(dy)));
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(m) : "f"(fabsf(dz)));
  // A component near zero is taken as `least`: 1e-30, of directions above unit
  // length 1e-30 of the largest component, of those below 1e-12 1e-18 of it (the
  // ray drifts by that share of its way, far inside the slab margins); never a
  // subnormal, whose reciprocal overflows.  1e-30 of the largest at every length
  // left axis-parallel rays of length 1e-6 without culling: 199 ms instead of 0.21
  // for 262,144 of them.
  const float least = fmaxf(fmaxf(1e-30f * m, fminf(1e-30f, 1e-18f * m)), 1.17549435e-38f);
  auto inverse = [least](float d) {
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(fabsf(d) > least ? d : copysignf(least, d)));
    return r;
  };
  R.ix = inverse(dx); R.iy = inverse(dy); R.iz = inverse(dz);
  R.oct = (R.ix < 0.0f ? 4u : 0u) | (R.iy < 0.0f ? 2u : 0u) | (R.iz < 0.0f ? 1u : 0u);
  wr = trav_setup(ox, oy, oz, dx, dy, dz);
  return m > 0.0f && m < CUDART_INF_F;
}

// Does the ray pass slot j of the node at nb within [tmin, closest]?  (one slot
// of the packed test below: the same operations)
__device__ __forceinline__ bool slot_hit(const uint8_t* nb, uint32_t j, const LaneRay& R, float tmin, float closest,
                                         const Slab& sx, const Slab& sy, const Slab& sz) {
  auto plane = [](uint32_t q, float adj, float off) {
    return fmaf(__uint_as_float(q * 256u + 0x3F800000u), adj, off);
  };
  const uint32_t nx = ((R.oct & 4u) ? 56u : 32u) + j, ny = ((R.oct & 2u) ? 64u : 40u) + j,
                 nz = ((R.oct & 1u) ? 72u : 48u) + j;
  const uint32_t fx = ((R.oct & 4u) ? 32u : 56u) + j, fy = ((R.oct & 2u) ? 40u : 64u) + j,
                 fz = ((R.oct & 1u) ? 48u : 72u) + j;
  const uint32_t qnx = __ldg(nb + nx), qny = __ldg(nb + ny), qnz = __ldg(nb + nz);
  const uint32_t qfx = __ldg(nb + fx), qfy = __ldg(nb + fy), qfz = __ldg(nb + fz);
  const float tn = max3f(plane(qnx, sx.adj, sx.on), plane(qny, sy.adj, sy.on),
                         fmaxf(plane(qnz, sz.adj, sz.on), tmin));
  const float tf = min3f(plane(qfx, sx.adj, sx.of), plane(qfy, sy.adj, sy.of),
                         fminf(plane(qfz, sz.adj, sz.of), closest));
  return !(__float_as_uint(tf - tn) >> 31);
}

// Reorders an 8-bit slot mask into key order: bit s moves to bit s ^ oct.
__device__ __forceinline__ uint32_t xor_permute8(uint32_t m, uint32_t oct) {
  if (oct & 1u) m = ((m & 0x55u) << 1) | ((m >> 1) & 0x55u);
  if (oct & 2u) m = ((m & 0x33u) << 2) | ((m >> 2) & 0x33u);
  if (oct & 4u) m = ((m & 0x0Fu) << 4) | ((m >> 4) & 0x0Fu);
  return m;
}

// Spreads bit s of an 8-bit mask to nibble s (0xF) of a 32-bit word.
__device__ __forceinline__ uint32_t nibble_spread8(uint32_t m) {
  m = (m | (m << 12)) & 0x000F000Fu;
  m = (m | (m << 6)) & 0x03030303u;
  m = (m | (m << 3)) & 0x11111111u;
  return m * 15u;
}

// Resident CTAs per SM the register budget is cut for (80 registers).  Measured
// (B200) at 5 / 6 / 7 / 8: the 1,048,576-ray query 914 / 854 / 862 / 884 us, the
// box-room frame 24.6 / 23.0 / 22.6 / 22.7 ms, the instanced frame 22.0 / 21.0 /
// 21.0 / 21.5 ms.
constexpr int kTraceBlocks = 6;

// Idle lanes a warp gathers before it refills them.  Setting a ray up costs
// about as much as expanding a node and a warp of the box-room frame finishes
// 4.4 rays per iteration: refilling every idle lane at once ran the set-up in
// 94 % of the iterations for those few lanes.  Measured at 4 / 8 / 12: box-room
// frame 23.5 / 23.0 / 23.2 ms, instanced frame 21.0 / 21.0 / 21.3 ms, query 840 /
// 853 / 891 us.
constexpr int kRefillLanes = 8;

// The last rays of an occlusion query's warp whose pool is spent (single-level
// trees; at most kTailRays, the lanes of `live`): eight lanes go on with each, lane
// j at slot j of a node and at that slot's triangles, from where the ray stands --
// its next node (`expand`), its triangle groups (tb, th), (ub, uh) and its stack,
// which moves to the group's first lane.  Any order finds the same answer.  Such a
// launch ends with its longest rays, each some 600 dependent instructions a step
// in the loop: 300,001 segments in a room of 262,146 triangles 236 -> 170 us,
// 20,000 124 -> 83, 30,000 in one of 16,384 69 -> 54, 30,000 through 65,536 loose
// triangles 126 -> 121.  Closest hits gained less (30,000 in the room 147 -> 121 us)
// and lost elsewhere (the loop beside it 2.7 % slower, 60,000 through loose triangles
// 162 -> 172); waiting 8 to 32 iterations before the change was slower in both.
constexpr int kTailRays = 4;
__device__ __noinline__ void finish_occlusion(const uint4* nodes, const float4* tris, const float4* rays,
                                              uint8_t* occluded, int* status, int stk, uint2* stack, uint32_t live,
                                              uint32_t ray, uint32_t node, bool expand, int sp, uint32_t tb,
                                              uint32_t th, uint32_t ub, uint32_t uh) {
  constexpr uint32_t kFull = 0xFFFFFFFFu;
  const uint32_t lane = threadIdx.x & 31u, j = lane & 7u, shift = lane & 24u;
  // group g takes the g-th live lane's ray
  uint32_t rest = live;
  for (uint32_t g = lane >> 3; g > 0; --g) rest &= rest - 1u;
  bool alive = rest != 0;
  const int own = alive ? __ffs(rest) - 1 : (int)lane;
  // (all lanes read entry i of their own stacks before any first lane writes its own)
  const int deepest = __reduce_max_sync(kFull, (live >> lane) & 1u ? sp : 0);
  for (int i = 0; i < deepest; ++i) {
    uint2 g = stack[i];
    g.x = __shfl_sync(kFull, g.x, own);
    g.y = __shfl_sync(kFull, g.y, own);
    if (j == 0) stack[i] = g;
  }
  ray = __shfl_sync(kFull, ray, own);
  node = __shfl_sync(kFull, node, own);
  expand = __shfl_sync(kFull, expand ? 1 : 0, own) != 0;
  sp = __shfl_sync(kFull, sp, own);
  tb = __shfl_sync(kFull, tb, own);
  th = __shfl_sync(kFull, th, own);
  ub = __shfl_sync(kFull, ub, own);
  uh = __shfl_sync(kFull, uh, own);
  LaneRay R;
  TravRay wr;
  if (alive) {
    const float4 r0 = __ldg(rays + 2 * (size_t)ray), r1 = __ldg(rays + 2 * (size_t)ray + 1);
    R.tmin = r0.w;
    R.closest = r1.w;
    set_ray(R, wr, r0.x, r0.y, r0.z, r1.x, r1.y, r1.z);
  }
  while (__ballot_sync(kFull, alive)) {
    // ---- the next node, once no triangles are in hand: this lane's slot
    const bool step = alive && expand && th == 0;
    bool hit = false;
    uint32_t imask = 0, base = 0, valid = 0;
    if (step) {
      const uint4* np = nodes + (size_t)node * 5;
      const uint4 w0 = __ldg(np), w1 = __ldg(np + 1);
      const uint32_t e = w0.w;
      const Slab sx = make_slab(__uint_as_float(w0.x), __uint_as_float((e & 0xFFu) << 23), R.ix, wr.o[0]);
      const Slab sy = make_slab(__uint_as_float(w0.y), __uint_as_float(((e >> 8) & 0xFFu) << 23), R.iy, wr.o[1]);
      const Slab sz = make_slab(__uint_as_float(w0.z), __uint_as_float(((e >> 16) & 0xFFu) << 23), R.iz, wr.o[2]);
      hit = slot_hit(reinterpret_cast<const uint8_t*>(np), j, R, R.tmin, R.closest, sx, sy, sz);
      imask = e >> 24;
      base = w1.x;
      tb = w1.y;
      valid = w1.z;
    }
    const uint32_t hm = (__ballot_sync(kFull, hit) >> shift) & 0xFFu;
    uint32_t nh = 0;
    if (step) {
      expand = false;
      nh = xor_permute8(hm & imask, R.oct);
      th = nibble_spread8(hm & ~imask) & valid;
    }
    // ---- the triangles in hand, a slot's one after the other
    bool found = false;
    uint32_t nib = alive ? (th >> (4u * j)) & 0xFu : 0u;
#pragma unroll 1
    while (__ballot_sync(kFull, nib != 0)) {
#pragma unroll 1
      for (int rep = 0; rep < 1; ++rep) {
        if (nib == 0) break;
        const float4* rec = tris + 4 * (size_t)(tb + 4u * j + (uint32_t)(__ffs(nib) - 1));
        nib &= nib - 1u;
        const float4 a = __ldg(rec), b = __ldg(rec + 1), c = __ldg(rec + 2);
        const uint32_t fl = __float_as_uint(c.w);
        if (fl & VT_MATERIAL_NO_SHADOW) break;
        found = found || wt_candidate(wr, rec, a, b, c, R.tmin, R.closest, (fl & VT_MATERIAL_SINGLE_SIDED) != 0) >= 0.0f;
      }
    }
    th = 0;
    const bool blocked = ((__ballot_sync(kFull, found) >> shift) & 0xFFu) != 0;
    // ---- what comes next (the group's lanes agree)
    const bool go = alive && !blocked && !expand, pop = go && nh == 0 && uh == 0 && sp > 0;
    uint2 g = make_uint2(0u, 0u);
    if (pop && j == 0) g = stack[sp - 1];
    g.x = __shfl_sync(kFull, g.x, (int)shift);
    g.y = __shfl_sync(kFull, g.y, (int)shift);
    bool done = alive && blocked;
    if (go) {
      if (nh == 0 && uh) {
        tb = ub;
        th = uh;
        uh = 0;
      } else if (pop) {
        --sp;
        if (g.x & 0x80000000u) {
          base = g.x & 0x7FFFFFFFu;
          nh = g.y & 0xFFu;
          imask = g.y >> 8;
        } else {
          tb = g.x;
          th = g.y;
        }
      } else if (nh == 0) {
        done = true;
      }
      if (nh) {
        const uint32_t slot = (uint32_t)(__ffs(nh) - 1) ^ R.oct;
        nh &= nh - 1u;
        node = base + __popc(imask & ((1u << slot) - 1u));
        expand = true;
        if (nh) {
          if (sp < stk) {
            if (j == 0) stack[sp] = make_uint2(base | 0x80000000u, nh | (imask << 8));
            ++sp;
          } else {
            atomicOr(status, kTraceStackOverflow);
          }
        }
      }
    }
    if (done) {
      alive = false;
      if (j == 0) occluded[ray] = blocked ? 1 : 0;
    }
  }
}

template <bool ANY, bool TWO, bool HOT>
__global__ void __launch_bounds__(kBlock, kTraceBlocks)
    k_trace(const uint4* __restrict__ nodes, const float4* __restrict__ tris,
                                                  const float4* __restrict__ rays, size_t n,
                                                  int4* __restrict__ hits, uint8_t* __restrict__ occluded,
                                                  int* __restrict__ status,
                                                  unsigned long long* __restrict__ ray_counter,
                                                  const uint32_t* __restrict__ n_dev,
                                                  const float4* __restrict__ insts, uint32_t root,
                                                  const uint32_t* __restrict__ roots, uint32_t hot_count,
                                                  int stk, long long stage_wait,
                                                  const uint32_t* __restrict__ order,
                                                  const float4* __restrict__ inst_table) {
  // Persistent warps, one ray per lane.  Every iteration each live lane
  // (1) expands at most one wide node, (2) runs at most one watertight
  // triangle test from a two-entry queue of triangle groups, and (3) picks
  // its next node without waiting for its queued triangles.  Node work and
  // triangle work therefore proceed in lock-step phases with most lanes
  // busy in each, and a lane whose ray finished takes the next unclaimed
  // ray from its warp's pool (one atomicAdd per kChunk rays).
  // The group stack is a per-thread local array: the hardware interleaves it
  // across the warp, it is cached in L1 only where it is touched (rays rarely
  // go deep), and no shared memory is reserved for it, so the SM keeps its
  // largest L1 for nodes and triangle records.  `stk` <= kMaxStack entries are
  // used.  Dynamic shared memory holds only the hot_count staged nodes (80
  // bytes each) starting at nodes[root].
  extern __shared__ __align__(16) uint4 hot_mem[];
  __shared__ uint64_t hot_bar;
  uint2 stack[kMaxStack];
  const uint4* const hot = hot_mem;
  uint32_t hot_n = hot_count;  // staged nodes this CTA reads from shared memory
  if (HOT && hot_count) {
    // one bulk copy (TMA engine, no multicast) into shared memory, completed
    // on an mbarrier by transaction bytes
    if (threadIdx.x == 0) {
      const uint32_t bar = tc::smem_u32(&hot_bar), bytes = hot_count * 80u;
      tc::mbar_init(&hot_bar, 1);
      tc::fence_mbar_init();
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                   ::"r"(tc::smem_u32(hot)), "l"(nodes + (size_t)root * 5), "r"(bytes), "r"(bar)
                   : "memory");
    }
    __syncthreads();
    if (!tc::mbar_wait(&hot_bar, 0, stage_wait)) {
      // report, let a late copy land (full limit) so nothing writes this
      // CTA's shared memory after it, and traverse from global memory: the
      // results stay complete, the host reads the status bit
      atomicOr(status, kTraceStagingWait);
      tc::mbar_wait(&hot_bar, 0, kStagingWaitCycles);
      hot_n = 0;
    }
  }
  const uint32_t lane = threadIdx.x & 31u;
  constexpr uint32_t kFull = 0xFFFFFFFFu;
  // stack entry tags in x: bit 31 node group, bit 30 instance group, both: return
  // marker of an instance (two-level only); neither: triangle group
  constexpr uint32_t kNodeGroup = 0x80000000u;
  constexpr uint32_t kInstGroup = 0x40000000u;
  constexpr uint32_t kTagMask = 0xC0000000u;
  // rays per pool refill: small enough to spread short launches over all warps
  // (16 / 32 / 64: instanced frame 25.1 / 24.7 / 25.7 ms, box room 26.7 / 25.9 /
  // 25.5 ms, a 1,000-ray query 55 / 54 / 98 us)
  constexpr uint32_t kChunk = 32;

  bool live = false, exhausted = false;
  uint32_t ray = 0, pool_next = 0, pool_end = 0;
  const uint32_t n32 = n_dev ? *n_dev : (uint32_t)n;
  LaneRay R;
  TravRay wr;
  float wox = 0.f, woy = 0.f, woz = 0.f, wdx = 0.f, wdy = 0.f, wdz = 0.f;  // world ray (two-level)
  int cur_inst = -1, best_inst = -1;
  int best_mat = -1;       // material word of the closest hit so far (single-level)
  uint32_t cur_flags = 0;  // material flags of the instance being traversed (two-level)
  uint32_t gbase = 0, ghits = 0, gimask = 0, node = 0;
  uint32_t q0b = 0, q0m = 0, q1b = 0, q1m = 0;  // triangle-group queue (base, hit mask)
  bool expand = false;
  int sp = 0;

  while (true) {
    // ---- refill idle lanes from the warp's ray pool
    const uint32_t idle = __ballot_sync(kFull, !live);
    if (ANY && !TWO && exhausted && pool_next >= pool_end && __popc(idle) >= 32 - kTailRays) break;
    // (a warp whose pool is spent only counts them; the last lane to finish ends it)
    if (idle == kFull || (__popc(idle) >= kRefillLanes && !(exhausted && pool_next >= pool_end))) {
      if (pool_next >= pool_end && !exhausted) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(ray_counter, (unsigned long long)kChunk);
        base = __shfl_sync(kFull, base, 0);
        pool_next = (uint32_t)(base < n32 ? base : n32);
        pool_end = base + kChunk < n32 ? (uint32_t)(base + kChunk) : n32;
        exhausted = base + kChunk >= n32;
      }
      const uint32_t avail = pool_end > pool_next ? pool_end - pool_next : 0u;
      const uint32_t rank = __popc(idle & ((1u << lane) - 1u));
      if (!live && rank < avail) {
        ray = pool_next + rank;
        if (order) ray = __ldg(order + ray);  // trace order differs from queue order
        const float4 r0 = __ldg(rays + 2 * (size_t)ray), r1 = __ldg(rays + 2 * (size_t)ray + 1);
        R.tmin = r0.w;
        R.closest = r1.w;
        expand = set_ray(R, wr, r0.x, r0.y, r0.z, r1.x, r1.y, r1.z);  // (else it finishes below, a miss)
        if (TWO) { wox = r0.x; woy = r0.y; woz = r0.z; wdx = r1.x; wdy = r1.y; wdz = r1.z; }
        cur_inst = best_inst = -1;
        cur_flags = 0;
        R.best = -1;
        gbase = ghits = gimask = 0;
        q0m = q1m = 0;
        node = roots ? __ldg(roots + ray) : root;
        sp = 0;
        live = true;
      }
      const uint32_t cnt = (uint32_t)__popc(idle);
      pool_next += avail < cnt ? avail : cnt;
      if (exhausted && pool_next >= pool_end && __ballot_sync(kFull, live) == 0) break;
    }
    if (!live) continue;

    // ---- (1) expand one node
    if (expand) {
      expand = false;
      const uint4* np = nodes + (size_t)node * 5;
      uint4 w0, w1, w2, w3, w4;
      if (HOT) {
        // staged prefix from shared memory, the rest from global (one generic load path)
        const uint32_t hrel = node - root;
        if (hrel < hot_n) np = hot + hrel * 5;
        w0 = np[0]; w1 = np[1]; w2 = np[2]; w3 = np[3]; w4 = np[4];
      } else {
        w0 = __ldg(np); w1 = __ldg(np + 1); w2 = __ldg(np + 2); w3 = __ldg(np + 3); w4 = __ldg(np + 4);
      }
      const uint32_t e = w0.w;
      const Slab sx = make_slab(__uint_as_float(w0.x), __uint_as_float((e & 0xFFu) << 23), R.ix, wr.o[0]);
      const Slab sy = make_slab(__uint_as_float(w0.y), __uint_as_float(((e >> 8) & 0xFFu) << 23), R.iy, wr.o[1]);
      const Slab sz = make_slab(__uint_as_float(w0.z), __uint_as_float(((e >> 16) & 0xFFu) << 23), R.iz, wr.o[2]);
      const uint32_t imask = e >> 24;
      const bool nx = R.oct & 4u, ny = R.oct & 2u, nz = R.oct & 1u;
      // q words: lo_x = w2.xy, lo_y = w2.zw, lo_z = w3.xy, hi_x = w3.zw, hi_y = w4.xy, hi_z = w4.zw
      const uint32_t nx0 = nx ? w3.z : w2.x, nx1 = nx ? w3.w : w2.y;
      const uint32_t fx0 = nx ? w2.x : w3.z, fx1 = nx ? w2.y : w3.w;
      const uint32_t ny0 = ny ? w4.x : w2.z, ny1 = ny ? w4.y : w2.w;
      const uint32_t fy0 = ny ? w2.z : w4.x, fy1 = ny ? w2.w : w4.y;
      const uint32_t nz0 = nz ? w4.z : w3.x, nz1 = nz ? w4.w : w3.y;
      const uint32_t fz0 = nz ? w3.x : w4.z, fz1 = nz ? w3.y : w4.w;
      const uint64_t ax2 = pack2(sx.adj, sx.adj), ay2 = pack2(sy.adj, sy.adj), az2 = pack2(sz.adj, sz.adj);
      const uint64_t ox2 = pack2(sx.on, sx.of), oy2 = pack2(sy.on, sy.of), oz2 = pack2(sz.on, sz.of);
      uint32_t hm = 0;  // slot-indexed hit mask
#pragma unroll
      for (int j = 7; j >= 0; --j) {
        const uint32_t sel = (uint32_t)(j & 3);
        // near and far plane of one axis: one packed FMA of the two bytes as floats
        const uint64_t tx = slab2(j < 4 ? nx0 : nx1, j < 4 ? fx0 : fx1, sel, ax2, ox2);
        const uint64_t ty = slab2(j < 4 ? ny0 : ny1, j < 4 ? fy0 : fy1, sel, ay2, oy2);
        const uint64_t tz = slab2(j < 4 ? nz0 : nz1, j < 4 ? fz0 : fz1, sel, az2, oz2);
        const float tn = max3f(lo32(tx), lo32(ty), fmaxf(lo32(tz), R.tmin));
        const float tf = min3f(hi32(tx), hi32(ty), fminf(hi32(tz), R.closest));
        hm = __funnelshift_l(__float_as_uint(tf - tn), hm, 1);
      }
      hm = ~hm & 0xFFu;  // the differences' signs, shifted in from slot 7 down: no sign (or NaN), a hit
      const uint32_t nh = xor_permute8(hm & imask, R.oct);
      uint32_t th = nibble_spread8(hm & ~imask) & w1.z;
      gbase = w1.x;
      ghits = nh;
      gimask = imask;
      if (TWO && cur_inst < 0 && th) {
        // top level: the leaf records are instances, entered through the stack
        // before this node's internal children (which wait below them)
        if (ghits) {
          if (sp < stk) {
            stack[sp] = make_uint2(gbase | kNodeGroup, ghits | (gimask << 8));
            ++sp;
          } else {
            atomicOr(status, kTraceStackOverflow);
          }
          ghits = 0;
        }
        if (sp < stk) {
          stack[sp] = make_uint2(w1.y | kInstGroup, th);
          ++sp;
        } else {
          atomicOr(status, kTraceStackOverflow);
        }
        th = 0;
      }
      if (th) {
        if (q0m == 0) { q0b = w1.y; q0m = th; }
        else if (q1m == 0) { q1b = w1.y; q1m = th; }
        else if (sp < stk) { stack[sp] = make_uint2(w1.y, th); ++sp; }
        else {
          // no room anywhere: test the group now (correct, only slower)
          while (th) {
            const uint32_t tri = w1.y + (uint32_t)(__ffs(th) - 1);
            th &= th - 1;
            const float4* rec = tris + 4 * (size_t)tri;
            const uint32_t fl = __float_as_uint(__ldg(rec + 2).w) | cur_flags;
            if (ANY && (fl & VT_MATERIAL_NO_SHADOW)) continue;
            const float t = trav_exact(wr.o[0], wr.o[1], wr.o[2], wr.d[0], wr.d[1], wr.d[2], rec, fmaxf(R.tmin, 0.0f),
                                       R.closest, (fl & VT_MATERIAL_SINGLE_SIDED) != 0);
            if (t >= 0.0f) {
              R.closest = t;
              R.best = (int)tri;
              best_inst = cur_inst;
              if (!TWO) best_mat = __float_as_int(__ldg(rec + 1).w);
            }
          }
        }
      }
    }

    // ---- (2) one triangle test from the queue head.  Measured: two a step made
    // the query 4 % faster and the box-room frame 4 % slower; running the phase
    // only once 8 lanes want it or 4 wait for it, two tests at a time, made the
    // box room 3 % faster and the query and the instanced frame 4-6 % slower.
    // (A loop, so that the compiler brings the lanes together again behind it:
    // with a plain branch the lanes went on apart, 25 % slower; __syncwarp
    // between the phases, 20 %.)
    bool done = false;
#pragma unroll 1
    for (int rep = 0; rep < 1; ++rep) {
      if (q0m == 0) break;
      const uint32_t tri = q0b + (uint32_t)(__ffs(q0m) - 1);
      q0m &= q0m - 1;
      if (q0m == 0) { q0b = q1b; q0m = q1m; q1m = 0; }
      const float4* rec = tris + 4 * (size_t)tri;
      const float4 a = __ldg(rec), b = __ldg(rec + 1), c = __ldg(rec + 2);
      const uint32_t fl = __float_as_uint(c.w) | cur_flags;
      if (!(ANY && (fl & VT_MATERIAL_NO_SHADOW))) {
        const float t = wt_candidate(wr, rec, a, b, c, R.tmin, R.closest, (fl & VT_MATERIAL_SINGLE_SIDED) != 0);
        if (t >= 0.0f) {
          R.closest = t;
          R.best = (int)tri;
          best_inst = cur_inst;
          if (!TWO) best_mat = __float_as_int(b.w);
          if (ANY) done = true;
        }
      }
    }

    // ---- (3) next node: current group, else the top of the stack, one entry an
    // iteration (a triangle group joins the queue; leaving an instance goes on to
    // the entry below its marker, and one set_ray serves leaving and entering).
    // As a loop until a node was found, lanes that popped ran the common tail a
    // second time: query 975 -> 908 us, instanced frame 24.6 -> 22.2 ms, box room
    // 24.6 -> 24.3 ms without it.
#pragma unroll 1
    for (int rep = 0; rep < 1; ++rep) {
      if (done || expand) break;
      bool moved = false;
      float nox = 0.f, noy = 0.f, noz = 0.f, ndx = 0.f, ndy = 0.f, ndz = 0.f;
      if (ghits == 0 && sp > 0) {
        uint2 g = stack[sp - 1];
        if (TWO && (g.x & kTagMask) == kTagMask && q0m == 0) {
          // return marker: leave the instance, its queued triangles are tested
          --sp;
          cur_inst = -1;
          cur_flags = 0;
          moved = true;
          nox = wox; noy = woy; noz = woz; ndx = wdx; ndy = wdy; ndz = wdz;
          g = sp > 0 ? stack[sp - 1] : make_uint2(kTagMask, 0u);
        }
        const uint32_t tag = g.x & kTagMask;
        if (tag == kNodeGroup) {
          --sp;
          gbase = g.x & ~kNodeGroup;
          ghits = g.y & 0xFFu;
          gimask = g.y >> 8;
        } else if (TWO && tag == kInstGroup) {
          // enter the next instance of the group
          --sp;
          const uint32_t k = (uint32_t)(__ffs(g.y) - 1);
          const uint32_t rest = g.y & (g.y - 1);
          if (rest) { stack[sp] = make_uint2(g.x, rest); ++sp; }
          if (sp < stk) {
            stack[sp] = make_uint2(kTagMask, 0u);
            ++sp;
            const float4* ir = insts + 4 * (size_t)((g.x & ~kTagMask) + k);
            const float4 m0 = __ldg(ir), m1 = __ldg(ir + 1), m2 = __ldg(ir + 2);
            const uint4 meta = __ldg(reinterpret_cast<const uint4*>(ir + 3));
            nox = fmaf(m0.x, wox, fmaf(m0.y, woy, fmaf(m0.z, woz, m0.w)));
            noy = fmaf(m1.x, wox, fmaf(m1.y, woy, fmaf(m1.z, woz, m1.w)));
            noz = fmaf(m2.x, wox, fmaf(m2.y, woy, fmaf(m2.z, woz, m2.w)));
            ndx = fmaf(m0.x, wdx, fmaf(m0.y, wdy, m0.z * wdz));
            ndy = fmaf(m1.x, wdx, fmaf(m1.y, wdy, m1.z * wdz));
            ndz = fmaf(m2.x, wdx, fmaf(m2.y, wdy, m2.z * wdz));
            moved = true;
            cur_inst = (int)meta.y;
            cur_flags = meta.w;
            node = meta.x;
            expand = true;
          } else {
            atomicOr(status, kTraceStackOverflow);
          }
        } else if (tag == 0u && q1m == 0) {
          --sp;
          if (q0m == 0) { q0b = g.x; q0m = g.y; } else { q1b = g.x; q1m = g.y; }
        }
      }
      if (TWO && moved && !set_ray(R, wr, nox, noy, noz, ndx, ndy, ndz)) expand = false;
      if (ghits) {
        const uint32_t k = (uint32_t)(__ffs(ghits) - 1);
        ghits &= ghits - 1;
        const uint32_t slot = k ^ R.oct;
        node = gbase + __popc(gimask & ((1u << slot) - 1u));
        expand = true;
        if (ghits) {
          if (sp < stk) {
            stack[sp] = make_uint2(gbase | kNodeGroup, ghits | (gimask << 8));
            ++sp;
          } else {
            atomicOr(status, kTraceStackOverflow);  // stack capacity exceeded: result incomplete, reported to the host
          }
          ghits = 0;
        }
      }
      if (!expand && q0m == 0 && sp == 0) done = true;
    }
    if (!done) continue;

    // ---- ray finished: write its record, the lane is refilled next iteration
    live = false;
    if (ANY) {
      occluded[ray] = (uint8_t)(R.best >= 0 ? 1 : 0);
      continue;
    }
    // closest: (triangle record, watertight t, instance, material id); the
    // material lets shading skip the record -> material load.  k_refine_hits
    // turns the record into (source id, t, u, v) in a coalesced pass with every
    // lane busy
    int mat = -1;
    if (R.best >= 0) {
      if (!TWO) mat = best_mat;
      else mat = (best_inst >= 0 && inst_table) ? __float_as_int(__ldg(inst_table + 4 * (size_t)best_inst + 3).z)
                                                : __float_as_int(__ldg(tris + 4 * (size_t)R.best + 1).w);
    }
    hits[ray] = make_int4(R.best, __float_as_int(R.closest), best_inst, mat);
  }
  if (ANY && !TWO) {
    const uint32_t left = __ballot_sync(kFull, live);
    if (left)
      finish_occlusion(nodes, tris, rays, occluded, status, stk, stack, left, ray, node, expand, sp, q0b, q0m, q1b,
                       q1m);
  }
}

// The closest hits of a warp's four rays exactly as lanes of k_trace find them
// (single-level trees): the same nodes, tests and queue, step for step, so that of
// triangles hit at the same f32 t the same one wins.  For the rays k_trace_group
// cannot decide by t alone (`run`); called by whole warps, eight lanes a ray that
// test a node's slots side by side and agree on everything else.  A ray through a
// shared edge ends here, so all rays of a picture aligned with a mesh may: 1,000 and
// 16,384 such rays on a grid of 200,000 triangles took 116 and 145 us with one lane
// per ray, one of a warp's four rays after the other; so 56 and 66.
struct OrderedHit {
  int best, mat;
  float closest;
};
__device__ __noinline__ OrderedHit closest_in_order(bool run, const uint4* nodes, const float4* tris, const float4* rays,
                                                    uint32_t ray, uint32_t node, int stk, uint2* stack, int* status) {
  constexpr uint32_t kFull = 0xFFFFFFFFu;
  const uint32_t lane = threadIdx.x & 31u, j = lane & 7u, shift = lane & 24u;
  LaneRay R;
  TravRay wr;
  OrderedHit h{-1, -1, 0.0f};
  if (run) {
    const float4 r0 = __ldg(rays + 2 * (size_t)ray), r1 = __ldg(rays + 2 * (size_t)ray + 1);
    R.tmin = r0.w;
    h.closest = r1.w;
    set_ray(R, wr, r0.x, r0.y, r0.z, r1.x, r1.y, r1.z);
  }
  uint32_t gbase = 0, ghits = 0, gimask = 0, q0b = 0, q0m = 0, q1b = 0, q1m = 0;
  bool expand = true;
  int sp = 0;
  while (__ballot_sync(kFull, run)) {
    const bool step = run && expand;
    bool hit = false;
    uint32_t imask = 0, over = 0, over_base = 0;
    uint4 w1 = make_uint4(0u, 0u, 0u, 0u);
    if (step) {
      const uint4* np = nodes + (size_t)node * 5;
      const uint4 w0 = __ldg(np);
      w1 = __ldg(np + 1);
      const uint32_t e = w0.w;
      const Slab sx = make_slab(__uint_as_float(w0.x), __uint_as_float((e & 0xFFu) << 23), R.ix, wr.o[0]);
      const Slab sy = make_slab(__uint_as_float(w0.y), __uint_as_float(((e >> 8) & 0xFFu) << 23), R.iy, wr.o[1]);
      const Slab sz = make_slab(__uint_as_float(w0.z), __uint_as_float(((e >> 16) & 0xFFu) << 23), R.iz, wr.o[2]);
      hit = slot_hit(reinterpret_cast<const uint8_t*>(np), j, R, R.tmin, h.closest, sx, sy, sz);
      imask = e >> 24;
    }
    const uint32_t hm = (__ballot_sync(kFull, hit) >> shift) & 0xFFu;
    if (step) {
      expand = false;
      gbase = w1.x;
      ghits = xor_permute8(hm & imask, R.oct);
      gimask = imask;
      const uint32_t th = nibble_spread8(hm & ~imask) & w1.z;
      if (th) {
        if (q0m == 0) { q0b = w1.y; q0m = th; }
        else if (q1m == 0) { q1b = w1.y; q1m = th; }
        else if (sp < stk) {
          if (j == 0) stack[sp] = make_uint2(w1.y, th);
          ++sp;
        } else {
          over_base = w1.y;
          over = th;
        }
      }
    }
    __syncwarp();
    // the triangles that found no room, then the queue's next
    bool more = run && (over != 0 || q0m != 0);
#pragma unroll 1
    while (__ballot_sync(kFull, more)) {
      if (more) {
        const bool queued = over == 0;
        uint32_t tri;
        if (queued) {
          tri = q0b + (uint32_t)(__ffs(q0m) - 1);
          q0m &= q0m - 1;
          if (q0m == 0) { q0b = q1b; q0m = q1m; q1m = 0; }
        } else {
          tri = over_base + (uint32_t)(__ffs(over) - 1);
          over &= over - 1;
        }
        const float4* rec = tris + 4 * (size_t)tri;
        const float4 a = __ldg(rec), b = __ldg(rec + 1), c = __ldg(rec + 2);
        const float t = wt_candidate(wr, rec, a, b, c, R.tmin, h.closest,
                                     (__float_as_uint(c.w) & VT_MATERIAL_SINGLE_SIDED) != 0);
        if (t >= 0.0f) h = {(int)tri, __float_as_int(b.w), t};
        more = !queued && (over != 0 || q0m != 0);
      }
    }
    uint2 g = make_uint2(0u, 0u);
    if (run && ghits == 0 && sp > 0) g = stack[sp - 1];
    __syncwarp();
    if (run) {
      if (ghits == 0 && sp > 0) {
        if (g.x & 0x80000000u) {
          --sp;
          gbase = g.x & 0x7FFFFFFFu;
          ghits = g.y & 0xFFu;
          gimask = g.y >> 8;
        } else if (q1m == 0) {
          --sp;
          if (q0m == 0) { q0b = g.x; q0m = g.y; } else { q1b = g.x; q1m = g.y; }
        }
      }
      if (ghits) {
        const uint32_t slot = (uint32_t)(__ffs(ghits) - 1) ^ R.oct;
        ghits &= ghits - 1;
        node = gbase + __popc(gimask & ((1u << slot) - 1u));
        expand = true;
        if (ghits) {
          if (sp < stk) {
            if (j == 0) stack[sp] = make_uint2(gbase | 0x80000000u, ghits | (gimask << 8));
            ++sp;
          } else {
            atomicOr(status, kTraceStackOverflow);
          }
          ghits = 0;
        }
      }
      if (!expand && q0m == 0 && sp == 0) run = false;
    }
    __syncwarp();
  }
  return h;
}

// Small launches on single-level trees: eight lanes per ray, lane j at slot j of
// each node, four rays a warp.  With few rays a launch lasts as long as its
// longest ray, and one ray's step through k_trace is some 600 dependent
// instructions (1.2 us); here a node's eight slabs, and then up to eight of its
// triangles, are tested side by side.  A node's triangles are tested at once,
// where k_trace queues them behind the next node: the closest t is the same, and
// a ray that meets two triangles at it is left to closest_in_order.
template <bool ANY>
__global__ void __launch_bounds__(kBlock) k_trace_group(const uint4* __restrict__ nodes, const float4* __restrict__ tris,
                                                        const float4* __restrict__ rays, size_t n,
                                                        int4* __restrict__ hits, uint8_t* __restrict__ occluded,
                                                        int* __restrict__ status, const uint32_t* __restrict__ n_dev,
                                                        uint32_t root, const uint32_t* __restrict__ roots, int stk,
                                                        const uint32_t* __restrict__ order) {
  constexpr uint32_t kFull = 0xFFFFFFFFu;
  constexpr uint32_t kGroups = kBlock / 8;
  __shared__ uint2 stacks[kGroups][kMaxStack];  // (child base, hits | internal mask << 8)
  __shared__ uint32_t lists[kGroups][32];         // a node's triangles in slot order
  const uint32_t lane = threadIdx.x & 31u, j = lane & 7u, shift = lane & 24u;
  uint2* const stack = stacks[threadIdx.x >> 3];
  uint32_t* const list = lists[threadIdx.x >> 3];
  const uint32_t n32 = n_dev ? *n_dev : (uint32_t)n, at = blockIdx.x * kGroups + (threadIdx.x >> 3);
  const bool mine = at < n32;  // the launch has a group for every ray
  uint32_t ray = 0, node = 0;
  bool live = false, tied = false;  // tied: two triangles at the closest t so far
  LaneRay R;
  TravRay wr;
  int best_mat = -1, sp = 0;
  R.best = -1;
  if (mine) {
    ray = order ? __ldg(order + at) : at;
    const float4 r0 = __ldg(rays + 2 * (size_t)ray), r1 = __ldg(rays + 2 * (size_t)ray + 1);
    R.tmin = r0.w;
    R.closest = r1.w;
    live = set_ray(R, wr, r0.x, r0.y, r0.z, r1.x, r1.y, r1.z);  // (else a miss)
    node = roots ? __ldg(roots + ray) : root;
  }
  while (__ballot_sync(kFull, live)) {
    // ---- the node: this lane's slot
    bool hit = false;
    uint32_t imask = 0, child_base = 0, tri = 0, nib = 0, valid = 0;
    if (live) {
      const uint4* np = nodes + (size_t)node * 5;
      const uint8_t* nb = reinterpret_cast<const uint8_t*>(np);
      const uint4 w0 = __ldg(np), w1 = __ldg(np + 1);
      const uint32_t e = w0.w;
      const Slab sx = make_slab(__uint_as_float(w0.x), __uint_as_float((e & 0xFFu) << 23), R.ix, wr.o[0]);
      const Slab sy = make_slab(__uint_as_float(w0.y), __uint_as_float(((e >> 8) & 0xFFu) << 23), R.iy, wr.o[1]);
      const Slab sz = make_slab(__uint_as_float(w0.z), __uint_as_float(((e >> 16) & 0xFFu) << 23), R.iz, wr.o[2]);
      hit = slot_hit(nb, j, R, R.tmin, R.closest, sx, sy, sz);
      imask = e >> 24;
      child_base = w1.x;
      valid = w1.z;
      tri = w1.y + 4u * j;
      nib = hit && !((imask >> j) & 1u) ? (w1.z >> (4u * j)) & 0xFu : 0u;
    }
    const uint32_t hm = (__ballot_sync(kFull, hit) >> shift) & 0xFFu;
    // ---- its triangles, eight a round
    bool done = false;
    if (__ballot_sync(kFull, nib != 0)) {
      // (a slot's records are contiguous from its first)
      const uint32_t th = live ? nibble_spread8(hm & ~imask) & valid : 0u, count = (uint32_t)__popc(th);
      const uint32_t first = (uint32_t)__popc(th & ((1u << (4u * j)) - 1u)), own = (uint32_t)__popc(nib);
      for (uint32_t i = 0; i < own; ++i) list[first + i] = tri + i;
      __syncwarp();
      float found = CUDART_INF_F, closest = R.closest;
      int best = -1, mat = -1;
      bool equal = false;  // another triangle at this lane's closest, or at the ray's
#pragma unroll 1
      for (uint32_t i = j; __ballot_sync(kFull, i < count); i += 8) {
#pragma unroll 1
        for (int rep = 0; rep < 1; ++rep) {
          if (i >= count) break;
          const uint32_t r = list[i];
          const float4* rec = tris + 4 * (size_t)r;
          const float4 a = __ldg(rec), b = __ldg(rec + 1), c = __ldg(rec + 2);
          const uint32_t fl = __float_as_uint(c.w);
          if (ANY && (fl & VT_MATERIAL_NO_SHADOW)) break;
          // (the next float above a hit's t, so that an equal one shows)
          const bool held = best >= 0 || R.best >= 0;
          const float limit = !ANY && held ? __uint_as_float(__float_as_uint(closest) + 1u) : closest;
          const float t = wt_candidate(wr, rec, a, b, c, R.tmin, limit, (fl & VT_MATERIAL_SINGLE_SIDED) != 0);
          if (t >= 0.0f) {
            equal = held && t == closest;
            if (!equal) {
              closest = found = t;
              best = (int)r;
              mat = __float_as_int(b.w);
            }
          }
        }
      }
      __syncwarp();
      float m = found;
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) m = fminf(m, __shfl_xor_sync(kFull, m, o));
      const uint32_t win = (__ballot_sync(kFull, best >= 0 && found == m) >> shift) & 0xFFu;
      const uint32_t same = (__ballot_sync(kFull, equal && closest == fminf(m, R.closest)) >> shift) & 0xFFu;
      const int src = (int)shift + (win ? __ffs(win) - 1 : 0);
      best = __shfl_sync(kFull, best, src);
      mat = __shfl_sync(kFull, mat, src);
      if (win) {
        R.closest = m;
        R.best = best;
        best_mat = mat;
        tied = (win & (win - 1u)) != 0;
        if (ANY) done = true;
      }
      tied = tied || same != 0;
    }
    // ---- the next node (the group's lanes agree)
    uint32_t nh = xor_permute8(hm & imask, R.oct), base = child_base, im = imask;
    if (live && !done && nh == 0) {
      if (sp == 0) {
        done = true;
      } else {
        const uint2 g = stack[--sp];
        base = g.x;
        nh = g.y & 0xFFu;
        im = g.y >> 8;
      }
    }
    __syncwarp();
    if (live && !done) {
      const uint32_t slot = (uint32_t)(__ffs(nh) - 1) ^ R.oct;
      nh &= nh - 1;
      node = base + __popc(im & ((1u << slot) - 1u));
      if (nh) {
        if (sp < stk) {
          if (j == 0) stack[sp] = make_uint2(base, nh | (im << 8));
          ++sp;
        } else {
          atomicOr(status, kTraceStackOverflow);
        }
      }
    }
    __syncwarp();
    if (done) live = false;
  }
  if (ANY) {
    if (mine && j == 0) occluded[ray] = (uint8_t)(R.best >= 0 ? 1 : 0);
    return;
  }
  if (__ballot_sync(kFull, tied)) {
    const OrderedHit h = closest_in_order(tied, nodes, tris, rays, ray, roots && mine ? __ldg(roots + ray) : root, stk,
                                          stack, status);
    if (tied) {
      R.best = h.best;
      R.closest = h.closest;
      best_mat = h.mat;
    }
  }
  if (mine && j == 0) hits[ray] = make_int4(R.best, __float_as_int(R.closest), -1, R.best >= 0 ? best_mat : -1);
}

// Second pass of the closest-hit query: one thread per ray, float-float
// re-evaluation of the chosen triangle for t and barycentrics, record index
// replaced by the source triangle id (-1 and tmax for a miss).  Instance hits
// are re-evaluated in world space (the placed triangle against the world ray).
__global__ void __launch_bounds__(256) k_refine_hits(const float4* __restrict__ tris,
                                                      const float4* __restrict__ rays, size_t n,
                                                      int4* __restrict__ hits, const float4* __restrict__ inst_table,
                                                      const float4* __restrict__ inst_l2w,
                                                      int* __restrict__ inst_out) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int4 h = hits[i];
  if (inst_out) inst_out[i] = h.x < 0 ? -1 : h.z;
  if (h.x < 0) {
    hits[i] = make_int4(-1, h.y, 0, 0);
    return;
  }
  float4 r0 = __ldg(rays + 2 * i), r1 = __ldg(rays + 2 * i + 1);
  const float4* rec = tris + 4 * (size_t)(uint32_t)h.x;
  const float4 a = __ldg(rec), b = __ldg(rec + 1), c = __ldg(rec + 2);
  const float3 A = make_float3(a.x, a.y, a.z), B = make_float3(b.x, b.y, b.z), C = make_float3(c.x, c.y, c.z);
  float t = __int_as_float(h.y), u = 0.0f, v = 0.0f;
  float tr, ur, vr;
  const bool placed = inst_table && h.z >= 0;
  bool ok;
  if (placed && inst_l2w) {
    const float4* lr = inst_l2w + 3 * (size_t)h.z;
    ok = ff_refine_placed(make_float3(r0.x, r0.y, r0.z), make_float3(r1.x, r1.y, r1.z), __ldg(lr), __ldg(lr + 1),
                          __ldg(lr + 2), A, B, C, &tr, &ur, &vr);
  } else {
    if (placed) {
      // the instance's local ray, computed as the traversal computed it
      const float4* ir = inst_table + 4 * (size_t)h.z;
      const float4 m0 = __ldg(ir), m1 = __ldg(ir + 1), m2 = __ldg(ir + 2);
      const float ox = r0.x, oy = r0.y, oz = r0.z, dx = r1.x, dy = r1.y, dz = r1.z;
      r0.x = fmaf(m0.x, ox, fmaf(m0.y, oy, fmaf(m0.z, oz, m0.w)));
      r0.y = fmaf(m1.x, ox, fmaf(m1.y, oy, fmaf(m1.z, oz, m1.w)));
      r0.z = fmaf(m2.x, ox, fmaf(m2.y, oy, fmaf(m2.z, oz, m2.w)));
      r1.x = fmaf(m0.x, dx, fmaf(m0.y, dy, m0.z * dz));
      r1.y = fmaf(m1.x, dx, fmaf(m1.y, dy, m1.z * dz));
      r1.z = fmaf(m2.x, dx, fmaf(m2.y, dy, m2.z * dz));
    }
    ok = ff_refine(make_float3(r0.x, r0.y, r0.z), make_float3(r1.x, r1.y, r1.z), A, B, C, &tr, &ur, &vr);
  }
  if (ok) {
    t = tr;
    u = ur;
    v = vr;
  } else if (!placed) {
    // degenerate in float-float too: report the watertight barycentrics
    WtRay wr = wt_setup(r0.x, r0.y, r0.z, r1.x, r1.y, r1.z);
    WtHit wh;
    if (wt_intersect(wr, A, B, C, r0.w, &wh)) {
      u = wh.bary[1];
      v = wh.bary[2];
    }
  }
  hits[i] = make_int4((int)__float_as_uint(a.w), __float_as_int(t), __float_as_int(u), __float_as_int(v));
}

__global__ void k_watertight_eval(const float* __restrict__ cases, size_t n, vt_watertight_result* out) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float* c = cases + 16 * i;
  WtRay r = wt_setup(c[0], c[1], c[2], c[3], c[4], c[5]);
  WtHit h;
  vt_watertight_result res;
  res.hit = wt_intersect(r, make_float3(c[6], c[7], c[8]), make_float3(c[9], c[10], c[11]),
                         make_float3(c[12], c[13], c[14]), c[15], &h)
                ? 1
                : 0;
  res.t = res.hit ? h.t : CUDART_INF_F;
  res.bary[0] = res.hit ? h.bary[0] : 0.0f;
  res.bary[1] = res.hit ? h.bary[1] : 0.0f;
  res.bary[2] = res.hit ? h.bary[2] : 0.0f;
  res.side = res.hit ? h.side : 0;
  res.zero_edge_mask = res.hit ? h.mask : 0;
  out[i] = res;
}

// Resident CTAs per SM of one instantiation with `smem` dynamic bytes (the
// opt-in above 48 KB is set first).
template <class K>
int resident_per_sm(K kern, size_t smem) {
  if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kBlock, smem);
  return per_sm;
}

template <bool ANY, bool TWO>
void launch_trace_k(const TraceArgs& a, cudaStream_t s) {
  auto plain = k_trace<ANY, TWO, false>;
  auto staged = k_trace<ANY, TWO, true>;
  const int stk = std::min(std::max(a.stack_depth, 4), kMaxStack);
  const size_t stack_bytes = 0;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int per_sm = resident_per_sm(plain, stack_bytes);
  if (a.blocks_per_sm > 0) per_sm = std::min(per_sm, a.blocks_per_sm);
  // staged prefix: the nodes from nodes[root] on, for launches with one root,
  // a 16-aligned start (bulk copies), and no loss of resident CTAs
  uint32_t hot = 0;
  if (a.stage_nodes && !a.roots && a.node_count > a.root &&
      reinterpret_cast<uintptr_t>(a.nodes + (size_t)a.root * 5) % 16 == 0) {
    hot = (uint32_t)std::min<size_t>(kHotNodes, a.node_count - a.root);
    if (resident_per_sm(staged, stack_bytes + 80 * (size_t)hot) < per_sm) hot = 0;
  }
  // persistent grid: every resident slot once, never more blocks than rays need
  size_t grid = (size_t)std::max(1, sms) * (size_t)std::max(1, per_sm);
  grid = std::min(grid, (a.n + kBlock - 1) / kBlock);
  cudaMemsetAsync(a.counter, 0, sizeof(unsigned long long), s);
  (hot ? staged : plain)<<<(unsigned)grid, kBlock, stack_bytes + 80 * (size_t)hot, s>>>(
      a.nodes, a.tris, a.rays, a.n, a.hits, a.occluded, a.status, a.counter, a.n_dev, a.insts, a.root, a.roots, hot,
      stk, a.stage_wait_cycles > 0 ? a.stage_wait_cycles : kStagingWaitCycles, a.order, a.inst_table);
}

template <bool ANY>
void launch_trace_t(const TraceArgs& a, cudaStream_t s) {
  if (a.n == 0) return;
  // Up to here eight lanes per ray win (k_trace_group); measured, k_trace / group:
  // closest hits of 1,000 rays on 4,096 loose triangles 53 / 35 us, 20,000 56 / 64,
  // 12,000 on 65,536 133 / 88, 16,384 140 / 122, 30,000 143 / 146, 16,384 in a room of
  // 16,384 80 / 60, 44,000 85 / 96; occlusion of 12,000 in a room of 262,146 80 / 57,
  // 44,000 in one of 16,384 55 / 61, 30,000 on loose triangles 120 / 132
  constexpr size_t kGroupRays = 16384;
  if (!a.insts && a.n <= kGroupRays && !a.stage_nodes) {
    const int stk = std::min(std::max(a.stack_depth, 4), kMaxStack);
    const size_t groups = kBlock / 8, grid = (a.n + groups - 1) / groups;
    k_trace_group<ANY><<<(unsigned)grid, kBlock, 0, s>>>(a.nodes, a.tris, a.rays, a.n, a.hits, a.occluded, a.status,
                                                         a.n_dev, a.root, a.roots, stk, a.order);
    return;
  }
  if (a.insts) launch_trace_k<ANY, true>(a, s);
  else launch_trace_k<ANY, false>(a, s);
}

}  // namespace

void launch_trace_closest(const TraceArgs& a, cudaStream_t s) {
  launch_trace_t<false>(a, s);
  if (a.n)
    k_refine_hits<<<(unsigned)((a.n + 255) / 256), 256, 0, s>>>(a.tris, a.rays, a.n, a.hits, a.inst_table,
                                                                a.inst_l2w, a.inst_out);
}
void launch_trace_any(const TraceArgs& a, cudaStream_t s) { launch_trace_t<true>(a, s); }
void launch_trace_closest_records(const TraceArgs& a, cudaStream_t s) { launch_trace_t<false>(a, s); }

const char* trace_status_message(int status) {
  if (status & kTraceStackOverflow) return "traversal stack capacity exceeded";
  if (status & kTraceStagingWait) return "traversal node staging did not complete in time";
  return "traversal failed";
}

void launch_watertight_eval(const float* cases, size_t n, vt_watertight_result* out, cudaStream_t s) {
  if (n == 0) return;
  k_watertight_eval<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(cases, n, out);
}

}  // namespace vt
