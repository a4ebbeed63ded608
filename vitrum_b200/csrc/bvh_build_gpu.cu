// bvh_build_gpu.cu -- binned-SAH binary BVH built on the GPU, identical to
// the host build (and so to the reference's buildArrayBvh,
// packages/shared-bvh/src/buildArrayBvh.ts:342-780) word for word.
//
// Two regimes, by the size of a node:
//   large (more than kSmall triangles): level by level over all nodes of the
//     level at once, chunks of kChunk triangles per CTA, three launches a level:
//       k_bin      each chunk bins its triangles on the three axes in shared
//                  memory and adds its bins to the node's;
//       k_choose   one CTA per node, one warp per axis: sweeps, SAH costs, the
//                  split, each chunk's first left slot, the two children;
//       k_scatter  each chunk writes its part of the stable partition into the
//                  other index buffer and reduces the children's centroid bounds;
//     the levels follow one another on the stream without the host, which reads
//     the counters once per batch of levels;
//   small: k_small, one CTA per subtree: its boxes, index list and nodes stay in
//     shared memory down to the leaves, one warp per node of the current level
//     (nodes of at most eight triangles evaluate their splits directly, eight
//     lanes per axis).
// k_top numbers the tree (subtree sizes bottom up, preorder top down; left
// child = i + 1, right = i + 1 + size(left)) and k_emit writes the nodes.
//
// Bounds are minima / maxima of f32 coordinates, kept as order-preserving
// integer keys (-0 below +0: -0 wins a min tie, +0 a max tie, as in JS Math.min
// / Math.max), every other operation is a single IEEE-double operation
// (__dadd_rn & co., no contraction), so the decisions equal the host's.  A
// leaf's triangle offset is the start of its index range, which partitioning
// never moves again.  Where no split beats a leaf the range is sorted by
// (centroid on the widest axis, triangle index) and halved: by counting ranks
// inside a subtree, in one CTA's shared memory (k_sort) up to kSort triangles, by
// two stable device radix passes above.  The level waits for the host there, which
// launches the sorts: once a level, whatever the number of nodes.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include <cub/device/device_radix_sort.cuh>

#include "bvh_host.h"
#include "vt_common.h"

namespace vt {

namespace {

constexpr int kMaxBins = 256;       // binCount in [2, 256], as the options allow
// Subtrees of up to kSmall triangles are built by one CTA.  A level of large
// nodes costs three launches (about 25 us with the gaps), a subtree the serial
// depth of one warp per node: at 128 / 256 / 512 a binary tree of 262,146
// triangles took 1.19 / 1.03 / 1.02 ms, of 65,536 0.49 / 0.47 / 0.47 ms, of 2,047
// 0.25 / 0.25 / 0.32 ms (host clock, with the copies of the counters); one CTA
// per node and a host round trip per level took 20, 5.1 and 1.7 ms.
constexpr int kSmall = 256;
constexpr int kSmallThreads = 256;
constexpr int kChunk = 512;         // triangles of a large node per CTA
constexpr int kChunkThreads = 256;
// Nodes without a split of up to kSort triangles are sorted by one CTA each, side by
// side: what fits the 48 KB of shared memory that need no opt-in.  262,144 triangles
// of one centroid (1,023 nodes above kSmall in either tree) build in 27 ms, with
// every one of those nodes sorted on the host's call in 164; 256 groups of 1,024 in
// 5.5 instead of 110, as many spread triangles in 4.1.
constexpr uint32_t kSort = 4096;
constexpr int kSortThreads = 1024;
constexpr size_t kSortSmem = (size_t)kSort * 12;
constexpr uint32_t kFull = 0xFFFFFFFFu;

using u64 = unsigned long long;

// ---------------------------------------------------------------- keys
__device__ __forceinline__ uint32_t fkey(float f) {
  const uint32_t u = __float_as_uint(f);
  return u ^ ((u >> 31) ? 0xFFFFFFFFu : 0x80000000u);
}
__device__ __forceinline__ float funkey(uint32_t k) {
  return __uint_as_float(k ^ ((k >> 31) ? 0x80000000u : 0xFFFFFFFFu));
}
// Order-preserving 64-bit key of a double: key(a) < key(b) iff a < b, key(-0) < key(+0).
__device__ __forceinline__ u64 okey(double d) {
  const u64 u = (u64)__double_as_longlong(d);
  return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double okey_value(u64 k) {
  return __longlong_as_double((long long)((k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k));
}
__device__ __forceinline__ u64 warp_min64(u64 k) {
  const uint32_t hi = (uint32_t)(k >> 32), h = __reduce_min_sync(kFull, hi);
  const uint32_t lo = __reduce_min_sync(kFull, hi == h ? (uint32_t)k : 0xFFFFFFFFu);
  return ((u64)h << 32) | lo;
}
__device__ __forceinline__ u64 warp_max64(u64 k) {
  const uint32_t hi = (uint32_t)(k >> 32), h = __reduce_max_sync(kFull, hi);
  const uint32_t lo = __reduce_max_sync(kFull, hi == h ? (uint32_t)k : 0u);
  return ((u64)h << 32) | lo;
}

// centroid of one axis from the two bound keys
__device__ __forceinline__ double centroid(uint32_t lo, uint32_t hi) {
  return __dmul_rn(0.5, __dadd_rn((double)funkey(lo), (double)funkey(hi)));
}
__device__ __forceinline__ double half_sa(uint32_t mnx, uint32_t mny, uint32_t mnz, uint32_t mxx, uint32_t mxy,
                                          uint32_t mxz) {
  double dx = __dsub_rn((double)funkey(mxx), (double)funkey(mnx)), dy = __dsub_rn((double)funkey(mxy), (double)funkey(mny)),
         dz = __dsub_rn((double)funkey(mxz), (double)funkey(mnz));
  dx = dx > 0 ? dx : 0;
  dy = dy > 0 ? dy : 0;
  dz = dz > 0 ? dz : 0;
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dy), __dmul_rn(dy, dz)), __dmul_rn(dz, dx));
}
__device__ __forceinline__ double split_cost(double lsa, uint32_t lc, double rsa, uint32_t rc, double parent_sa) {
  const double num = __dadd_rn(__dmul_rn(lsa, (double)lc), __dmul_rn(rsa, (double)rc));
  return parent_sa > 0 ? __ddiv_rn(num, parent_sa) : num;
}
__device__ __forceinline__ int bin_of(double c, double cmin, double span, int bins) {
  const double x = __ddiv_rn(__dsub_rn(c, cmin), span);
  const double f = floor(__dmul_rn(x, (double)bins));
  return f < (double)(bins - 1) ? (f > 0.0 ? (int)f : 0) : bins - 1;
}
constexpr u64 kNoCost = ~0ull;  // above every finite cost's bits

// ---------------------------------------------------------------- large nodes
struct LNode {
  uint32_t begin, count, depth;
  int32_t left;                 // first child (the second follows it); -1: none (a small subtree)
  int32_t axis, split, decision;  // decision: 1 SAH split, 3 sorted halves
  uint32_t nl;
  uint32_t size, pre;           // subtree node count, preorder index
  uint32_t slot;                // bin slot within its level
  uint32_t chunk0, chunks;      // its chunks within its level
  uint32_t pad;
  uint32_t mn[3], mx[3];        // bounds (fkey)
  u64 cmn[3], cmx[3];           // centroid bounds (okey)
};

struct Ctl {
  uint32_t nodes;               // nodes created
  uint32_t small;               // small subtrees listed
  uint32_t large[2], chunks[2]; // of a level, by its parity
  uint32_t bad;                 // input errors: 1 vertex out of range, 2 not finite; 4 capacity (never)
  uint32_t depth_error;
  uint32_t stop;                // level + 1 whose fallback sorts wait for the host
  uint32_t big;                 // one of them is above kSort
  uint32_t levels;              // levels of large nodes processed
  uint32_t max_depth;           // deepest node
  uint32_t total;               // nodes of the finished tree
  uint32_t mark[kMaxBinaryDepth + 2];  // nodes of depth <= level
};

// Device arrays of one build, carved out of one scratch block.
struct Work {
  Ctl* ctl;
  LNode* nodes;
  uint4* boxes;                 // 2 per triangle: (lo keys, -), (hi keys, -)
  uint32_t* idx[2];             // index buffers by level parity
  uint32_t* list[2];            // large nodes of a level
  uint32_t* chunk_node[2];      // node of each chunk of a level
  uint32_t* chunk_left;         // triangles left of the split in the node's earlier chunks
  uint32_t* hist;               // per chunk: counts per axis and bin
  uint32_t* bins[2];            // per slot: [axis][mn xyz, mx xyz, count][bin]
  uint32_t* small;              // small subtrees
  BinaryNode* temp;             // subtrees' nodes in their own preorder, at 2 * begin
  uint32_t ntri, node_cap, max_chunks, max_large;
  int nbins, max_leaf, max_depth;
};

__device__ __forceinline__ uint32_t bin_identity(int k) { return k < 3 ? 0xFFFFFFFFu : 0u; }

__device__ __forceinline__ void init_node(LNode& n, uint32_t begin, uint32_t count, uint32_t depth) {
  n.begin = begin;
  n.count = count;
  n.depth = depth;
  n.left = -1;
  n.axis = -1;
  n.split = 0;
  n.decision = 0;
  n.nl = 0;
  n.size = 1;
  n.pre = 0;
  n.slot = n.chunk0 = n.chunks = n.pad = 0;
  for (int k = 0; k < 3; ++k) {
    n.mn[k] = 0xFFFFFFFFu;
    n.mx[k] = 0u;
    n.cmn[k] = ~0ull;
    n.cmx[k] = 0ull;
  }
}

__global__ void k_init(Work w) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool large = w.ntri > (uint32_t)kSmall;
  const uint32_t chunks = (w.ntri + kChunk - 1) / kChunk;
  if (i == 0) {
    Ctl c;
    memset(&c, 0, sizeof c);
    c.nodes = 1;
    c.mark[0] = 1;
    c.large[0] = large ? 1u : 0u;
    c.chunks[0] = large ? chunks : 0u;
    c.small = large ? 0u : 1u;
    *w.ctl = c;
    LNode n;
    init_node(n, 0u, w.ntri, 0u);
    n.chunks = chunks;
    w.nodes[0] = n;
    w.list[0][0] = 0u;
    w.small[0] = 0u;
  }
  if (!large) return;
  if (i < chunks) w.chunk_node[0][i] = 0u;
  if (i < (uint32_t)(21 * w.nbins)) w.bins[0][i] = bin_identity((int)((i / w.nbins) % 7));
}

// Triangle bounds from the f32 vertices, and the root's bounds.
__global__ void __launch_bounds__(256) k_prep(Work w, const float* __restrict__ pos, int ps, size_t nvert,
                                              const uint32_t* __restrict__ tri, int is) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t mn[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, mx[3] = {0u, 0u, 0u};
  u64 cmn[3] = {~0ull, ~0ull, ~0ull}, cmx[3] = {0ull, 0ull, 0ull};
  uint32_t bad = 0;
  if (t < w.ntri) {
    w.idx[0][t] = t;
    const uint32_t* iv = tri + (size_t)t * is;
    const uint32_t a = iv[0], b = iv[1], c = iv[2];
    if (a >= nvert || b >= nvert || c >= nvert) {
      bad = 1;  // out-of-range vertex: reported, nothing read
    } else {
      for (int k = 0; k < 3; ++k) {
        const float va = pos[(size_t)a * ps + k], vb = pos[(size_t)b * ps + k], vc = pos[(size_t)c * ps + k];
        if (!isfinite(va) || !isfinite(vb) || !isfinite(vc)) bad = 2;
        const uint32_t ka = fkey(va), kb = fkey(vb), kc = fkey(vc);
        mn[k] = min(min(ka, kb), kc);
        mx[k] = max(max(ka, kb), kc);
        cmn[k] = cmx[k] = okey(centroid(mn[k], mx[k]));
      }
      w.boxes[2 * (size_t)t] = make_uint4(mn[0], mn[1], mn[2], 0u);
      w.boxes[2 * (size_t)t + 1] = make_uint4(mx[0], mx[1], mx[2], 0u);
    }
  }
  if (bad) atomicOr(&w.ctl->bad, bad);
  __shared__ uint32_t sk[8][6];
  __shared__ u64 sc[8][6];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int k = 0; k < 3; ++k) {
    const uint32_t a = __reduce_min_sync(kFull, mn[k]), b = __reduce_max_sync(kFull, mx[k]);
    const u64 c = warp_min64(cmn[k]), d = warp_max64(cmx[k]);
    if (lane == 0) {
      sk[wid][k] = a;
      sk[wid][3 + k] = b;
      sc[wid][k] = c;
      sc[wid][3 + k] = d;
    }
  }
  __syncthreads();
  if (threadIdx.x < 12) {
    const int k = threadIdx.x % 6;
    LNode& r = w.nodes[0];
    if (threadIdx.x < 6) {
      uint32_t v = sk[0][k];
      for (int q = 1; q < 8; ++q) v = k < 3 ? min(v, sk[q][k]) : max(v, sk[q][k]);
      if (k < 3) atomicMin(&r.mn[k], v); else atomicMax(&r.mx[k - 3], v);
    } else {
      u64 v = sc[0][k];
      for (int q = 1; q < 8; ++q) v = k < 3 ? min(v, sc[q][k]) : max(v, sc[q][k]);
      if (k < 3) atomicMin(&r.cmn[k], v); else atomicMax(&r.cmx[k - 3], v);
    }
  }
}

// A level's kernel does nothing once the input is bad or an earlier level waits for the host.
__device__ __forceinline__ bool halted(const Ctl* c, uint32_t level) {
  return c->bad || c->depth_error || (c->stop && c->stop - 1u < level);
}

__global__ void __launch_bounds__(kChunkThreads) k_bin(Work w, uint32_t level) {
  extern __shared__ uint32_t sb[];  // [axis][7][bin]
  Ctl* ctl = w.ctl;
  if (halted(ctl, level)) return;
  const uint32_t p = level & 1u, c = blockIdx.x, nch = ctl->chunks[p];
  if (c == 0 && threadIdx.x == 0) {
    // the next level's counters (last read by the previous level), and this level's place in the numbering
    ctl->large[p ^ 1u] = 0u;
    ctl->chunks[p ^ 1u] = 0u;
    if (nch) {
      ctl->mark[level] = ctl->nodes;
      ctl->levels = level + 1u;
    }
  }
  if (c >= nch) return;
  const LNode& N = w.nodes[w.chunk_node[p][c]];
  const int nb = w.nbins;
  for (int i = threadIdx.x; i < 21 * nb; i += blockDim.x) sb[i] = bin_identity((i / nb) % 7);
  double cmin[3], span[3];
  for (int a = 0; a < 3; ++a) {
    cmin[a] = okey_value(N.cmn[a]);
    span[a] = __dsub_rn(okey_value(N.cmx[a]), cmin[a]);
  }
  __syncthreads();
  const uint32_t off = (c - N.chunk0) * kChunk, cnt = min((uint32_t)kChunk, N.count - off);
  const uint32_t* src = w.idx[p] + N.begin + off;
  for (uint32_t i = threadIdx.x; i < cnt; i += blockDim.x) {
    const uint32_t t = src[i];
    const uint4 l = w.boxes[2 * (size_t)t], h = w.boxes[2 * (size_t)t + 1];
    const uint32_t lo[3] = {l.x, l.y, l.z}, hi[3] = {h.x, h.y, h.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      if (!(span[a] > 1e-9)) continue;
      const int j = bin_of(centroid(lo[a], hi[a]), cmin[a], span[a], nb);
      uint32_t* b = sb + 7 * a * nb + j;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        atomicMin(b + k * nb, lo[k]);
        atomicMax(b + (3 + k) * nb, hi[k]);
      }
      atomicAdd(b + 6 * nb, 1u);
    }
  }
  __syncthreads();
  uint32_t* g = w.bins[p] + (size_t)N.slot * 21 * nb;
  uint32_t* hist = w.hist + (size_t)c * 3 * nb;
  for (int i = threadIdx.x; i < 3 * nb; i += blockDim.x) {
    const int a = i / nb, j = i % nb;
    const uint32_t* b = sb + 7 * a * nb + j;
    const uint32_t n = b[6 * nb];
    hist[i] = n;
    if (!n) continue;
    uint32_t* o = g + 7 * a * nb + j;
    for (int k = 0; k < 3; ++k) {
      atomicMin(o + k * nb, b[k * nb]);
      atomicMax(o + (3 + k) * nb, b[(3 + k) * nb]);
    }
    atomicAdd(o + 6 * nb, n);
  }
}

// Best split of one node over the axes so far; cost as the bits of a non-negative double.
struct Best {
  u64 cost = kNoCost;
  int axis = 0, split = 0;
  uint32_t nl = 0;
};

// Sweeps and costs of one axis by one warp.  B: the bins [7][nb]; suf: scratch
// of the same size; cb: the best split's child bounds (left, right; mn then mx
// keys).  Ties keep the earlier axis and the lower split, as the sequential
// scan with a strict comparison does.
__device__ void warp_axis(const uint32_t* B, uint32_t* suf, int nb, int axis, double parent_sa, Best& best,
                          uint32_t* cb) {
  const int lane = threadIdx.x & 31;
  uint32_t carry[7];
#pragma unroll
  for (int k = 0; k < 7; ++k) carry[k] = k < 6 ? bin_identity(k) : 0u;
  for (int g = (nb - 1) / 32; g >= 0; --g) {
    const int b = 32 * g + lane;
    uint32_t v[7];
#pragma unroll
    for (int k = 0; k < 7; ++k) v[k] = b < nb ? B[k * nb + b] : (k < 6 ? bin_identity(k) : 0u);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
      for (int k = 0; k < 7; ++k) {
        const uint32_t t = __shfl_down_sync(kFull, v[k], o);
        if (lane + o < 32) v[k] = k < 3 ? min(v[k], t) : (k < 6 ? max(v[k], t) : v[k] + t);
      }
    }
#pragma unroll
    for (int k = 0; k < 7; ++k) {
      v[k] = k < 3 ? min(v[k], carry[k]) : (k < 6 ? max(v[k], carry[k]) : v[k] + carry[k]);
      carry[k] = __shfl_sync(kFull, v[k], 0);
      if (b < nb) suf[k * nb + b] = v[k];
    }
  }
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 7; ++k) carry[k] = k < 6 ? bin_identity(k) : 0u;
  u64 cost = kNoCost;
  int split = nb;
  uint32_t nl = 0, l[6] = {0, 0, 0, 0, 0, 0};
  for (int g = 0; g <= (nb - 1) / 32; ++g) {
    const int b = 32 * g + lane;
    uint32_t v[7];
#pragma unroll
    for (int k = 0; k < 7; ++k) v[k] = b < nb ? B[k * nb + b] : (k < 6 ? bin_identity(k) : 0u);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
      for (int k = 0; k < 7; ++k) {
        const uint32_t t = __shfl_up_sync(kFull, v[k], o);
        if (lane >= o) v[k] = k < 3 ? min(v[k], t) : (k < 6 ? max(v[k], t) : v[k] + t);
      }
    }
#pragma unroll
    for (int k = 0; k < 7; ++k) {
      v[k] = k < 3 ? min(v[k], carry[k]) : (k < 6 ? max(v[k], carry[k]) : v[k] + carry[k]);
      carry[k] = __shfl_sync(kFull, v[k], 31);
    }
    if (b < nb - 1) {
      const uint32_t* r = suf + b + 1;
      const uint32_t lc = v[6], rc = r[6 * nb];
      if (lc && rc) {
        const double lsa = half_sa(v[0], v[1], v[2], v[3], v[4], v[5]);
        const double rsa = half_sa(r[0], r[nb], r[2 * nb], r[3 * nb], r[4 * nb], r[5 * nb]);
        const double c = split_cost(lsa, lc, rsa, rc, parent_sa);
        const u64 cbits = (u64)__double_as_longlong(c);
        if (c < INFINITY && cbits < cost) {
          cost = cbits;
          split = b;
          nl = lc;
#pragma unroll
          for (int k = 0; k < 6; ++k) l[k] = v[k];
        }
      }
    }
  }
  const u64 m = warp_min64(cost);
  if (m == kNoCost || !(m < best.cost)) {
    __syncwarp();
    return;
  }
  const uint32_t s = __reduce_min_sync(kFull, cost == m ? (uint32_t)split : 0xFFFFFFFFu);
  const bool own = cost == m && (uint32_t)split == s;
  const int owner = __ffs(__ballot_sync(kFull, own)) - 1;
  best.cost = m;
  best.axis = axis;
  best.split = (int)s;
  best.nl = __shfl_sync(kFull, nl, owner);
  if (own)
    for (int k = 0; k < 6; ++k) {
      cb[k] = l[k];
      cb[6 + k] = suf[k * nb + s + 1];
    }
  __syncwarp();
}

__device__ __forceinline__ bool beats_leaf(u64 cost, uint32_t count) {
  return cost != kNoCost && __longlong_as_double((long long)cost) < (double)count;
}
// widest centroid axis, the first on ties
__device__ __forceinline__ int widest_axis(const double span[3]) {
  int ax = 0;
  double m = span[0];
  for (int k = 1; k < 3; ++k)
    if (span[k] > m) { ax = k; m = span[k]; }
  return ax;
}

__global__ void __launch_bounds__(128) k_choose(Work w, uint32_t level) {
  extern __shared__ uint32_t sm[];  // bins [axis][7][bin], then the suffix scratch
  __shared__ Best res[3];
  __shared__ uint32_t cb[3][12];
  __shared__ int s_axis, s_split, s_decision, s_left;
  __shared__ uint32_t s_nl, wsum[4], s_carry;
  Ctl* ctl = w.ctl;
  if (__syncthreads_or(halted(ctl, level))) return;  // (another CTA may set the depth error meanwhile)
  const uint32_t p = level & 1u;
  if (blockIdx.x >= ctl->large[p]) return;
  LNode& N = w.nodes[w.list[p][blockIdx.x]];
  const int nb = w.nbins, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t count = N.count;
  const uint32_t* g = w.bins[p] + (size_t)N.slot * 21 * nb;
  for (int i = threadIdx.x; i < 21 * nb; i += blockDim.x) sm[i] = g[i];
  double span[3];
  for (int a = 0; a < 3; ++a) span[a] = __dsub_rn(okey_value(N.cmx[a]), okey_value(N.cmn[a]));
  const double parent_sa = half_sa(N.mn[0], N.mn[1], N.mn[2], N.mx[0], N.mx[1], N.mx[2]);
  __syncthreads();
  if (wid < 3) {
    Best b;
    if (span[wid] > 1e-9) warp_axis(sm + 7 * wid * nb, sm + (21 + 7 * wid) * nb, nb, wid, parent_sa, b, cb[wid]);
    if (lane == 0) res[wid] = b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    Best b;
    for (int a = 0; a < 3; ++a)
      if (res[a].cost < b.cost) b = res[a];
    s_left = -1;
    s_decision = beats_leaf(b.cost, count) ? 1 : 3;
    s_axis = s_decision == 1 ? b.axis : widest_axis(span);
    s_split = b.split;
    s_nl = s_decision == 1 ? b.nl : count / 2;
    if ((int)N.depth >= w.max_depth) {
      ctl->depth_error = 1u;
    } else {
      const uint32_t l = atomicAdd(&ctl->nodes, 2u);
      if (l + 2u > w.node_cap) {
        atomicOr(&ctl->bad, 4u);
      } else {
        N.axis = s_axis;
        N.split = s_split;
        N.nl = s_nl;
        N.decision = s_decision;
        N.left = (int)l;
        s_left = (int)l;
        for (int i = 0; i < 2; ++i) {
          LNode ch;
          init_node(ch, i ? N.begin + s_nl : N.begin, i ? count - s_nl : s_nl, N.depth + 1u);
          if (s_decision == 1)
            for (int k = 0; k < 3; ++k) {
              ch.mn[k] = cb[s_axis][6 * i + k];
              ch.mx[k] = cb[s_axis][6 * i + 3 + k];
            }
          if (ch.count > (uint32_t)kSmall) {
            ch.slot = atomicAdd(&ctl->large[p ^ 1u], 1u);
            ch.chunks = (ch.count + kChunk - 1) / kChunk;
            ch.chunk0 = atomicAdd(&ctl->chunks[p ^ 1u], ch.chunks);
            w.list[p ^ 1u][ch.slot] = l + (uint32_t)i;
          } else {
            w.small[atomicAdd(&ctl->small, 1u)] = l + (uint32_t)i;
          }
          w.nodes[l + i] = ch;
        }
        if (s_decision == 3) {
          ctl->stop = level + 1u;
          if (count > kSort) ctl->big = 1u;
        }
      }
    }
    s_carry = 0u;
  }
  __syncthreads();
  if (s_left < 0) return;
  for (int i = 0; i < 2; ++i) {
    const LNode& ch = w.nodes[s_left + i];
    if (ch.count <= (uint32_t)kSmall) continue;
    for (uint32_t q = threadIdx.x; q < ch.chunks; q += blockDim.x) w.chunk_node[p ^ 1u][ch.chunk0 + q] = (uint32_t)(s_left + i);
    uint32_t* b = w.bins[p ^ 1u] + (size_t)ch.slot * 21 * nb;
    for (int q = threadIdx.x; q < 21 * nb; q += blockDim.x) b[q] = bin_identity((q / nb) % 7);
  }
  if (s_decision != 1) return;
  // triangles left of the split before each chunk: an exclusive scan over the node's chunks
  for (uint32_t base = 0; base < N.chunks; base += blockDim.x) {
    const uint32_t q = base + threadIdx.x;
    uint32_t left = 0;
    if (q < N.chunks) {
      const uint32_t* h = w.hist + ((size_t)(N.chunk0 + q) * 3 + s_axis) * nb;
      for (int j = 0; j <= s_split; ++j) left += h[j];
    }
    uint32_t inc = left;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(kFull, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) wsum[wid] = inc;
    __syncthreads();
    uint32_t before = s_carry;
    for (int q2 = 0; q2 < wid; ++q2) before += wsum[q2];
    if (q < N.chunks) w.chunk_left[N.chunk0 + q] = before + inc - left;
    __syncthreads();
    if (threadIdx.x == 0) s_carry += wsum[0] + wsum[1] + wsum[2] + wsum[3];
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kChunkThreads) k_scatter(Work w, uint32_t level) {
  __shared__ u64 red[kChunkThreads / 32][2][6];
  __shared__ uint32_t wcnt[kChunkThreads / 32];
  const Ctl* ctl = w.ctl;
  if (halted(ctl, level) || ctl->stop) return;
  const uint32_t p = level & 1u, c = blockIdx.x;
  if (c >= ctl->chunks[p]) return;
  const LNode& N = w.nodes[w.chunk_node[p][c]];
  if (N.decision != 1) return;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, ax = N.axis;
  const double cmin = okey_value(N.cmn[ax]), span = __dsub_rn(okey_value(N.cmx[ax]), cmin);
  const uint32_t off = (c - N.chunk0) * kChunk, cnt = min((uint32_t)kChunk, N.count - off);
  const uint32_t* src = w.idx[p] + N.begin + off;
  uint32_t* dst = w.idx[p ^ 1u] + N.begin;
  uint32_t lefts = w.chunk_left[c];  // left triangles before this round
  u64 acc[2][6];
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int k = 0; k < 6; ++k) acc[s][k] = k < 3 ? ~0ull : 0ull;
  for (uint32_t base = 0; base < cnt; base += kChunkThreads) {
    const uint32_t i = base + threadIdx.x;
    const bool valid = i < cnt;
    uint32_t t = 0;
    bool left = false;
    u64 key[3] = {0, 0, 0};
    if (valid) {
      t = src[i];
      const uint4 l = w.boxes[2 * (size_t)t], h = w.boxes[2 * (size_t)t + 1];
      const double cen[3] = {centroid(l.x, h.x), centroid(l.y, h.y), centroid(l.z, h.z)};
#pragma unroll
      for (int k = 0; k < 3; ++k) key[k] = okey(cen[k]);
      left = bin_of(ax == 0 ? cen[0] : (ax == 1 ? cen[1] : cen[2]), cmin, span, w.nbins) <= N.split;
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (left != (s == 0)) continue;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          acc[s][k] = min(acc[s][k], key[k]);
          acc[s][3 + k] = max(acc[s][3 + k], key[k]);
        }
      }
    }
    const uint32_t m = __ballot_sync(kFull, left);
    if (lane == 0) wcnt[wid] = (uint32_t)__popc(m);
    __syncthreads();
    uint32_t before = lefts;
    uint32_t round = 0;
    for (int q = 0; q < kChunkThreads / 32; ++q) {
      if (q < wid) before += wcnt[q];
      round += wcnt[q];
    }
    before += (uint32_t)__popc(m & ((1u << lane) - 1u));
    if (valid) dst[left ? before : N.nl + (off + i - before)] = t;
    lefts += round;
    __syncthreads();
  }
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const u64 v = k < 3 ? warp_min64(acc[s][k]) : warp_max64(acc[s][k]);
      if (lane == 0) red[wid][s][k] = v;
    }
  __syncthreads();
  if (threadIdx.x < 12) {
    const int s = threadIdx.x / 6, k = threadIdx.x % 6;
    u64 v = red[0][s][k];
    for (int q = 1; q < kChunkThreads / 32; ++q) v = k < 3 ? min(v, red[q][s][k]) : max(v, red[q][s][k]);
    LNode& ch = w.nodes[N.left + s];
    if (k < 3) atomicMin(&ch.cmn[k], v); else atomicMax(&ch.cmx[k - 3], v);
  }
}

// Bounds of a node whose range was sorted (ids: its index range), the part of the
// threads first, first + step, ...; by whole warps.
__device__ __forceinline__ void range_bounds(const Work& w, LNode& N, const uint32_t* ids, uint32_t first,
                                             uint32_t step) {
  uint32_t mn[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, mx[3] = {0u, 0u, 0u};
  u64 cmn[3] = {~0ull, ~0ull, ~0ull}, cmx[3] = {0ull, 0ull, 0ull};
  for (uint32_t i = first; i < N.count; i += step) {
    const uint4 l = w.boxes[2 * (size_t)ids[i]], h = w.boxes[2 * (size_t)ids[i] + 1];
    const uint32_t lo[3] = {l.x, l.y, l.z}, hi[3] = {h.x, h.y, h.z};
    for (int k = 0; k < 3; ++k) {
      const u64 c = okey(centroid(lo[k], hi[k]));
      mn[k] = min(mn[k], lo[k]);
      mx[k] = max(mx[k], hi[k]);
      cmn[k] = min(cmn[k], c);
      cmx[k] = max(cmx[k], c);
    }
  }
  for (int k = 0; k < 3; ++k) {
    const uint32_t a = __reduce_min_sync(kFull, mn[k]), b = __reduce_max_sync(kFull, mx[k]);
    const u64 c = warp_min64(cmn[k]), d = warp_max64(cmx[k]);
    if ((threadIdx.x & 31) == 0) {
      atomicMin(&N.mn[k], a);
      atomicMax(&N.mx[k], b);
      atomicMin(&N.cmn[k], c);
      atomicMax(&N.cmx[k], d);
    }
  }
}
__global__ void __launch_bounds__(256) k_range_bounds(Work w, uint32_t node, const uint32_t* __restrict__ ids) {
  range_bounds(w, w.nodes[node], ids, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// Key of the fallback sort: -0 canonicalised to +0 (the reference's comparator
// subtracts, so equal centroids tie and fall to the index), then mapped to an
// order-preserving integer.
__device__ __forceinline__ u64 sort_key(const uint4* boxes, uint32_t t, int axis) {
  const uint4 l = boxes[2 * (size_t)t], h = boxes[2 * (size_t)t + 1];
  double v = axis == 0 ? centroid(l.x, h.x) : (axis == 1 ? centroid(l.y, h.y) : centroid(l.z, h.z));
  if (v == 0.0) v = 0.0;
  return okey(v);
}
__global__ void k_sort_keys(const uint4* __restrict__ boxes, const uint32_t* __restrict__ ids, uint32_t c, int axis,
                            u64* __restrict__ keys) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < c) keys[i] = sort_key(boxes, ids[i], axis);
}

// A stopped level's nodes without a split of up to kSort triangles, one CTA each: a
// bitonic sort of (key, triangle) pairs (all different) in shared memory, padded to
// a power of two with pairs above every real one, then the children's bounds.
__global__ void __launch_bounds__(kSortThreads) k_sort(Work w, uint32_t level) {
  extern __shared__ __align__(16) unsigned char dyn[];
  u64* key = reinterpret_cast<u64*>(dyn);
  uint32_t* id = reinterpret_cast<uint32_t*>(dyn + 8 * (size_t)kSort);
  const uint32_t p = level & 1u;
  const LNode& N = w.nodes[w.list[p][blockIdx.x]];
  const uint32_t count = N.count;
  if (N.decision != 3 || count > kSort) return;
  const uint32_t* src = w.idx[p] + N.begin;
  uint32_t* dst = w.idx[p ^ 1u] + N.begin;
  uint32_t m = 2;
  while (m < count) m <<= 1;
  for (uint32_t i = threadIdx.x; i < m; i += kSortThreads) {
    id[i] = i < count ? src[i] : 0xFFFFFFFFu;
    key[i] = i < count ? sort_key(w.boxes, id[i], N.axis) : ~0ull;
  }
  for (uint32_t k = 2; k <= m; k <<= 1)
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      __syncthreads();
      for (uint32_t q = threadIdx.x; q < m / 2; q += kSortThreads) {
        const uint32_t a = 2 * q - (q & (j - 1u)), b = a + j;
        const u64 ka = key[a], kb = key[b];
        const uint32_t ia = id[a], ib = id[b];
        const bool above = ka > kb || (ka == kb && ia > ib);
        if (above == ((a & k) == 0u)) {
          key[a] = kb;
          key[b] = ka;
          id[a] = ib;
          id[b] = ia;
        }
      }
    }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < count; i += kSortThreads) dst[i] = id[i];
  for (int i = 0; i < 2; ++i)
    range_bounds(w, w.nodes[N.left + i], id + (i ? N.nl : 0u), threadIdx.x, kSortThreads);
}

// ---------------------------------------------------------------- small subtrees
// Shared memory of one subtree; the warps' bins (and suffix scratch) follow it.
struct Small {
  uint32_t box[6][kSmall];            // bounds (fkey) by slot
  uint32_t src[kSmall];               // triangle of each slot
  uint32_t nbox[6][2 * kSmall];       // node bounds
  uint32_t cb[kSmallThreads / 32][12];
  uint32_t nodes, listed[2], error;
  uint16_t idx[kSmall], tmp[kSmall];  // slots in tree order
  uint16_t nbeg[2 * kSmall], ncnt[2 * kSmall], nleft[2 * kSmall], nsize[2 * kSmall], npre[2 * kSmall];
  uint16_t list[2][kSmall];           // nodes to split, by level parity
  uint16_t mark[kMaxBinaryDepth + 3]; // nodes of depth <= level
  uint8_t naxis[2 * kSmall];
};

struct SplitResult {
  int axis;
  uint32_t nl;
  bool bounds;  // cb holds the children's bounds
};

// A node of 2..8 triangles: lane 8 a + i looks at triangle i on axis a.  Only
// the bins that hold a triangle can be the first of equal splits, so lane
// (a, i) evaluates the split after triangle i's bin against all the others.
__device__ SplitResult split_tiny(Small& S, uint32_t* cb, uint32_t b, uint32_t c, double parent_sa, int nb) {
  const int lane = threadIdx.x & 31, a = lane >> 3;
  const uint32_t i = lane & 7u;
  const bool on = a < 3 && i < c;
  const uint32_t t = S.idx[b + (i < c ? i : 0)];
  const double cen = a < 3 ? centroid(S.box[a][t], S.box[3 + a][t]) : 0.0;
  double lo = cen, hi = cen;  // padding lanes repeat triangle 0
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    lo = fmin(lo, __shfl_xor_sync(kFull, lo, o));
    hi = fmax(hi, __shfl_xor_sync(kFull, hi, o));
  }
  const double span = __dsub_rn(hi, lo);
  const bool use = on && span > 1e-9;
  const int bin = use ? bin_of(cen, lo, span, nb) : 0;
  uint32_t l[6], r[6], nl = 0;
#pragma unroll
  for (int k = 0; k < 6; ++k) l[k] = r[k] = bin_identity(k);
  for (uint32_t j = 0; j < c; ++j) {
    const int bj = __shfl_sync(kFull, bin, (lane & 24) | (int)j);
    const uint32_t tj = S.idx[b + j];
    const bool left = bj <= bin;
    nl += left ? 1u : 0u;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const uint32_t v = S.box[k][tj];
      if (k < 3) {
        l[k] = min(l[k], left ? v : 0xFFFFFFFFu);
        r[k] = min(r[k], left ? 0xFFFFFFFFu : v);
      } else {
        l[k] = max(l[k], left ? v : 0u);
        r[k] = max(r[k], left ? 0u : v);
      }
    }
  }
  u64 cost = kNoCost;
  if (use && nl < c) {
    const double v = split_cost(half_sa(l[0], l[1], l[2], l[3], l[4], l[5]), nl,
                                half_sa(r[0], r[1], r[2], r[3], r[4], r[5]), c - nl, parent_sa);
    if (v < INFINITY) cost = (u64)__double_as_longlong(v);
  }
  const u64 m = warp_min64(cost);
  SplitResult out;
  if (beats_leaf(m, c)) {
    const uint32_t id = (uint32_t)(a << 8) | (uint32_t)bin;
    const uint32_t w = __reduce_min_sync(kFull, cost == m ? id : 0xFFFFFFFFu);
    const uint32_t own = __ballot_sync(kFull, cost == m && id == w);
    const int owner = __ffs(own) - 1;
    if (lane == owner)
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        cb[k] = l[k];
        cb[6 + k] = r[k];
      }
    out.axis = (int)(w >> 8);
    out.nl = __shfl_sync(kFull, nl, owner);
    out.bounds = true;
    const uint32_t split = w & 255u;
    const uint32_t ml = __ballot_sync(kFull, on && (uint32_t)bin <= split) >> (8 * out.axis) & 255u;
    if (a == out.axis && on) {
      const uint32_t before = (uint32_t)__popc(ml & ((1u << i) - 1u));
      S.idx[b + ((ml >> i) & 1u ? before : out.nl + (i - before))] = (uint16_t)t;
    }
    __syncwarp();
    return out;
  }
  // no split beats a leaf: order by (centroid on the widest axis, triangle), split in half
  double sp[3];
  for (int k = 0; k < 3; ++k) sp[k] = __shfl_sync(kFull, span, 8 * k);
  out.axis = widest_axis(sp);
  out.nl = c / 2;
  out.bounds = false;
  const uint32_t id = S.src[t];
  uint32_t rank = 0;
  for (uint32_t j = 0; j < c; ++j) {
    const double cj = __shfl_sync(kFull, cen, (lane & 24) | (int)j);
    const uint32_t ij = __shfl_sync(kFull, id, (lane & 24) | (int)j);
    if (cj < cen || (cj == cen && ij < id)) ++rank;
  }
  __syncwarp();
  if (a == out.axis && on) S.idx[b + rank] = (uint16_t)t;
  __syncwarp();
  return out;
}

// A larger node of a subtree, by one warp through its bins in shared memory.
__device__ SplitResult split_warp(Small& S, uint32_t* cb, uint32_t* bins, uint32_t b, uint32_t c, double parent_sa,
                                  int nb) {
  const int lane = threadIdx.x & 31;
  u64 cmn[3] = {~0ull, ~0ull, ~0ull}, cmx[3] = {0ull, 0ull, 0ull};
  for (uint32_t i = lane; i < c; i += 32) {
    const uint32_t t = S.idx[b + i];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const u64 v = okey(centroid(S.box[k][t], S.box[3 + k][t]));
      cmn[k] = min(cmn[k], v);
      cmx[k] = max(cmx[k], v);
    }
  }
  double cmin[3], span[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    cmin[k] = okey_value(warp_min64(cmn[k]));
    span[k] = __dsub_rn(okey_value(warp_max64(cmx[k])), cmin[k]);
  }
  Best best;
  for (int a = 0; a < 3; ++a) {
    if (!(span[a] > 1e-9)) continue;
    for (int i = lane; i < 7 * nb; i += 32) bins[i] = i < 3 * nb ? 0xFFFFFFFFu : 0u;
    __syncwarp();
    for (uint32_t i = lane; i < c; i += 32) {
      const uint32_t t = S.idx[b + i];
      uint32_t* o = bins + bin_of(centroid(S.box[a][t], S.box[3 + a][t]), cmin[a], span[a], nb);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        atomicMin(o + k * nb, S.box[k][t]);
        atomicMax(o + (3 + k) * nb, S.box[3 + k][t]);
      }
      atomicAdd(o + 6 * nb, 1u);
    }
    __syncwarp();
    warp_axis(bins, bins + 7 * nb, nb, a, parent_sa, best, cb);
  }
  SplitResult out;
  out.bounds = beats_leaf(best.cost, c);
  if (out.bounds) {
    out.axis = best.axis;
    out.nl = best.nl;
    uint32_t left = 0;
    const double c0 = best.axis == 0 ? cmin[0] : (best.axis == 1 ? cmin[1] : cmin[2]);
    const double sp = best.axis == 0 ? span[0] : (best.axis == 1 ? span[1] : span[2]);
    for (uint32_t base = 0; base < c; base += 32) {
      const uint32_t i = base + lane;
      uint32_t t = 0;
      bool go = false;
      if (i < c) {
        t = S.idx[b + i];
        go = bin_of(centroid(S.box[best.axis][t], S.box[3 + best.axis][t]), c0, sp, nb) <= best.split;
      }
      const uint32_t m = __ballot_sync(kFull, go);
      const uint32_t before = left + (uint32_t)__popc(m & ((1u << lane) - 1u));
      if (i < c) S.tmp[b + (go ? before : out.nl + (i - before))] = (uint16_t)t;
      left += (uint32_t)__popc(m);
    }
  } else {
    out.axis = widest_axis(span);
    out.nl = c / 2;
    for (uint32_t i = lane; i < c; i += 32) {
      const uint32_t t = S.idx[b + i], id = S.src[t];
      const double v = centroid(S.box[out.axis][t], S.box[3 + out.axis][t]);
      uint32_t rank = 0;
      for (uint32_t j = 0; j < c; ++j) {
        const uint32_t tj = S.idx[b + j];
        const double vj = centroid(S.box[out.axis][tj], S.box[3 + out.axis][tj]);
        if (vj < v || (vj == v && S.src[tj] < id)) ++rank;
      }
      S.tmp[b + rank] = (uint16_t)t;
    }
  }
  __syncwarp();
  for (uint32_t i = lane; i < c; i += 32) S.idx[b + i] = S.tmp[b + i];
  __syncwarp();
  return out;
}

__global__ void __launch_bounds__(kSmallThreads) k_small(Work w, uint32_t* __restrict__ order) {
  extern __shared__ __align__(16) unsigned char dyn[];
  Small& S = *reinterpret_cast<Small*>(dyn);
  Ctl* ctl = w.ctl;
  if (__syncthreads_or(ctl->bad || ctl->depth_error)) return;  // (another CTA may set the depth error meanwhile)
  LNode& N = w.nodes[w.small[blockIdx.x]];
  const int nb = w.nbins, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t* bins = reinterpret_cast<uint32_t*>(dyn + sizeof(Small)) + (size_t)wid * 14 * nb;
  const uint32_t count = N.count, depth0 = N.depth, begin = N.begin;
  const uint32_t* src = w.idx[depth0 & 1u] + begin;
  for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) {
    const uint32_t t = src[i];
    const uint4 l = w.boxes[2 * (size_t)t], h = w.boxes[2 * (size_t)t + 1];
    S.src[i] = t;
    S.idx[i] = (uint16_t)i;
    S.box[0][i] = l.x; S.box[1][i] = l.y; S.box[2][i] = l.z;
    S.box[3][i] = h.x; S.box[4][i] = h.y; S.box[5][i] = h.z;
  }
  if (threadIdx.x < 6) S.nbox[threadIdx.x][0] = threadIdx.x < 3 ? N.mn[threadIdx.x] : N.mx[threadIdx.x - 3];
  if (threadIdx.x == 0) {
    S.nodes = 1;
    S.error = 0;
    S.nbeg[0] = 0;
    S.ncnt[0] = (uint16_t)count;
    S.nleft[0] = 0;
    S.naxis[0] = 0;
    S.listed[0] = count > (uint32_t)w.max_leaf ? 1u : 0u;
    S.listed[1] = 0;
    S.list[0][0] = 0;
    S.mark[0] = 1;
  }
  __syncthreads();
  uint32_t level = 0;
  while (true) {
    const uint32_t cur = level & 1u, n = S.listed[cur];
    if (n == 0) break;
    if ((int)(depth0 + level) >= w.max_depth) {  // the cap leaves a node above max_leaf: an error
      if (threadIdx.x == 0) ctl->depth_error = 1u;
      return;
    }
    for (uint32_t q = wid; q < n; q += kSmallThreads / 32) {
      const uint32_t id = S.list[cur][q], b = S.nbeg[id], c = S.ncnt[id];
      const double parent_sa = half_sa(S.nbox[0][id], S.nbox[1][id], S.nbox[2][id], S.nbox[3][id], S.nbox[4][id],
                                       S.nbox[5][id]);
      const SplitResult r = c <= 8 ? split_tiny(S, S.cb[wid], b, c, parent_sa, nb)
                                   : split_warp(S, S.cb[wid], bins, b, c, parent_sa, nb);
      uint32_t ch = 0;
      if (lane == 0) ch = atomicAdd(&S.nodes, 2u);
      ch = __shfl_sync(kFull, ch, 0);
      if (lane < 12) {
        const uint32_t side = lane / 6, k = lane % 6;
        uint32_t v = S.cb[wid][lane];
        if (!r.bounds) {
          const uint32_t e = side ? c : r.nl;
          v = bin_identity((int)k);
          for (uint32_t j = side ? r.nl : 0u; j < e; ++j) {
            const uint32_t x = S.box[k][S.idx[b + j]];
            v = k < 3 ? min(v, x) : max(v, x);
          }
        }
        S.nbox[k][ch + side] = v;
      }
      if (lane < 2) {
        const uint32_t x = ch + lane, cn = lane ? c - r.nl : r.nl;
        S.nbeg[x] = (uint16_t)(lane ? b + r.nl : b);
        S.ncnt[x] = (uint16_t)cn;
        S.nleft[x] = 0;
        S.naxis[x] = 0;
        if (cn > (uint32_t)w.max_leaf) S.list[cur ^ 1u][atomicAdd(&S.listed[cur ^ 1u], 1u)] = (uint16_t)x;
      }
      if (lane == 0) {
        S.nleft[id] = (uint16_t)ch;
        S.naxis[id] = (uint8_t)r.axis;
      }
      __syncwarp();
    }
    __syncthreads();
    ++level;
    if (threadIdx.x == 0) {
      S.listed[cur] = 0;
      S.mark[level] = (uint16_t)S.nodes;
    }
    __syncthreads();
  }
  // subtree sizes bottom up, preorder numbers top down (children follow their parents' level)
  for (int L = (int)level; L >= 0; --L) {
    for (uint32_t x = (L ? S.mark[L - 1] : 0u) + threadIdx.x; x < S.mark[L]; x += blockDim.x) {
      const uint32_t l = S.nleft[x];
      S.nsize[x] = (uint16_t)(l ? 1u + S.nsize[l] + S.nsize[l + 1] : 1u);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) S.npre[0] = 0;
  __syncthreads();
  for (uint32_t L = 0; L < level; ++L) {
    for (uint32_t x = (L ? S.mark[L - 1] : 0u) + threadIdx.x; x < S.mark[L]; x += blockDim.x) {
      const uint32_t l = S.nleft[x];
      if (!l) continue;
      S.npre[l] = (uint16_t)(S.npre[x] + 1u);
      S.npre[l + 1] = (uint16_t)(S.npre[x] + 1u + S.nsize[l]);
    }
    __syncthreads();
  }
  const uint32_t total = S.nodes;
  BinaryNode* out = w.temp + 2 * (size_t)begin;
  for (uint32_t x = threadIdx.x; x < total; x += blockDim.x) {
    BinaryNode o;
    for (int k = 0; k < 3; ++k) {
      o.mn[k] = funkey(S.nbox[k][x]);
      o.mx[k] = funkey(S.nbox[3 + k][x]);
    }
    const uint32_t l = S.nleft[x];
    if (l) {
      o.w6 = (uint32_t)S.npre[l + 1] - S.npre[x];
      o.w7 = S.naxis[x];
    } else {
      o.w6 = begin + S.nbeg[x];
      o.w7 = kLeafFlag | S.ncnt[x];
    }
    out[S.npre[x]] = o;
  }
  for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) order[begin + i] = S.src[S.idx[i]];
  if (threadIdx.x == 0) {
    N.size = total;
    atomicMax(&ctl->max_depth, depth0 + level);
  }
}

// ---------------------------------------------------------------- numbering and output
__global__ void __launch_bounds__(1024) k_top(Work w) {
  Ctl* ctl = w.ctl;
  if (ctl->bad || ctl->depth_error) return;
  const int levels = (int)ctl->levels;  // nodes of depth L: mark[L - 1] .. mark[L]; children of the last level follow
  for (int L = levels - 1; L >= 0; --L) {
    for (uint32_t x = (L ? ctl->mark[L - 1] : 0u) + threadIdx.x; x < ctl->mark[L]; x += blockDim.x) {
      const int l = w.nodes[x].left;
      if (l >= 0) w.nodes[x].size = 1u + w.nodes[l].size + w.nodes[l + 1].size;
    }
    __syncthreads();
  }
  for (int L = 0; L < levels; ++L) {
    for (uint32_t x = (L ? ctl->mark[L - 1] : 0u) + threadIdx.x; x < ctl->mark[L]; x += blockDim.x) {
      const int l = w.nodes[x].left;
      if (l < 0) continue;
      w.nodes[l].pre = w.nodes[x].pre + 1u;
      w.nodes[l + 1].pre = w.nodes[x].pre + 1u + w.nodes[l].size;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) ctl->total = w.nodes[0].size;
}

__global__ void __launch_bounds__(128) k_emit(Work w, BinaryNode* __restrict__ out) {
  const Ctl* ctl = w.ctl;
  if (ctl->bad || ctl->depth_error || blockIdx.x >= ctl->nodes) return;
  const LNode& N = w.nodes[blockIdx.x];
  if (N.left < 0) {
    // a subtree: its nodes' links are relative, so its block moves as it is
    const uint4* s = reinterpret_cast<const uint4*>(w.temp + 2 * (size_t)N.begin);
    uint4* d = reinterpret_cast<uint4*>(out + N.pre);
    for (uint32_t i = threadIdx.x; i < 2 * N.size; i += blockDim.x) d[i] = s[i];
    return;
  }
  if (threadIdx.x) return;
  BinaryNode o;
  for (int k = 0; k < 3; ++k) {
    o.mn[k] = funkey(N.mn[k]);
    o.mx[k] = funkey(N.mx[k]);
  }
  o.w6 = w.nodes[N.left + 1].pre - N.pre;
  o.w7 = (uint32_t)N.axis;
  out[N.pre] = o;
}

// Sorts src[0, c) by (centroid on axis, index) into dst with two stable device radix passes.
void sort_range(const uint4* boxes, const uint32_t* src, uint32_t* dst, uint32_t c, int axis, cudaStream_t s) {
  ScratchBuffer<uint32_t> a2(c, s);
  ScratchBuffer<u64> k1(c, s), k2(c, s);
  size_t t1 = 0, t2 = 0;
  VT_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, t1, src, a2.ptr, (int)c, 0, 32, s));
  VT_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, t2, k1.ptr, k2.ptr, a2.ptr, dst, (int)c, 0, 64, s));
  ScratchBuffer<unsigned char> tmp(std::max(t1, t2), s);
  size_t tb = tmp.count;
  VT_CUDA(cub::DeviceRadixSort::SortKeys(tmp.ptr, tb, src, a2.ptr, (int)c, 0, 32, s));  // by index
  k_sort_keys<<<(c + 255) / 256, 256, 0, s>>>(boxes, a2.ptr, c, axis, k1.ptr);
  VT_CUDA(cudaGetLastError());
  tb = tmp.count;
  VT_CUDA(cub::DeviceRadixSort::SortPairs(tmp.ptr, tb, k1.ptr, k2.ptr, a2.ptr, dst, (int)c, 0, 64, s));  // stable
  VT_CUDA(cudaStreamSynchronize(s));
}

}  // namespace

BinaryBvhHost build_binary_gpu(const float* d_pos, size_t position_words, const uint32_t* d_idx, size_t index_words,
                               const BuildOptions& o, cudaStream_t s, BinaryBvhDevice* keep, bool host_copy) {
  validate_options(o);
  if (position_words % o.position_stride) fail(VT_ERR_RANGE, "positions.length must be divisible by positionStride");
  if (index_words % o.index_stride) fail(VT_ERR_RANGE, "indices.length must be divisible by indexStride");
  const size_t ntri = index_words / o.index_stride;
  BinaryBvhHost out;
  if (ntri == 0) {
    BinaryNode n{};
    n.w7 = kLeafFlag;
    out.nodes.push_back(n);
    return out;
  }
  if (ntri >= (1u << 30)) fail(VT_ERR_RANGE, "too many triangles for one tree");
  // ---- scratch
  Work w{};
  w.ntri = (uint32_t)ntri;
  w.nbins = o.bins;
  w.max_leaf = o.max_leaf;
  w.max_depth = o.max_depth;
  w.max_large = (uint32_t)(ntri / (kSmall + 1) + 1);  // disjoint ranges of more than kSmall triangles
  w.max_chunks = (uint32_t)(ntri / kChunk + w.max_large + 1);
  w.node_cap = (uint32_t)std::min<size_t>(2 * ntri, 1 + 2 * (size_t)w.max_large * (size_t)(o.max_depth + 1));
  size_t bytes = 0;
  auto place = [&](size_t n) {
    const size_t at = bytes;
    bytes += (n + 255) & ~(size_t)255;
    return at;
  };
  const size_t bin_words = (size_t)w.max_large * 21 * o.bins;
  const size_t at_ctl = place(sizeof(Ctl)), at_nodes = place(w.node_cap * sizeof(LNode)),
               at_boxes = place(2 * ntri * sizeof(uint4)), at_idx0 = place(ntri * 4), at_idx1 = place(ntri * 4),
               at_list0 = place(w.max_large * 4), at_list1 = place(w.max_large * 4),
               at_cn0 = place(w.max_chunks * 4), at_cn1 = place(w.max_chunks * 4), at_cl = place(w.max_chunks * 4),
               at_hist = place((size_t)w.max_chunks * 3 * o.bins * 4), at_b0 = place(bin_words * 4),
               at_b1 = place(bin_words * 4), at_small = place(w.node_cap * 4), at_temp = place(2 * ntri * sizeof(BinaryNode));
  ScratchBuffer<unsigned char> mem(bytes, s);
  w.ctl = reinterpret_cast<Ctl*>(mem.ptr + at_ctl);
  w.nodes = reinterpret_cast<LNode*>(mem.ptr + at_nodes);
  w.boxes = reinterpret_cast<uint4*>(mem.ptr + at_boxes);
  w.idx[0] = reinterpret_cast<uint32_t*>(mem.ptr + at_idx0);
  w.idx[1] = reinterpret_cast<uint32_t*>(mem.ptr + at_idx1);
  w.list[0] = reinterpret_cast<uint32_t*>(mem.ptr + at_list0);
  w.list[1] = reinterpret_cast<uint32_t*>(mem.ptr + at_list1);
  w.chunk_node[0] = reinterpret_cast<uint32_t*>(mem.ptr + at_cn0);
  w.chunk_node[1] = reinterpret_cast<uint32_t*>(mem.ptr + at_cn1);
  w.chunk_left = reinterpret_cast<uint32_t*>(mem.ptr + at_cl);
  w.hist = reinterpret_cast<uint32_t*>(mem.ptr + at_hist);
  w.bins[0] = reinterpret_cast<uint32_t*>(mem.ptr + at_b0);
  w.bins[1] = reinterpret_cast<uint32_t*>(mem.ptr + at_b1);
  w.small = reinterpret_cast<uint32_t*>(mem.ptr + at_small);
  w.temp = reinterpret_cast<BinaryNode*>(mem.ptr + at_temp);
  ScratchBuffer<uint32_t> order(ntri, s);
  ScratchBuffer<BinaryNode> dout(2 * ntri, s);
  const size_t small_smem = sizeof(Small) + (size_t)(kSmallThreads / 32) * 14 * o.bins * 4;
  static PerDevice<bool> opted_in;
  opted_in.get(current_device(), [] {
    VT_CUDA(cudaFuncSetAttribute(k_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(Small) + (size_t)(kSmallThreads / 32) * 14 * kMaxBins * 4)));
    return true;
  });
  const uint32_t init = std::max<uint32_t>({1u, (uint32_t)((ntri + kChunk - 1) / kChunk), (uint32_t)(21 * o.bins)});
  k_init<<<(init + 255) / 256, 256, 0, s>>>(w);
  VT_CUDA(cudaGetLastError());
  k_prep<<<(unsigned)((ntri + 255) / 256), 256, 0, s>>>(w, d_pos, o.position_stride, position_words / o.position_stride,
                                                        d_idx, o.index_stride);
  VT_CUDA(cudaGetLastError());
  // ---- large nodes: batches of levels; the host reads the counters after each
  Ctl ctl{};
  auto read_ctl = [&] {
    VT_CUDA(cudaMemcpyAsync(&ctl, w.ctl, sizeof ctl, cudaMemcpyDeviceToHost, s));
    VT_CUDA(cudaStreamSynchronize(s));
    if (ctl.bad & 1u) fail(VT_ERR_RANGE, "a triangle references an out-of-range vertex");
    if (ctl.bad & 2u) fail(VT_ERR_RANGE, "positions must be finite");
    if (ctl.bad) fail(VT_ERR_BUILD, "binary build: more nodes than bounded");
    if (ctl.depth_error)
      fail(VT_ERR_BUILD, "maxDepth=" + std::to_string(o.max_depth) + " prevents enforcing maxLeafTriangles=" +
                             std::to_string(o.max_leaf));
  };
  ctl.nodes = ctl.small = 1;
  if (ntri > (size_t)kSmall) {
    uint32_t level = 0;
    uint32_t batch = 3;
    for (size_t c = ntri; c > (size_t)kSmall; c >>= 1) ++batch;
    const size_t bin_smem = (size_t)21 * o.bins * 4;
    while (true) {
      for (uint32_t q = 0; q < batch; ++q, ++level) {
        k_bin<<<w.max_chunks, kChunkThreads, bin_smem, s>>>(w, level);
        k_choose<<<w.max_large, 128, 2 * bin_smem, s>>>(w, level);
        k_scatter<<<w.max_chunks, kChunkThreads, 0, s>>>(w, level);
      }
      VT_CUDA(cudaGetLastError());
      read_ctl();
      if (ctl.stop) {
        // the level's fallback sorts, then its scatter, which waited with them
        level = ctl.stop - 1u;
        const uint32_t p = level & 1u, n = ctl.large[p];
        VT_CUDA(cudaMemsetAsync(&w.ctl->stop, 0, sizeof ctl.stop, s));
        VT_CUDA(cudaMemsetAsync(&w.ctl->big, 0, sizeof ctl.big, s));
        k_scatter<<<w.max_chunks, kChunkThreads, 0, s>>>(w, level);
        k_sort<<<n, kSortThreads, kSortSmem, s>>>(w, level);
        VT_CUDA(cudaGetLastError());
        std::vector<LNode> nodes;  // the level's (they were made one after another)
        if (ctl.big) {
          const uint32_t first = level ? ctl.mark[level - 1] : 0u;
          nodes.resize(ctl.mark[level] - first);
          VT_CUDA(cudaMemcpyAsync(nodes.data(), w.nodes + first, nodes.size() * sizeof(LNode), cudaMemcpyDeviceToHost,
                                  s));
          VT_CUDA(cudaStreamSynchronize(s));
        }
        for (const LNode& N : nodes) {
          if (N.decision != 3 || N.count <= kSort) continue;
          uint32_t* dst = w.idx[p ^ 1u] + N.begin;
          sort_range(w.boxes, w.idx[p] + N.begin, dst, N.count, N.axis, s);
          for (int i = 0; i < 2; ++i) {
            const uint32_t c = i ? N.count - N.nl : N.nl;
            k_range_bounds<<<std::min<uint32_t>((c + 255) / 256, 592), 256, 0, s>>>(w, (uint32_t)(N.left + i),
                                                                                    dst + (i ? N.nl : 0));
          }
          VT_CUDA(cudaGetLastError());
        }
        ++level;
      }
      if (!ctl.large[level & 1u]) break;
      batch = 2;
    }
  }
  k_small<<<ctl.small, kSmallThreads, small_smem, s>>>(w, order.ptr);
  k_top<<<1, 1024, 0, s>>>(w);
  k_emit<<<ctl.nodes, 128, 0, s>>>(w, dout.ptr);
  VT_CUDA(cudaGetLastError());
  read_ctl();
  if (host_copy) {
    out.nodes.resize(ctl.total);
    out.reordered_to_source.resize(ntri);
    VT_CUDA(cudaMemcpyAsync(out.nodes.data(), dout.ptr, ctl.total * sizeof(BinaryNode), cudaMemcpyDeviceToHost, s));
    VT_CUDA(cudaMemcpyAsync(out.reordered_to_source.data(), order.ptr, ntri * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    VT_CUDA(cudaStreamSynchronize(s));
  }
  // deepest internal node: the last level holds only leaves
  out.depth = ctl.max_depth ? (int)ctl.max_depth - 1 : 0;
  if (keep) {
    keep->nodes = std::move(dout);
    keep->order = std::move(order);
    keep->n_nodes = (size_t)ctl.total;
    keep->ntri = ntri;
  }
  return out;
}

}  // namespace vt
