// bvh_encode_gpu.cu -- the 8-wide collapse and compressed-node encoding of
// bvh_encode.cpp on the GPU, producing the same node words and records.
//
//   1. parents of the binary nodes (children follow their parent: left at
//      i + 1, right at i + w6);
//   2. SAH-optimal collapse plan (Ylitie, Karras & Laine 2017, sec. 3.1),
//      bottom up: one thread per binary leaf climbs towards the root, the
//      second child to arrive at a node (an atomic counter per node) computes
//      its costs C(n), G(n, k) and splits from the children's, every value an
//      IEEE-double operation in the host's order, ties to the first minimum;
//   3. wide levels, top down, as the host's breadth-first queue, eight lanes per
//      wide node: per level the node's children (the plan's frontier or the
//      reference's greedy rule) are picked and put into slots (lane i holds child
//      i); an exclusive scan over the level gives each node its child base and
//      record block, so numbering equals the host's queue order; then lane s
//      quantises slot s, writes its records or lists its child for the next level.
//      The levels follow one another on the stream; the host reads their sizes
//      once per batch.  Bound by the dependent loads of a level, a dozen levels
//      deep: one thread per node and a host round trip per level took 0.67 ms for
//      65,536 triangles and 1.2 ms for 262,146, this 0.31 and 0.50 ms.
// Quantised child bounds are rounded outward exactly: each grid corner
// origin + q * 2^e is compared with the child bound through a nonoverlapping
// expansion of the sum (Shewchuk's grow-expansion of TwoSums), whose largest
// component carries the exact sign.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "bvh_exact.h"
#include "bvh_host.h"
#include "vt_common.h"

namespace vt {

namespace {

constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint32_t kMerged = 0x80000000u;  // frontier entry: the leaf slot of a subtree (not its node)

struct DpNode {
  double c;        // C(n)
  double g[7];     // G(n, k), k = 2 .. 8
  uint32_t first, count;
  uint8_t split[7];
  uint8_t as_leaf;
};

__device__ __forceinline__ bool leaf_word(uint32_t w7) { return (w7 & kLeafFlag) != 0; }

__device__ __forceinline__ double half_area_d(const BinaryNode& n) {
  double dx = __dsub_rn((double)n.mx[0], (double)n.mn[0]);
  double dy = __dsub_rn((double)n.mx[1], (double)n.mn[1]);
  double dz = __dsub_rn((double)n.mx[2], (double)n.mn[2]);
  dx = dx > 0.0 ? dx : 0.0;  // std::max(0.0, x): x when x > 0, else 0
  dy = dy > 0.0 ? dy : 0.0;
  dz = dz > 0.0 ? dz : 0.0;
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dy), __dmul_rn(dy, dz)), __dmul_rn(dz, dx));
}

__device__ __forceinline__ double dmin(double a, double b) { return b < a ? b : a; }  // std::min

__global__ void k_parents(const BinaryNode* __restrict__ nodes, uint32_t n, uint32_t* __restrict__ parent) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const BinaryNode b = nodes[i];
  if (leaf_word(b.w7)) return;
  parent[i + 1] = i;
  parent[i + b.w6] = i;
}

// loads a plan entry another thread wrote (L2, not a stale L1 line)
__device__ __forceinline__ void load_dp(const DpNode* p, DpNode& o) {
  const unsigned long long* s = reinterpret_cast<const unsigned long long*>(p);
  unsigned long long* d = reinterpret_cast<unsigned long long*>(&o);
#pragma unroll
  for (int k = 0; k < (int)(sizeof(DpNode) / 8); ++k) d[k] = __ldcg(s + k);
}

__global__ void k_plan(const BinaryNode* __restrict__ nodes, uint32_t n, const uint32_t* __restrict__ parent,
                       unsigned int* __restrict__ visits, DpNode* __restrict__ dp, double c_node, double c_tri,
                       int width) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const BinaryNode b = nodes[i];
  if (!leaf_word(b.w7)) return;
  DpNode d;
  d.first = b.w6;
  d.count = b.w7 & 0xFFFFu;
  d.c = __dmul_rn(__dmul_rn(c_tri, half_area_d(b)), (double)d.count);
  d.as_leaf = 1;
  for (int k = 0; k < 7; ++k) { d.g[k] = 0.0; d.split[k] = 0; }
  dp[i] = d;
  uint32_t x = parent[i];
  while (x != kNone) {
    __threadfence();
    if (atomicAdd(&visits[x], 1u) == 0u) return;  // the other child is not done yet
    __threadfence();
    const BinaryNode nb = nodes[x];
    const uint32_t l = x + 1, r = x + nb.w6;
    DpNode L, R;
    load_dp(dp + l, L);
    load_dp(dp + r, R);
    const bool lleaf = leaf_word(nodes[l].w7), rleaf = leaf_word(nodes[r].w7);
    DpNode o;
    o.first = L.first;
    o.count = L.count + R.count;
    const bool contiguous = R.first == L.first + L.count;
    for (int k = 2; k <= 8; ++k) {
      double best = INFINITY;
      int at = 1;
      for (int a = 1; a < k; ++a) {
        const double fl = (a < 2 || lleaf) ? L.c : dmin(L.c, L.g[a - 2]);
        const int bk = k - a;
        const double fr = (bk < 2 || rleaf) ? R.c : dmin(R.c, R.g[bk - 2]);
        const double v = __dadd_rn(fl, fr);
        if (v < best) { best = v; at = a; }
      }
      o.g[k - 2] = best;
      o.split[k - 2] = (uint8_t)at;
    }
    const double area = half_area_d(nb);
    o.c = __dadd_rn(__dmul_rn(c_node, area), o.g[width - 2]);
    o.as_leaf = 0;
    if (o.count <= 4 && contiguous) {
      const double leaf = __dmul_rn(__dmul_rn(c_tri, area), (double)o.count);
      if (leaf < o.c) {
        o.c = leaf;
        o.as_leaf = 1;
      }
    }
    dp[x] = o;
    x = parent[x];
  }
}

// The frontier of x over a slots (the host's SahCollapse::frontier), left first.
__device__ __forceinline__ void frontier(const BinaryNode* nodes, const DpNode* dp, uint32_t x, int a, uint32_t* out,
                                         int& m) {
  uint32_t sx[16];
  int sa[16], top = 0;
  sx[top] = x;
  sa[top++] = a;
  while (top > 0) {
    --top;
    const uint32_t y = sx[top];
    const int b = sa[top];
    const BinaryNode& ny = nodes[y];
    const DpNode& dy = dp[y];
    if (b >= 2 && !leaf_word(ny.w7) && dy.g[b - 2] < dy.c) {
      const int s = dy.split[b - 2];
      if (top + 2 > 16) { out[m++] = y; continue; }  // not reached: a frontier has at most 8 entries
      sx[top] = y + ny.w6;
      sa[top++] = b - s;
      sx[top] = y + 1;
      sa[top++] = s;
      continue;
    }
    if (m < 8) out[m++] = dy.as_leaf ? (y | kMerged) : y;
  }
}

// The reference's greedy rule (collectWideChildren, compressedWideBvh.ts:215-242).
__device__ __forceinline__ int greedy_children(const BinaryNode* nodes, uint32_t root, uint32_t out[8]) {
  const BinaryNode& r = nodes[root];
  if (leaf_word(r.w7)) { out[0] = root; return 1; }
  int n = 2;
  out[0] = root + 1;
  out[1] = root + r.w6;
  while (n < 8) {
    int at = -1;
    double best = -1;
    for (int i = 0; i < n; ++i) {
      const BinaryNode& c = nodes[out[i]];
      if (leaf_word(c.w7)) continue;
      const double a = half_area_d(c);
      if (a > best) { best = a; at = i; }
    }
    if (at < 0) break;
    const uint32_t x = out[at];
    for (int j = n; j > at + 1; --j) out[j] = out[j - 1];
    out[at] = x + 1;
    out[at + 1] = x + nodes[x].w6;
    ++n;
  }
  return n;
}

// Greedy slot assignment (the host's assign_slots), IEEE doubles in its order,
// by the eight lanes of a node's group: lane i holds child i (i < n) and finds
// its cheapest free slot, the group takes the cheapest (child, slot) of all, ties
// to the lower child and slot.  Returns the slot of child i in lane i.
__device__ __forceinline__ int assign_slots(const BinaryNode* nodes, const BinaryNode& parent, uint32_t ch, int n) {
  const int i = (int)(threadIdx.x & 7u);
  double dx = 0.0, dy = 0.0, dz = 0.0;
  if (i < n) {
    const BinaryNode c = nodes[ch & ~kMerged];
    const double pcx = __dmul_rn(0.5, __dadd_rn((double)parent.mn[0], (double)parent.mx[0]));
    const double pcy = __dmul_rn(0.5, __dadd_rn((double)parent.mn[1], (double)parent.mx[1]));
    const double pcz = __dmul_rn(0.5, __dadd_rn((double)parent.mn[2], (double)parent.mx[2]));
    dx = __dsub_rn(__dmul_rn(0.5, __dadd_rn((double)c.mn[0], (double)c.mx[0])), pcx);
    dy = __dsub_rn(__dmul_rn(0.5, __dadd_rn((double)c.mn[1], (double)c.mx[1])), pcy);
    dz = __dsub_rn(__dmul_rn(0.5, __dadd_rn((double)c.mn[2], (double)c.mx[2])), pcz);
  }
  uint32_t used = 0;
  int slot = -1;
  const int rounds = (int)__reduce_max_sync(0xFFFFFFFFu, (unsigned)n);  // the warp's four groups go together
  for (int round = 0; round < rounds; ++round) {
    double bc = INFINITY;
    int at = 64;  // 8 * child + slot; 64: nothing to offer
    if (i < n && slot < 0) {
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        if ((used >> s) & 1u) continue;
        const double sx = (s & 4) ? -1.0 : 1.0, sy = (s & 2) ? -1.0 : 1.0, sz = (s & 1) ? -1.0 : 1.0;
        const double cost = __dadd_rn(__dadd_rn(__dmul_rn(dx, sx), __dmul_rn(dy, sy)), __dmul_rn(dz, sz));
        if (at == 64 || cost < bc) { bc = cost; at = 8 * i + s; }
      }
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      const double oc = __shfl_xor_sync(0xFFFFFFFFu, bc, o);
      const int oa = __shfl_xor_sync(0xFFFFFFFFu, at, o);
      if (oa != 64 && (at == 64 || oc < bc || (oc == bc && oa < at))) { bc = oc; at = oa; }
    }
    if (at != 64) {
      used |= 1u << (at & 7);
      if ((at >> 3) == i) slot = at & 7;
    }
  }
  return slot;
}

// is child entry e a leaf slot?  (a merged subtree, or a binary leaf)
__device__ __forceinline__ bool entry_is_leaf(const BinaryNode* nodes, uint32_t e) {
  return (e & kMerged) || leaf_word(nodes[e].w7);
}

// A level of wide nodes: its node count, first node and first record; entry L + 1
// is written by level L's scan.
struct LevelState {
  uint32_t n, start, rec;
};
constexpr int kMaxLevels = 64;  // the binary tree is at most 58 deep
struct EncodeState {
  LevelState level[kMaxLevels + 1];
  uint32_t stop;   // level + 1 that ran out of records (its emission waits for a larger array); ~0: too many nodes
  uint32_t err;    // records beyond 2^30
};
// Device arrays of one encoding.
struct EncodeWork {
  EncodeState* state;
  uint32_t* list[2];   // binary nodes of a level's wide nodes, by level parity
  uint32_t* slots;     // per node of the level: the child entry of each slot (kNone: empty)
  uint32_t* n_int;     // per node: internal children, then their offset
  uint32_t* span;      // per node: records, then their offset
  uint32_t max_wide;
};
constexpr int kEncodeThreads = 128;
constexpr int kEncodeNodes = kEncodeThreads / 8;

// sah: 0 the reference's greedy collapse, else the SAH-optimal collapse at that width (2..8)
__global__ void __launch_bounds__(kEncodeThreads) k_level_plan(const BinaryNode* __restrict__ nodes,
                                                               const DpNode* __restrict__ dp, int sah, EncodeWork w,
                                                               int level) {
  constexpr uint32_t kAll = 0xFFFFFFFFu;
  if (w.state->stop) return;
  const uint32_t n_level = w.state->level[level].n;
  const int i = (int)(threadIdx.x & 7u), shift = (int)(threadIdx.x & 24u);
  __shared__ uint32_t pick[kEncodeNodes][8];
  uint32_t* mine = pick[threadIdx.x >> 3];
  for (uint32_t base = blockIdx.x * kEncodeNodes; base < n_level; base += gridDim.x * kEncodeNodes) {
    const uint32_t j = base + (threadIdx.x >> 3);
    const bool on = j < n_level;
    const uint32_t x = on ? w.list[level & 1][j] : 0u;
    int n = 0;
    if (on && i == 0) {
      if (sah) {
        if (leaf_word(nodes[x].w7)) {
          mine[0] = x;
          n = 1;
        } else {
          const int s = dp[x].split[sah - 2];
          frontier(nodes, dp, x + 1, s, mine, n);
          frontier(nodes, dp, x + nodes[x].w6, sah - s, mine, n);
        }
      } else {
        n = greedy_children(nodes, x, mine);
      }
    }
    __syncwarp();
    n = __shfl_sync(kAll, n, shift);
    const uint32_t ch = i < n ? mine[i] : kNone;
    const int slot = assign_slots(nodes, nodes[x], ch, n);
    const bool leaf = i < n && entry_is_leaf(nodes, ch);
    // the masks by slot: lane i speaks for slot `slot`
    uint32_t at = i < n ? 1u << slot : 0u, leaves = leaf ? at : 0u;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      at |= __shfl_xor_sync(kAll, at, o);
      leaves |= __shfl_xor_sync(kAll, leaves, o);
    }
    if (on) {
      uint32_t* out = w.slots + 8 * (size_t)j;
      if (i < n) out[slot] = ch;
      if (!((at >> i) & 1u)) out[i] = kNone;
      if (i == 0) {
        w.n_int[j] = (uint32_t)__popc(at & ~leaves);
        w.span[j] = leaves ? 4u * (uint32_t)((31 - __clz(leaves)) - (__ffs(leaves) - 1)) + 4u : 0u;
      }
    }
    __syncwarp();
  }
}

// Exclusive scans of a level's two counts in one CTA (levels are at most a few
// 100 k nodes), and the next level's state.
__global__ void __launch_bounds__(1024) k_level_scan(EncodeWork w, int level, uint32_t rec_cap) {
  __shared__ unsigned long long wa[32], wb[32];
  __shared__ unsigned long long carry_a, carry_b;
  EncodeState* st = w.state;
  if (st->stop) return;
  uint32_t* a = w.n_int;
  uint32_t* b = w.span;
  const LevelState cur = st->level[level];
  const uint32_t n = cur.n;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (threadIdx.x == 0) { carry_a = 0; carry_b = 0; }
  __syncthreads();
  for (uint32_t base = 0; base < n; base += blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    const unsigned long long va = i < n ? a[i] : 0, vb = i < n ? b[i] : 0;
    unsigned long long sa = va, sb = vb;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long ta = __shfl_up_sync(0xFFFFFFFFu, sa, o), tb = __shfl_up_sync(0xFFFFFFFFu, sb, o);
      if (lane >= o) { sa += ta; sb += tb; }
    }
    if (lane == 31) { wa[wid] = sa; wb[wid] = sb; }
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long ra = carry_a, rb = carry_b;
      for (int q = 0; q < (int)(blockDim.x >> 5); ++q) {
        const unsigned long long xa = wa[q], xb = wb[q];
        wa[q] = ra;
        wb[q] = rb;
        ra += xa;
        rb += xb;
      }
      carry_a = ra;
      carry_b = rb;
    }
    __syncthreads();
    if (i < n) {
      a[i] = (uint32_t)(wa[wid] + sa - va);
      b[i] = (uint32_t)(wb[wid] + sb - vb);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    st->level[level + 1] = {(uint32_t)carry_a, cur.start + cur.n, (uint32_t)(cur.rec + carry_b)};
    if (cur.start + cur.n + carry_a > w.max_wide) st->stop = ~0u;
    else if (cur.rec + carry_b > rec_cap) st->stop = (uint32_t)level + 1u;
  }
}

// smallest e with origin + 255 2^e >= hi (exactly), clamped to the normal range (the host's grid_exponent)
__device__ __forceinline__ int grid_exponent(float origin, float hi) {
  const double extent = __dsub_rn((double)hi, (double)origin);
  if (!(extent > 0)) return -126;
  int e;
  frexp(__ddiv_rn(extent, 255.0), &e);
  while (e > -126 && ldexp(255.0, e - 1) >= extent) --e;
  while (e < 127 && corner_sign(origin, 255, e, hi) < 0) ++e;
  return min(127, max(-126, e));
}

// Unit normal as the reference's watertight test derives it (the host's
// reference_normal): single precision, every operation rounded on its own.
__device__ __forceinline__ bool reference_normal(const float a[3], const float b[3], const float c[3], float nn[3]) {
  float e1r[3], e2r[3];
  for (int k = 0; k < 3; ++k) { e1r[k] = __fsub_rn(b[k], a[k]); e2r[k] = __fsub_rn(c[k], a[k]); }
  float es = 0.0f;
  for (int k = 0; k < 3; ++k) es = fmaxf(es, fabsf(e1r[k]));
  for (int k = 0; k < 3; ++k) es = fmaxf(es, fabsf(e2r[k]));
  if (!(es > 0.0f) || !isfinite(es)) return false;
  float s1[3], s2[3];
  for (int k = 0; k < 3; ++k) { s1[k] = __fdiv_rn(e1r[k], es); s2[k] = __fdiv_rn(e2r[k], es); }
  const float nr[3] = {__fsub_rn(__fmul_rn(s1[1], s2[2]), __fmul_rn(s1[2], s2[1])),
                       __fsub_rn(__fmul_rn(s1[2], s2[0]), __fmul_rn(s1[0], s2[2])),
                       __fsub_rn(__fmul_rn(s1[0], s2[1]), __fmul_rn(s1[1], s2[0]))};
  const float ns = fmaxf(fmaxf(fabsf(nr[0]), fabsf(nr[1])), fabsf(nr[2]));
  if (!(ns > 0.0f) || !isfinite(ns)) return false;
  const float nd[3] = {__fdiv_rn(nr[0], ns), __fdiv_rn(nr[1], ns), __fdiv_rn(nr[2], ns)};
  const float l2 = __fadd_rn(__fadd_rn(__fmul_rn(nd[0], nd[0]), __fmul_rn(nd[1], nd[1])), __fmul_rn(nd[2], nd[2]));
  const float nl = __fsqrt_rn(l2);
  if (!(nl > 0.0f) || !isfinite(nl)) return false;
  for (int k = 0; k < 3; ++k) nn[k] = __fdiv_rn(nd[k], nl);
  return true;
}

struct EmitArgs {
  const BinaryNode* nodes;
  const DpNode* dp;          // SAH plan (first / count of merged subtrees), null for the greedy rule
  const uint32_t* order;     // BVH-order triangle (or instance) permutation
  const float* pos;          // triangles: vertex positions (stride ps)
  int ps;
  const uint32_t* idx;       // triangles: indices (stride is)
  int is;
  const uint32_t* tri_mat;   // optional, one per source triangle
  const uint32_t* mat_flags; // optional, one per material: flags word of its records
  const float* inst_recs;    // top level: 16 floats per instance (else null)
  uint32_t node_base, rec_base;
};

// The record of triangle (or instance) src.
__device__ __forceinline__ void write_record(const EmitArgs& A, uint32_t src, float4* rec) {
  if (A.inst_recs) {
    const float4* in = reinterpret_cast<const float4*>(A.inst_recs) + 4 * (size_t)src;
    for (int k = 0; k < 4; ++k) rec[k] = in[k];
    return;
  }
  const uint32_t* iv = A.idx + (size_t)src * A.is;
  float v[3][3];
  for (int vi = 0; vi < 3; ++vi)
    for (int k = 0; k < 3; ++k) v[vi][k] = A.pos[(size_t)iv[vi] * A.ps + k];
  const uint32_t mat = A.tri_mat ? A.tri_mat[src] : 0u;
  float nn[3] = {0, 0, 0};
  const bool valid = reference_normal(v[0], v[1], v[2], nn);
  const uint32_t flags = valid && A.mat_flags && A.tri_mat ? A.mat_flags[mat] : 0u;
  rec[0] = make_float4(v[0][0], v[0][1], v[0][2], __uint_as_float(src));
  rec[1] = make_float4(v[1][0], v[1][1], v[1][2], A.tri_mat ? __uint_as_float(mat) : 0.0f);
  rec[2] = make_float4(v[2][0], v[2][1], v[2][2], __uint_as_float(flags));
  rec[3] = make_float4(nn[0], nn[1], nn[2], valid ? 1.0f : 0.0f);
}

__global__ void __launch_bounds__(kEncodeThreads) k_level_emit(EmitArgs A, EncodeWork w, int level,
                                                               uint32_t* __restrict__ words, float* __restrict__ recs) {
  constexpr uint32_t kAll = 0xFFFFFFFFu;
  if (w.state->stop) return;
  const LevelState st = w.state->level[level];
  const int s = (int)(threadIdx.x & 7u), shift = (int)(threadIdx.x & 24u);
  uint32_t* next = w.list[(level & 1) ^ 1];
  for (uint32_t base = blockIdx.x * kEncodeNodes; base < st.n; base += gridDim.x * kEncodeNodes) {
    const uint32_t j = base + (threadIdx.x >> 3);
    const bool on = j < st.n;
    const uint32_t e = on ? w.slots[8 * (size_t)j + s] : kNone;
    const bool child = e != kNone, leaf = child && entry_is_leaf(A.nodes, e);
    const uint32_t all = (__ballot_sync(kAll, child) >> shift) & 0xFFu;
    const uint32_t leaves = (__ballot_sync(kAll, leaf) >> shift) & 0xFFu, imask = all & ~leaves;
    const BinaryNode parent = A.nodes[on ? w.list[level & 1][j] : 0u];
    const float pm[3] = {parent.mn[0], parent.mn[1], parent.mn[2]};
    int mine = 0;  // lane k < 3: axis k's grid exponent
    if (s < 3) mine = grid_exponent(s == 0 ? pm[0] : (s == 1 ? pm[1] : pm[2]),
                                    s == 0 ? parent.mx[0] : (s == 1 ? parent.mx[1] : parent.mx[2]));
    int ex[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) ex[k] = __shfl_sync(kAll, mine, shift + k);
    const uint32_t first_leaf = leaves ? (uint32_t)(__ffs(leaves) - 1) : 0u;
    const uint32_t int_off = on ? w.n_int[j] : 0u, block = st.rec + (on ? w.span[j] : 0u);
    uint32_t* out = words + 20 * (size_t)(st.start + j);
    uint32_t valid = 0;
    if (on) {
      uint8_t* bytes = reinterpret_cast<uint8_t*>(out);
      uint8_t* qlo = bytes + 32 + s;
      uint8_t* qhi = bytes + 56 + s;
      if (!child) {
        for (int k = 0; k < 3; ++k) { qlo[8 * k] = 255; qhi[8 * k] = 0; }
      } else {
        const uint32_t id = e & ~kMerged;
        const BinaryNode c = A.nodes[id];
        for (int k = 0; k < 3; ++k) {
          const double step = ldexp(1.0, ex[k]);
          const double lo = floor(__ddiv_rn(__dsub_rn((double)c.mn[k], (double)pm[k]), step));
          const double hi = ceil(__ddiv_rn(__dsub_rn((double)c.mx[k], (double)pm[k]), step));
          int ql = (int)fmin(255.0, fmax(0.0, lo));
          int qh = (int)fmin(255.0, fmax(0.0, hi));
          while (ql > 0 && corner_sign(pm[k], ql, ex[k], c.mn[k]) > 0) --ql;
          while (qh < 255 && corner_sign(pm[k], qh, ex[k], c.mx[k]) < 0) ++qh;
          qlo[8 * k] = (uint8_t)ql;
          qhi[8 * k] = (uint8_t)qh;
        }
        if (leaf) {
          uint32_t first, cnt;
          if (e & kMerged) {
            first = A.dp[id].first;
            cnt = A.dp[id].count;
          } else {
            first = c.w6;
            cnt = c.w7 & 0xFFFFu;
          }
          valid = ((1u << cnt) - 1u) << (4 * s);
          float* to = recs + 16 * ((size_t)block + 4 * (s - first_leaf));
          for (uint32_t t = 0; t < cnt; ++t) write_record(A, A.order[first + t], reinterpret_cast<float4*>(to + 16 * t));
        } else {
          next[int_off + (uint32_t)__popc(imask & ((1u << s) - 1u))] = id;
        }
      }
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) valid |= __shfl_xor_sync(kAll, valid, o);
    if (on && s == 0) {
      if ((unsigned long long)A.rec_base + block + 32 >= 0x40000000ull) atomicOr(&w.state->err, 1u);
      out[0] = __float_as_uint(pm[0]);
      out[1] = __float_as_uint(pm[1]);
      out[2] = __float_as_uint(pm[2]);
      out[3] = (uint32_t)(ex[0] + 127) | (uint32_t)(ex[1] + 127) << 8 | (uint32_t)(ex[2] + 127) << 16 | imask << 24;
      out[4] = A.node_base + st.start + st.n + int_off;
      out[5] = A.rec_base + block - 4u * first_leaf;
      out[6] = valid;
      out[7] = 0u;
    }
  }
}

}  // namespace

WideBvhHost encode_wide_gpu(const BinaryBvhDevice& bin, const float* d_pos, int pos_stride, const uint32_t* d_idx,
                            int idx_stride, const uint32_t* d_tri_mat, uint32_t node_base, uint32_t rec_base,
                            const WideCollapse* sah, const float* d_inst_recs, cudaStream_t s, WideBvhDevice* keep,
                            bool host_copy, const uint32_t* d_mat_flags) {
  WideBvhHost out;
  const uint32_t n = (uint32_t)bin.n_nodes;
  if (bin.ntri == 0 || n == 0) {
    // an empty tree: one node with all slots empty (inverted boxes), no records
    uint32_t w[20] = {};
    std::memset(reinterpret_cast<uint8_t*>(w) + 32, 0xFF, 24);
    out.nodes.assign(w, w + 20);
    out.depth = 1;
    if (keep) {
      keep->nodes.resize(20, s);
      VT_CUDA(cudaMemcpyAsync(keep->nodes.ptr, w, sizeof w, cudaMemcpyHostToDevice, s));
      keep->recs.resize(0, s);
      keep->n_nodes = 1;
      keep->n_recs = 0;
      keep->depth = 1;
      VT_CUDA(cudaStreamSynchronize(s));
    }
    return out;
  }
  ScratchBuffer<DpNode> dp;
  const int width = sah ? std::min(std::max(sah->width, 2), 8) : 0;
  if (sah) {
    ScratchBuffer<uint32_t> parent(n, s);
    ScratchBuffer<unsigned int> visits(n, s);
    dp.resize(n, s);
    VT_CUDA(cudaMemsetAsync(parent.ptr, 0xFF, n * sizeof(uint32_t), s));
    VT_CUDA(cudaMemsetAsync(visits.ptr, 0, n * sizeof(unsigned int), s));
    k_parents<<<(n + 255) / 256, 256, 0, s>>>(bin.nodes.ptr, n, parent.ptr);
    VT_CUDA(cudaGetLastError());
    k_plan<<<(n + 255) / 256, 256, 0, s>>>(bin.nodes.ptr, n, parent.ptr, visits.ptr, dp.ptr, sah->c_node, sah->c_tri,
                                           width);
    VT_CUDA(cudaGetLastError());
    VT_CUDA(cudaStreamSynchronize(s));
  }
  // wide nodes: at most one per binary interior node (a lone leaf root: one)
  const uint32_t max_wide = n / 2 + 1;
  ScratchBuffer<uint32_t> words((size_t)20 * max_wide, s);
  size_t rec_cap = 28 + 4 * (size_t)bin.ntri + 64;
  ScratchBuffer<float> recs(16 * rec_cap, s);
  VT_CUDA(cudaMemsetAsync(recs.ptr, 0, recs.bytes(), s));
  ScratchBuffer<uint32_t> lvl_a(max_wide, s), lvl_b(max_wide, s), n_int(max_wide, s), span(max_wide, s),
      slots(8 * (size_t)max_wide, s);
  ScratchBuffer<EncodeState> state(1, s);
  EncodeWork w{state.ptr, {lvl_a.ptr, lvl_b.ptr}, slots.ptr, n_int.ptr, span.ptr, max_wide};
  EncodeState st{};
  st.level[0] = {1u, 0u, 28u};
  VT_CUDA(cudaMemcpyAsync(state.ptr, &st, sizeof st, cudaMemcpyHostToDevice, s));
  VT_CUDA(cudaMemsetAsync(lvl_a.ptr, 0, sizeof(uint32_t), s));  // the root
  EmitArgs A{bin.nodes.ptr, sah ? dp.ptr : nullptr, bin.order.ptr, d_pos, pos_stride, d_idx, idx_stride, d_tri_mat,
             d_mat_flags, d_inst_recs, node_base, rec_base};
  // A level holds at most eight times the one above; levels beyond the last are empty
  // launches.  The first batch covers a tree of four children per wide node.
  auto blocks = [&](int level) {
    const uint32_t most = level < 8 ? (uint32_t)std::min<uint64_t>(1ull << (3 * level), max_wide) : max_wide;
    return std::min<unsigned>((most + kEncodeNodes - 1) / kEncodeNodes, 148 * 16);
  };
  int level = 0, batch = 2;
  for (uint32_t q = max_wide; q > 1; q >>= 2) ++batch;
  int depth = 0;
  while (true) {
    const int last = std::min(level + batch, kMaxLevels);
    for (; level < last; ++level) {
      k_level_plan<<<blocks(level), kEncodeThreads, 0, s>>>(bin.nodes.ptr, sah ? dp.ptr : nullptr, sah ? width : 0, w,
                                                            level);
      k_level_scan<<<1, 1024, 0, s>>>(w, level, (uint32_t)std::min<size_t>(rec_cap, 0xFFFFFFFFu));
      k_level_emit<<<blocks(level), kEncodeThreads, 0, s>>>(A, w, level, words.ptr, recs.ptr);
    }
    VT_CUDA(cudaGetLastError());
    VT_CUDA(cudaMemcpyAsync(&st, state.ptr, sizeof st, cudaMemcpyDeviceToHost, s));
    VT_CUDA(cudaStreamSynchronize(s));
    if (st.stop == ~0u) fail(VT_ERR_BUILD, "wide encoding: more nodes than bounded");
    if (st.stop) {
      // grow the record array (more leaf slots than the first estimate) and emit the level that waited
      level = (int)st.stop - 1;
      const size_t cap = std::max<size_t>((size_t)st.level[level + 1].rec + 64, rec_cap * 3 / 2);
      ScratchBuffer<float> bigger(16 * cap, s);
      VT_CUDA(cudaMemsetAsync(bigger.ptr, 0, bigger.bytes(), s));
      VT_CUDA(cudaMemcpyAsync(bigger.ptr, recs.ptr, 16 * sizeof(float) * (size_t)st.level[level].rec,
                              cudaMemcpyDeviceToDevice, s));
      recs = std::move(bigger);
      rec_cap = cap;
      VT_CUDA(cudaMemsetAsync(&state.ptr->stop, 0, sizeof(uint32_t), s));
      k_level_emit<<<blocks(level), kEncodeThreads, 0, s>>>(A, w, level, words.ptr, recs.ptr);
      VT_CUDA(cudaGetLastError());
      ++level;
    }
    if (level >= kMaxLevels || st.level[level].n == 0) break;
    batch = 3;
  }
  while (depth < level && st.level[depth].n) ++depth;
  const uint32_t level_start = st.level[depth].start, rec_used = st.level[depth].rec;
  const uint32_t bad = st.err;
  if (bad) fail(VT_ERR_BUILD, "leaf records exceed 2^30");
  out.depth = depth;
  if (host_copy) {
    out.nodes.resize((size_t)20 * level_start);
    out.tris.resize((size_t)16 * rec_used);
    VT_CUDA(cudaMemcpyAsync(out.nodes.data(), words.ptr, out.nodes.size() * 4, cudaMemcpyDeviceToHost, s));
    VT_CUDA(cudaMemcpyAsync(out.tris.data(), recs.ptr, out.tris.size() * 4, cudaMemcpyDeviceToHost, s));
    VT_CUDA(cudaStreamSynchronize(s));
  }
  if (keep) {
    keep->nodes = std::move(words);
    keep->recs = std::move(recs);
    keep->n_nodes = level_start;
    keep->n_recs = rec_used;
    keep->depth = depth;
  }
  return out;
}

}  // namespace vt
