// bvh_prove_gpu.cu -- the publication proofs of bvh_validate.cpp on the arrays
// a device build leaves on the GPU: the packed binary tree (the reference's
// validateBvhEncoding, packages/shared-bvh/src/validateBvhEncoding.ts:55) and
// the 8-wide encoding (exclusive reachability, record tiling, conservative
// culling boxes, the traversal's stack bound).
//
// One thread per node checks its own words, claims its children (each node but
// the root must be claimed exactly once, by a node before it: no cycle, nothing
// unreachable) and notes itself as their parent; a second pass, per binary node
// or per slot of a wide node, climbs to the root: the depth, and for a leaf
// slot the bounds of its valid triangles against its own box and every
// ancestor slot's -- the exact sign of each grid corner against each bound
// (bvh_exact.h).  Bound by the climbs' dependent loads (L2): 65,536 triangles
// prove in about 60 us; the host's walk in 113-bit arithmetic takes 23 ms, and
// runs only to name what a failed proof found.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "bvh_exact.h"
#include "bvh_host.h"
#include "vt_common.h"

namespace vt {

namespace {

struct Verdict {
  uint32_t bad;          // non-zero: a check failed
  uint32_t depth;        // deepest node (root 0)
  unsigned long long items;
};

__device__ __forceinline__ void flag(Verdict* v) { atomicOr(&v->bad, 1u); }

__device__ __forceinline__ bool leaf_word(uint32_t w7) { return (w7 >> 16) == 0xFFFFu; }

// ---------------------------------------------------------------- binary tree
__global__ void k_prove_binary_links(const BinaryNode* __restrict__ nodes, uint32_t n, uint32_t ntri,
                                     uint32_t* __restrict__ parent, uint32_t* __restrict__ covered, Verdict* v) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const BinaryNode b = nodes[i];
  bool ok = true;
  for (int k = 0; k < 3; ++k)
    ok = ok && isfinite(b.mn[k]) && isfinite(b.mx[k]) && b.mn[k] <= b.mx[k];
  if (leaf_word(b.w7)) {
    const uint32_t count = b.w7 & 0xFFFFu;
    if (b.w6 > ntri || count > ntri - b.w6) {
      ok = false;
    } else {
      for (uint32_t t = 0; t < count; ++t) ok = ok && atomicAdd(&covered[b.w6 + t], 1u) == 0u;
      atomicAdd(&v->items, (unsigned long long)count);
    }
  } else {
    ok = ok && b.w7 <= 2u && b.w6 > 1u && (unsigned long long)i + b.w6 < n;
    if (ok) {
      const uint32_t ch[2] = {i + 1u, i + b.w6};
      for (int c = 0; c < 2; ++c) {
        ok = ok && atomicExch(&parent[ch[c]], i) == 0xFFFFFFFFu;
        const BinaryNode q = nodes[ch[c]];
        for (int k = 0; k < 3; ++k) ok = ok && !(q.mn[k] < b.mn[k]) && !(q.mx[k] > b.mx[k]);
      }
    }
  }
  if (!ok) flag(v);
}

__global__ void k_prove_binary_depth(uint32_t n, const uint32_t* __restrict__ parent, Verdict* v) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (v->bad || i >= n) return;
  uint32_t x = i, depth = 0;
  while (x != 0u) {  // parents come before their children: the climb ends at the root
    const uint32_t p = parent[x];
    if (p >= x) {    // (unclaimed, or the root claimed)
      flag(v);
      return;
    }
    x = p;
    ++depth;
  }
  if (i == 0 && parent[0] != 0xFFFFFFFFu) flag(v);
  if (depth > v->depth) atomicMax(&v->depth, depth);
}

// ---------------------------------------------------------------- 8-wide tree
__device__ __forceinline__ uint32_t byte_of(const uint32_t* w, int i) { return (w[i >> 2] >> (8 * (i & 3))) & 0xFFu; }

__global__ void k_prove_wide_links(const uint32_t* __restrict__ words, uint32_t n, uint32_t* __restrict__ parent,
                                   Verdict* v) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t w[20];
  for (int k = 0; k < 20; ++k) w[k] = words[20 * (size_t)i + k];
  const uint32_t imask = byte_of(w, 15), child_base = w[4], valid = w[6];
  uint32_t seen = 0;
  bool ok = true;
  for (int s = 0; s < 8; ++s) {
    const uint32_t nib = (valid >> (4 * s)) & 0xFu;
    const bool internal = (imask >> s) & 1u;
    for (int k = 0; k < 3; ++k) {
      const uint32_t lo = byte_of(w, 32 + 8 * k + s), hi = byte_of(w, 56 + 8 * k + s);
      if (!internal && nib == 0) ok = ok && lo == 255u && hi == 0u;
      else ok = ok && lo <= hi;
    }
    if (internal) {
      const unsigned long long c = (unsigned long long)child_base + seen++;
      ok = ok && nib == 0 && c < n && c > i;
      if (c < n) ok = ok && atomicExch(&parent[c], (i << 3) | (uint32_t)s) == 0xFFFFFFFFu;
    } else if (nib) {
      ok = ok && (nib == 0x1u || nib == 0x3u || nib == 0x7u || nib == 0xFu);
    }
  }
  if (!ok) flag(v);
}

// thread per slot: leaf records, and the climb through the boxes that cull them
__global__ void __launch_bounds__(128) k_prove_wide_slots(const uint32_t* __restrict__ words, uint32_t n,
                                                          const float4* __restrict__ recs, size_t n_recs,
                                                          size_t n_items, const uint32_t* __restrict__ parent,
                                                          uint32_t* __restrict__ named, Verdict* v) {
  const unsigned long long at = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v->bad || at >= 8ull * n) return;
  uint32_t node = (uint32_t)(at >> 3);
  int s = (int)(at & 7u);
  const uint32_t* w = words + 20 * (size_t)node;
  const uint32_t nib = (w[6] >> (4 * s)) & 0xFu;
  float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  bool ok = true, boxed = false;
  if (nib) {
    const int cnt = __popc(nib);
    for (int i = 0; i < cnt; ++i) {
      const unsigned long long r = (unsigned long long)w[5] + 4u * (uint32_t)s + (uint32_t)i;
      if (r >= n_recs) {
        flag(v);
        return;
      }
      const float4* rec = recs + 4 * r;
      const float4 a = rec[0], b = rec[1], c = rec[2], q = rec[3];
      const uint32_t id = __float_as_uint(a.w);
      if (id >= n_items || atomicAdd(&named[id], 1u) != 0u) {
        flag(v);
        return;
      }
      if (q.w == 0.0f) continue;  // the watertight normal derivation rejects it: never hit
      boxed = true;
      const float x[3][3] = {{a.x, b.x, c.x}, {a.y, b.y, c.y}, {a.z, b.z, c.z}};
      for (int k = 0; k < 3; ++k)
        for (int j = 0; j < 3; ++j) {
          ok = ok && x[k][j] == x[k][j];  // a NaN is in no box
          lo[k] = fminf(lo[k], x[k][j]);
          hi[k] = fmaxf(hi[k], x[k][j]);
        }
    }
    atomicAdd(&v->items, (unsigned long long)cnt);
  }
  if (s != 0 && !boxed) {  // slot 0 climbs for its node's depth
    if (!ok) flag(v);
    return;
  }
  uint32_t depth = 0;
  while (true) {
    const uint32_t* q = words + 20 * (size_t)node;
    if (boxed) {
      const uint32_t ex = q[3];
      for (int k = 0; k < 3; ++k) {
        const float org = __uint_as_float(q[k]);
        const int e = (int)((ex >> (8 * k)) & 0xFFu) - 127;
        ok = ok && corner_sign(org, (int)byte_of(q, 32 + 8 * k + s), e, lo[k]) <= 0 &&
             corner_sign(org, (int)byte_of(q, 56 + 8 * k + s), e, hi[k]) >= 0;
      }
    }
    if (node == 0u) break;
    const uint32_t p = parent[node];
    if (p == 0xFFFFFFFFu) {  // nothing leads here
      flag(v);
      return;
    }
    node = p >> 3;  // before its child (k_prove_wide_links): the climb ends at the root
    s = (int)(p & 7u);
    ++depth;
  }
  if (!ok) flag(v);
  if (depth > v->depth) atomicMax(&v->depth, depth);
}

Verdict read_verdict(const Verdict* d, cudaStream_t s) {
  Verdict v;
  VT_CUDA(cudaGetLastError());
  VT_CUDA(cudaMemcpyAsync(&v, d, sizeof v, cudaMemcpyDeviceToHost, s));
  VT_CUDA(cudaStreamSynchronize(s));
  return v;
}

}  // namespace

void prove_binary_gpu(const BinaryNode* d_nodes, size_t n_nodes, size_t ntri, int stack_cap, cudaStream_t s) {
  ScratchBuffer<uint32_t> parent(n_nodes, s), covered(std::max<size_t>(ntri, 1), s);
  ScratchBuffer<Verdict> verdict(1, s);
  VT_CUDA(cudaMemsetAsync(parent.ptr, 0xFF, parent.bytes(), s));
  VT_CUDA(cudaMemsetAsync(covered.ptr, 0, covered.bytes(), s));
  VT_CUDA(cudaMemsetAsync(verdict.ptr, 0, sizeof(Verdict), s));
  const unsigned g = (unsigned)((n_nodes + 255) / 256);
  k_prove_binary_links<<<g, 256, 0, s>>>(d_nodes, (uint32_t)n_nodes, (uint32_t)ntri, parent.ptr, covered.ptr,
                                         verdict.ptr);
  k_prove_binary_depth<<<g, 256, 0, s>>>((uint32_t)n_nodes, parent.ptr, verdict.ptr);
  const Verdict v = read_verdict(verdict.ptr, s);
  if (!v.bad && v.items == ntri && (int)v.depth + 1 <= stack_cap) return;
  BinaryBvhHost h;
  h.nodes.resize(n_nodes);
  VT_CUDA(cudaMemcpyAsync(h.nodes.data(), d_nodes, n_nodes * sizeof(BinaryNode), cudaMemcpyDeviceToHost, s));
  VT_CUDA(cudaStreamSynchronize(s));
  validate_binary(h, (int64_t)ntri, stack_cap);
  fail(VT_ERR_BUILD, "binary encoding proof failed on the device");
}

void prove_wide_gpu(const uint32_t* d_words, size_t n_nodes, const float* d_recs, size_t n_recs, size_t n_items,
                    int stack_cap, cudaStream_t s) {
  if (n_nodes >= (1u << 29)) fail(VT_ERR_BUILD, "8-wide encoding proof: too many nodes");
  ScratchBuffer<uint32_t> parent(n_nodes, s), named(std::max<size_t>(n_items, 1), s);
  ScratchBuffer<Verdict> verdict(1, s);
  VT_CUDA(cudaMemsetAsync(parent.ptr, 0xFF, parent.bytes(), s));
  VT_CUDA(cudaMemsetAsync(named.ptr, 0, named.bytes(), s));
  VT_CUDA(cudaMemsetAsync(verdict.ptr, 0, sizeof(Verdict), s));
  k_prove_wide_links<<<(unsigned)((n_nodes + 127) / 128), 128, 0, s>>>(d_words, (uint32_t)n_nodes, parent.ptr,
                                                                       verdict.ptr);
  k_prove_wide_slots<<<(unsigned)((8 * n_nodes + 127) / 128), 128, 0, s>>>(
      d_words, (uint32_t)n_nodes, reinterpret_cast<const float4*>(d_recs), n_recs, n_items, parent.ptr, named.ptr,
      verdict.ptr);
  const Verdict v = read_verdict(verdict.ptr, s);
  if (!v.bad && v.items == n_items && 2 * ((int)v.depth + 1) + 2 <= stack_cap) return;
  std::vector<uint32_t> words(20 * n_nodes);
  std::vector<float> recs(16 * n_recs);
  VT_CUDA(cudaMemcpyAsync(words.data(), d_words, words.size() * 4, cudaMemcpyDeviceToHost, s));
  if (n_recs) VT_CUDA(cudaMemcpyAsync(recs.data(), d_recs, recs.size() * 4, cudaMemcpyDeviceToHost, s));
  VT_CUDA(cudaStreamSynchronize(s));
  validate_wide(words.data(), n_nodes, recs.data(), n_recs, 0, n_items, false, stack_cap);
  fail(VT_ERR_BUILD, "8-wide encoding proof failed on the device");
}

}  // namespace vt
