// nrc_kernels.cu -- neural radiance cache kernels for sm_100a.
//
// k_nrc_infer   persistent; per tile of 128 queries: encode
//               (hash grid + SH4 + surface features) into fp16 rows in TMEM, then six
//               tcgen05.mma layers (M=128, N=64, K=64 as four K=16 steps) with
//               A and the fp32 accumulator in TMEM, ReLU + fp16 repack in the epilogue
//               between layers, prediction read from TMEM.
// k_nrc_train   persistent; per tile: encode, forward keeping every layer's
//               activations in swizzled shared-memory tiles, relative-L2 output gradient,
//               backward: per layer dW += G^T X (tensor core, accumulated across
//               the CTA's tiles in TMEM) and dX = G W (tensor core), ReLU mask
//               from the stored activations; the input gradient of the 32
//               hash-grid features is scattered into the table gradient with the
//               trilinear weights (nrcEncoding.ts hashGridBackward:214).
// k_nrc_adam    Adam with the reference's non-finite guards and +-65504 clamp.
//
// Every mbarrier wait is bounded (about one second of clocks); on expiry the
// kernel records v.error, waits (bounded) for its issued MMAs, frees its TMEM
// and returns.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "nrc.h"
#include "tc_sm100.cuh"
#include "vt_common.h"

namespace vt {
namespace nrc {

namespace {

constexpr long long kWaitCycles = kDefaultWaitCycles;  // drains after an expired wait
constexpr uint32_t kTileBytes = kTile * kWidth * 2;   // 16 KB activation tile
constexpr uint32_t kWBytes = kWidth * kWidth * 2;      // 8 KB weight tile
constexpr uint32_t kIdesc = tc::idesc_f16(128, 64, false, false);     // X * W^T
constexpr uint32_t kIdescBwd = tc::idesc_f16(128, 64, false, true);   // G * W
constexpr uint32_t kIdescWgrad = tc::idesc_f16(128, 64, true, true);  // G^T * X (rows 64.. unused)

__device__ __forceinline__ uint32_t grid_hash(uint32_t x, uint32_t y, uint32_t z) {
  // Instant-NGP spatial hash, nrcEncoding.ts spatialHash3D:107-115 (x prime 1)
  return x ^ (y * 2654435761u) ^ (z * 805459861u);
}

__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float2 unpack_h2(uint32_t u) {
  const __half2 h = *reinterpret_cast<const __half2*>(&u);
  return __half22float2(h);
}

// normalised position in [0,1]^3 (normalizeToAabb, nrcEncoding.ts:166-178)
__device__ __forceinline__ float3 normalise(const View& v, float px, float py, float pz) {
  return make_float3(fminf(1.0f, fmaxf(0.0f, (px - v.aabb_min[0]) * v.aabb_inv[0])),
                     fminf(1.0f, fmaxf(0.0f, (py - v.aabb_min[1]) * v.aabb_inv[1])),
                     fminf(1.0f, fmaxf(0.0f, (pz - v.aabb_min[2]) * v.aabb_inv[2])));
}

// Real spherical harmonics of degree 4 (bands 0..3, 16 values) of unit d.
__device__ __forceinline__ void sh4(float x, float y, float z, float (&s)[16]) {
  const float xx = x * x, yy = y * y, zz = z * z, xy = x * y, yz = y * z, xz = x * z;
  s[0] = 0.28209479177387814f;
  s[1] = -0.48860251190291987f * y;
  s[2] = 0.48860251190291987f * z;
  s[3] = -0.48860251190291987f * x;
  s[4] = 1.0925484305920792f * xy;
  s[5] = -1.0925484305920792f * yz;
  s[6] = 0.94617469575755997f * zz - 0.31539156525251999f;
  s[7] = -1.0925484305920792f * xz;
  s[8] = 0.54627421529603959f * (xx - yy);
  s[9] = 0.59004358992664352f * y * (3.0f * xx - yy) * -1.0f;
  s[10] = 2.8906114426405538f * xy * z;
  s[11] = 0.45704579946446572f * y * (1.0f - 5.0f * zz);
  s[12] = 0.3731763325901154f * z * (5.0f * zz - 3.0f);
  s[13] = 0.45704579946446572f * x * (1.0f - 5.0f * zz);
  s[14] = 1.4453057213202769f * z * (xx - yy);
  s[15] = 0.59004358992664352f * x * (3.0f * yy - xx);
}

// Position of a point within level l's grid: cell corner and fractions.
struct Cell {
  uint32_t x, y, z;
  float fx, fy, fz;
};
__device__ __forceinline__ Cell grid_cell(const View& v, int l, float3 n01) {
  const float N = v.res[l];
  const float px = n01.x * N, py = n01.y * N, pz = n01.z * N;
  const float x0 = floorf(px), y0 = floorf(py), z0 = floorf(pz);
  return {(uint32_t)(int)x0, (uint32_t)(int)y0, (uint32_t)(int)z0, px - x0, py - y0, pz - z0};
}

// A lane pair's two points.  The pair gathers (and scatters) for both together,
// the even lane the corners at x, the odd lane those at x + 1: the hash's x prime
// is 1, so the two rows differ in a few low bits, and 31 of 32 pairs fall into one
// 128-byte line (7 of 8 into one 32-byte sector), which a warp's one access then
// touches once instead of twice.  1,048,576 queries of the 16 x 2^19 grid, bound by
// the L1's lookups: 383 -> 326 us (312 with the layer inputs in TMEM, k_nrc_infer).
struct PointPair {
  float3 even, odd;  // the even and the odd lane's point
  bool is_odd;       // this lane's place
};
__device__ __forceinline__ PointPair pair_points(float3 n01) {
  const float3 o = make_float3(__shfl_xor_sync(0xFFFFFFFFu, n01.x, 1), __shfl_xor_sync(0xFFFFFFFFu, n01.y, 1),
                               __shfl_xor_sync(0xFFFFFFFFu, n01.z, 1));
  const bool odd = threadIdx.x & 1u;
  return {odd ? o : n01, odd ? n01 : o, odd};
}

// The two features of level l at this lane's point: trilinear blend of the 8
// corner rows.  Called by whole warps.
__device__ __forceinline__ uint32_t encode_level(const View& v, int l, const PointPair& q) {
  float f0 = 0.0f, f1 = 0.0f;
  if (l < v.levels) {
    const Cell ce = grid_cell(v, l, q.even), co = grid_cell(v, l, q.odd);
    const float fx = q.is_odd ? co.fx : ce.fx, fy = q.is_odd ? co.fy : ce.fy, fz = q.is_odd ? co.fz : ce.fz;
    const uint32_t* tab = reinterpret_cast<const uint32_t*>(v.table16 + (size_t)l * (v.table_mask + 1u));
    const uint32_t h = q.is_odd ? 1u : 0u;
    uint32_t e0[4], e1[4];  // rows at x and x + 1 of this lane's point
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t cy = k & 1, cz = k >> 1;
      const uint32_t e = __ldg(tab + (grid_hash(ce.x + h, ce.y + cy, ce.z + cz) & v.table_mask));
      const uint32_t o = __ldg(tab + (grid_hash(co.x + h, co.y + cy, co.z + cz) & v.table_mask));
      const uint32_t theirs = __shfl_xor_sync(0xFFFFFFFFu, q.is_odd ? e : o, 1);
      e0[k] = q.is_odd ? theirs : e;
      e1[k] = q.is_odd ? o : theirs;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t cy = k & 1, cz = k >> 1;
      const float w0 = (1.0f - fx) * (cy ? fy : 1.0f - fy) * (cz ? fz : 1.0f - fz);
      const float w1 = fx * (cy ? fy : 1.0f - fy) * (cz ? fz : 1.0f - fz);
      const float2 a = unpack_h2(e0[k]), b = unpack_h2(e1[k]);
      f0 = fmaf(w0, a.x, f0);
      f1 = fmaf(w0, a.y, f1);
      f0 = fmaf(w1, b.x, f0);
      f1 = fmaf(w1, b.y, f1);
    }
  }
  return pack_h2(f0, f1);
}

// Encodes one record (4 float4) into 64 fp16 inputs packed as 32 half2 words.
__device__ __forceinline__ void encode(const View& v, float4 a, float4 b, float4 c, float4 d, uint32_t (&p)[32]) {
  const PointPair q = pair_points(normalise(v, a.x, a.y, a.z));
  // all levels unrolled: the 8 x levels table gathers are independent and in flight together
#pragma unroll
  for (int l = 0; l < kMaxLevels; ++l) p[l] = encode_level(v, l, q);
  float s[16];
  sh4(a.w, b.x, b.y, s);
#pragma unroll
  for (int k = 0; k < 8; ++k) p[16 + k] = pack_h2(s[2 * k], s[2 * k + 1]);
  // normal (b.z, b.w, c.x), roughness c.y, diffuse (c.z, c.w, d.x), specular (d.y, d.z, d.w), 1
  p[24] = pack_h2(b.z, b.w);
  p[25] = pack_h2(c.x, c.y);
  p[26] = pack_h2(c.z, c.w);
  p[27] = pack_h2(d.x, d.y);
  p[28] = pack_h2(d.z, d.w);
  p[29] = pack_h2(1.0f, 0.0f);
  p[30] = 0u;
  p[31] = 0u;
}

// Scatter of the input gradient (g0, g1) of level l's two features (already
// scaled) into the f32 table gradient with the trilinear weights, the pair for
// its two points in turn as in the gather: the L2 takes the neighbouring rows of
// one access as one operation per sector.  Called by whole warps; zero gradients
// add nothing.
__device__ __forceinline__ void scatter_level(const View& v, int l, const PointPair& q, float g0, float g1) {
  const float p0 = __shfl_xor_sync(0xFFFFFFFFu, g0, 1), p1 = __shfl_xor_sync(0xFFFFFFFFu, g1, 1);
  if (l >= v.levels) return;
  const uint32_t h = q.is_odd ? 1u : 0u;
  float2* gt = v.grad_table + (size_t)l * (v.table_mask + 1u);
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const float a0 = (s == 1) == q.is_odd ? g0 : p0, a1 = (s == 1) == q.is_odd ? g1 : p1;
    if (a0 == 0.0f && a1 == 0.0f) continue;
    const Cell c = grid_cell(v, l, s ? q.odd : q.even);
    const float wx = h ? c.fx : 1.0f - c.fx;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t cy = k & 1, cz = k >> 1;
      const float w = wx * (cy ? c.fy : 1.0f - c.fy) * (cz ? c.fz : 1.0f - c.fz);
      atomicAdd(gt + (grid_hash(c.x + h, c.y + cy, c.z + cz) & v.table_mask), make_float2(w * a0, w * a1));
    }
  }
}

// The dynamic shared memory from its first 1024-byte boundary on.
__device__ __forceinline__ uint8_t* align1024(uint8_t* p) {
  const uint32_t s = tc::smem_u32(p);
  return p + (((s + 1023u) & ~1023u) - s);
}

// Loads the six fp16 weight tiles (row-major [out][in]) into swizzled tiles.
__device__ __forceinline__ void load_weights(const View& v, uint8_t* w) {
  for (uint32_t q = threadIdx.x; q < (uint32_t)(kLayers * kWidth * 8); q += blockDim.x) {
    const uint32_t l = q / (kWidth * 8), r = (q / 8) % kWidth, j = q % 8;
    const uint4 val = __ldg(reinterpret_cast<const uint4*>(v.w16 + (size_t)l * kWidth * kWidth + r * kWidth) + j);
    *reinterpret_cast<uint4*>(w + l * kWBytes + tc::sw128_offset(r, 8 * j)) = val;
  }
}

// Issue one 128x64x64 product (four K=16 steps) and commit to the barrier.
__device__ __forceinline__ void issue_fwd(uint32_t tmem_d, uint32_t a_tile, uint32_t w_tile) {
  tc::fence_after_sync();
#pragma unroll
  for (uint32_t kk = 0; kk < 4; ++kk) tc::mma_f16(tmem_d, tc::desc_k(a_tile, kk), tc::desc_k(w_tile, kk), kIdesc, kk);
}

// 64 fp32 accumulator columns of this thread's row (its TMEM lane)
__device__ __forceinline__ void load_acc64(uint32_t taddr, uint32_t (&v)[64]) {
  uint32_t (&a)[16] = *reinterpret_cast<uint32_t(*)[16]>(&v[0]);
  uint32_t (&b)[16] = *reinterpret_cast<uint32_t(*)[16]>(&v[16]);
  uint32_t (&c)[16] = *reinterpret_cast<uint32_t(*)[16]>(&v[32]);
  uint32_t (&d)[16] = *reinterpret_cast<uint32_t(*)[16]>(&v[48]);
  tc::tmem_ld16(taddr, a);
  tc::tmem_ld16(taddr + 16, b);
  tc::tmem_ld16(taddr + 32, c);
  tc::tmem_ld16(taddr + 48, d);
  tc::tmem_wait_ld();
}

// On a timed-out wait: flag, give the issued MMAs a bounded chance to finish.
__device__ void fail_and_drain(const View& v, uint64_t* bar, uint32_t phase) {
  if (threadIdx.x == 0) {
    atomicExch(v.error, 1);
    tc::mbar_wait(bar, phase, kWaitCycles);
  }
  __syncthreads();
}

// ---------------------------------------------------------------- inference
// Named barrier of warpgroup g (ids 1..T; 0 is __syncthreads): the 128 threads
// of one tile synchronise without waiting for the CTA's other tiles.
__device__ __forceinline__ void group_sync(uint32_t id) {
  asm volatile("barrier.cta.sync %0, 128;" ::"r"(id) : "memory");
}
__device__ __forceinline__ bool group_and(uint32_t id, bool p) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred a, b;\n\tsetp.ne.u32 a, %1, 0;\n\tbarrier.cta.red.and.pred b, %2, 128, a;\n\t"
      "selp.u32 %0, 1, 0, b;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)p), "r"(id)
      : "memory");
  return r != 0;
}

// TMEM columns of T tiles: 64 of accumulators and 32 of layer input each, rounded
// up to a power of two
__host__ __device__ constexpr uint32_t infer_cols(int t) { return t == 1 ? 128u : (t == 2 ? 256u : 512u); }

// T tiles of 128 queries in flight per CTA, one per warpgroup (the MLP tile
// knob): the warpgroups share the CTA's weight tiles and TMEM allocation (96
// columns each: 64 of accumulators, 32 of layer input) and run independently --
// each encodes its tile (16 levels x 8 table gathers per query), issues its own
// MMA chain from its first thread and waits on its own mbarrier -- so one tile's
// gathers overlap another's MMAs.
// The layer inputs are the MMAs' A operands in TMEM, written by the thread that owns
// the row: shared memory holds the weights alone (50 KB instead of 66 to 114), and
// what it gives up is L1 for the gathers that bound the kernel: 1,048,576 queries of
// the 16 x 2^19 grid 326 -> 313 us.  (The coarsest level as a dense grid in shared
// memory, beside 114 KB: 328; the two coarsest: 535, the L1 gone.)
template <int T>
__global__ void __launch_bounds__(128 * T, T == 1 ? 3 : (T == 2 ? 2 : 1))
    k_nrc_infer(View v, const float4* __restrict__ recs, uint32_t stride, const uint32_t* __restrict__ n_dev,
                uint32_t n_host, float* __restrict__ rgb, float4* __restrict__ radiance) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = align1024(smem_raw);
  uint8_t* wt = base;
  const uint32_t tid = threadIdx.x & 127u, warp = tid >> 5, g = threadIdx.x >> 7, gid = g + 1;
  uint64_t* bar = reinterpret_cast<uint64_t*>(base + kLayers * kWBytes) + g;
  uint32_t* slot = reinterpret_cast<uint32_t*>(reinterpret_cast<uint64_t*>(base + kLayers * kWBytes) + T);
  constexpr uint32_t kCols = infer_cols(T);
  const uint32_t n = n_dev ? *n_dev : n_host;
  if ((uint32_t)blockIdx.x * T * kTile >= n) return;  // uniform per CTA: no tile, no TMEM
  if (threadIdx.x < 32) {
    tc::tmem_alloc(slot, kCols);
    tc::tmem_relinquish();
  }
  if (tid == 0) {
    tc::mbar_init(bar, 1);
    tc::fence_mbar_init();
  }
  load_weights(v, wt);
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *slot + 64u * g;
  const uint32_t lane_addr = tmem + ((warp * 32u) << 16);
  // this warpgroup's layer input, in TMEM (row = lane, 64 fp16 in 32 columns): each
  // layer's MMA has finished reading it before the epilogue writes the next one over it
  const uint32_t act = *slot + 64u * T + 32u * g, act_lane = act + ((warp * 32u) << 16);
  const uint32_t w_s = tc::smem_u32(wt);
  uint32_t phase = 0;
  bool failed = false;
  for (uint32_t tile = blockIdx.x * T + g; tile * kTile < n && !failed; tile += gridDim.x * T) {
    const uint32_t i = tile * kTile + tid;
    const bool valid = i < n;
    uint32_t p[32];
    const float4* r = recs + (size_t)(valid ? i : 0) * stride;
    encode(v, __ldg(r), __ldg(r + 1), __ldg(r + 2), __ldg(r + 3), p);
    tc::tmem_st32(act_lane, p);
    tc::tmem_wait_st();
    tc::fence_before_sync();
    group_sync(gid);
    for (int l = 0; l < kLayers; ++l) {
      if (tid == 0) {
        tc::fence_after_sync();
#pragma unroll
        for (uint32_t kk = 0; kk < 4; ++kk)
          tc::mma_f16_ta(tmem, act + 8u * kk, tc::desc_k(w_s + l * kWBytes, kk), kIdesc, kk);
        tc::mma_commit(bar);
      }
      // thread-uniform bounded wait (per warpgroup); on failure `phase` keeps the pending parity
      if (!group_and(gid, tc::mbar_wait(bar, phase, v.wait_cycles))) { failed = true; break; }
      phase ^= 1u;
      tc::fence_after_sync();
      if (l + 1 < kLayers) {
        uint32_t acc[64];
        load_acc64(lane_addr, acc);
#pragma unroll
        for (int k = 0; k < 32; ++k)
          p[k] = pack_h2(fmaxf(__uint_as_float(acc[2 * k]), 0.0f), fmaxf(__uint_as_float(acc[2 * k + 1]), 0.0f));
        tc::tmem_st32(act_lane, p);
        tc::tmem_wait_st();
        tc::fence_before_sync();
        group_sync(gid);
      } else {
        uint32_t o[16];
        tc::tmem_ld16(lane_addr, o);
        tc::tmem_wait_ld();
        tc::fence_before_sync();
        if (valid) {
          const float r0 = __uint_as_float(o[0]), r1 = __uint_as_float(o[1]), r2 = __uint_as_float(o[2]);
          if (radiance) {
            const float4 e = __ldg(recs + (size_t)i * stride + 4);  // (path bits, throughput rgb)
            const uint32_t path = __float_as_uint(e.x);
            float4 acc = radiance[path];
            acc.x += e.y * fmaxf(r0, 0.0f);
            acc.y += e.z * fmaxf(r1, 0.0f);
            acc.z += e.w * fmaxf(r2, 0.0f);
            radiance[path] = acc;
          } else {
            rgb[3 * (size_t)i] = r0;
            rgb[3 * (size_t)i + 1] = r1;
            rgb[3 * (size_t)i + 2] = r2;
          }
        }
      }
    }
  }
  if (failed) {
    // flag, give the issued MMAs a bounded chance to finish
    if (tid == 0) {
      atomicExch(v.error, 1);
      tc::mbar_wait(bar, phase, kWaitCycles);
    }
    group_sync(gid);
  }
  __syncthreads();
  if (threadIdx.x < 32) tc::tmem_dealloc(*slot, kCols);
}

// ---------------------------------------------------------------- training
// Relative L2 on luminance (fusedMlp.wgsl.ts:62-110): per-sample gradient
// 2/3 (p - t) / (lum(p)^2 + 1e-2) with the stop-gradient luminance
// lum = clamp(sum w_c p_c / max|p|, -1, 1) * max|p|; the 1/N of the mean is
// applied in fp32 when the accumulated gradients leave TMEM (loss scaling by
// N keeps the fp16 deltas in range); deltas clamp at +-65504, NaN -> 0.
__device__ __forceinline__ float rel_l2_lum(float p0, float p1, float p2) {
  const float s = fmaxf(fabsf(p0), fmaxf(fabsf(p1), fabsf(p2)));
  if (!(s > 0.0f)) return 0.0f;
  const float nl = 0.299f * (p0 / s) + 0.587f * (p1 / s) + 0.114f * (p2 / s);
  return fminf(1.0f, fmaxf(-1.0f, nl)) * s;
}

// 16-byte chunk `j` of row r of a tile
__device__ __forceinline__ uint4* chunk_at(uint8_t* tile, uint32_t r, uint32_t j) {
  return reinterpret_cast<uint4*>(tile + tc::sw128_offset(r, 8 * j));
}

// One tile of 128 samples at a time per CTA (one CTA per SM: its six stored
// activation tiles and 384 TMEM columns of weight gradients leave no room for
// another), four threads per sample, in four warpgroups that divide every phase
// by columns: warpgroup q encodes and scatters levels 4q .. 4q + 3 (input
// columns 8q .. 8q + 7) and one more 8-column block of the features, and takes
// 16 of the 64 accumulator columns in the epilogues (warps w and w + 4 read the
// same TMEM lanes).  Everything here waits on latency -- table gathers, the
// chain of twelve dependent products and epilogues, the gradient atomics -- so
// what the four-fold warps buy is overlap.
// Measured per 65,536-sample step (2^15 / 2^19 tables, optimiser included): one
// warpgroup 165 / 274 us; four 160 / 265; 16-byte atomics for the weight
// gradients (3.6 M single ones before) and for table rows that share 16 bytes
// 123 / 231; one barrier a layer 120 / 228; lane pairs for gathers and scatters
// instead of the 16-byte table atomics 106 / 211.  The chain of products alone
// is 46 us of that, the table atomics were 34 and the gathers 22 before the pairs.
constexpr int kTrainGroups = 4;
__global__ void __launch_bounds__(128 * kTrainGroups, 1)
    k_nrc_train(View v, const float4* __restrict__ samples, uint32_t n) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = align1024(smem_raw);
  uint8_t* wt = base;                             // 6 x 8 KB
  uint8_t* G = base + kLayers * kWBytes;          // gradient tile
  uint8_t* X = G + kTileBytes;                    // X[0] = encoded input, X[l] = H_l (l = 1..5)
  uint64_t* bar = reinterpret_cast<uint64_t*>(X + kLayers * kTileBytes);
  uint32_t* slot = reinterpret_cast<uint32_t*>(bar + 1);
  const uint32_t row = threadIdx.x & 127u, part = threadIdx.x >> 7, warp = threadIdx.x >> 5;
  if ((uint32_t)blockIdx.x * kTile >= n) return;
  if (warp == 0) {
    tc::tmem_alloc(slot, 512);
    tc::tmem_relinquish();
  }
  if (threadIdx.x == 0) {
    tc::mbar_init(bar, 1);
    tc::fence_mbar_init();
  }
  load_weights(v, wt);
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *slot;
  const uint32_t lane_addr = tmem + (((warp & 3u) * 32u) << 16);
  const uint32_t w_s = tc::smem_u32(wt), g_s = tc::smem_u32(G), x_s = tc::smem_u32(X);
  const float inv_n = 1.0f / (float)n;
  uint32_t phase = 0;
  bool failed = false;
  uint32_t tiles = 0;
  float loss = 0.0f;
  for (uint32_t tile = blockIdx.x; tile * kTile < n && !failed; tile += gridDim.x, ++tiles) {
    const uint32_t i = tile * kTile + row;
    const bool valid = i < n;
    const float4* r = samples + (size_t)(valid ? i : 0) * 5;
    const float4 ra = __ldg(r);
    const PointPair point = pair_points(normalise(v, ra.x, ra.y, ra.z));
    {
      uint32_t p[4];
#pragma unroll
      for (int l = 0; l < 4; ++l) p[l] = encode_level(v, 4 * (int)part + l, point);
      *chunk_at(X, row, part) = make_uint4(p[0], p[1], p[2], p[3]);
      // columns 32 + 8 part: the spherical harmonics' halves, then the surface features
      if (part < 2) {
        const float4 rb = __ldg(r + 1);
        float sh[16];
        sh4(ra.w, rb.x, rb.y, sh);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          p[k] = part == 0 ? pack_h2(sh[2 * k], sh[2 * k + 1]) : pack_h2(sh[8 + 2 * k], sh[9 + 2 * k]);
      } else if (part == 2) {
        const float4 rb = __ldg(r + 1), rc = __ldg(r + 2), rd = __ldg(r + 3);
        p[0] = pack_h2(rb.z, rb.w);
        p[1] = pack_h2(rc.x, rc.y);
        p[2] = pack_h2(rc.z, rc.w);
        p[3] = pack_h2(rd.x, rd.y);
      } else {
        const float4 rd = __ldg(r + 3);
        p[0] = pack_h2(rd.z, rd.w);
        p[1] = pack_h2(1.0f, 0.0f);
        p[2] = p[3] = 0u;
      }
      *chunk_at(X, row, 4 + part) = make_uint4(p[0], p[1], p[2], p[3]);
    }
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    // ---- forward, keeping H_1..H_5.  One barrier a layer: it publishes the next
    // input and carries the verdict on the wait (a failed one's epilogue wrote
    // garbage to shared memory only)
    float pr[3] = {0.0f, 0.0f, 0.0f};
    for (int l = 0; l < kLayers; ++l) {
      if (threadIdx.x == 0) {
        issue_fwd(tmem, x_s + l * kTileBytes, w_s + l * kWBytes);
        tc::mma_commit(bar);
      }
      const bool ok = tc::mbar_wait(bar, phase, v.wait_cycles);
      tc::fence_after_sync();
      uint32_t o[16];
      if (l + 1 < kLayers) {
        tc::tmem_ld16(lane_addr + 16u * part, o);
        tc::tmem_wait_ld();
        uint32_t p[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
          p[k] = pack_h2(fmaxf(__uint_as_float(o[2 * k]), 0.0f), fmaxf(__uint_as_float(o[2 * k + 1]), 0.0f));
        uint8_t* H = X + (l + 1) * kTileBytes;
        *chunk_at(H, row, 2 * part) = make_uint4(p[0], p[1], p[2], p[3]);
        *chunk_at(H, row, 2 * part + 1) = make_uint4(p[4], p[5], p[6], p[7]);
        tc::fence_async_smem();
      } else if (part == 0) {
        tc::tmem_ld16(lane_addr, o);
        tc::tmem_wait_ld();
        pr[0] = __uint_as_float(o[0]);
        pr[1] = __uint_as_float(o[1]);
        pr[2] = __uint_as_float(o[2]);
      }
      tc::fence_before_sync();
      if (__syncthreads_or(!ok)) { failed = true; break; }  // `phase` keeps the pending parity
      phase ^= 1u;
    }
    if (failed) break;
    // ---- output gradient (one thread per sample; the others clear its row's other columns)
    if (part == 0) {
      float g[3] = {0.0f, 0.0f, 0.0f};
      const float4 tgt = __ldg(r + 4);
      const bool fin = isfinite(pr[0]) && isfinite(pr[1]) && isfinite(pr[2]);
      if (valid && fin && isfinite(tgt.x) && isfinite(tgt.y) && isfinite(tgt.z)) {
        const float t3[3] = {tgt.x, tgt.y, tgt.z};
        const float lum = fminf(fabsf(rel_l2_lum(pr[0], pr[1], pr[2])), 1e19f);
        const float den = lum * lum + 1e-2f;
        const float sc = 2.0f / 3.0f / den;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const float dlt = pr[c] - t3[c];
          float raw = dlt * sc;
          if (isnan(raw)) raw = 0.0f;
          g[c] = fminf(65504.0f, fmaxf(-65504.0f, raw));
          loss += dlt * dlt / den / 3.0f;
        }
      }
      if (valid && v.tile_stats && __float_as_uint(tgt.w) != 0u && fin) {
        // cache error estimate of the sample's screen tile (prediction vs target luminance)
        const uint32_t pix = __float_as_uint(tgt.w) - 1u;
        const uint32_t st = (pix / v.tile_width / v.tile_size) * v.tiles_x + (pix % v.tile_width) / v.tile_size;
        float* ts = v.tile_stats + 3 * (size_t)st;
        atomicAdd(ts, 0.2126f * fmaxf(pr[0], 0.0f) + 0.7152f * fmaxf(pr[1], 0.0f) + 0.0722f * fmaxf(pr[2], 0.0f));
        atomicAdd(ts + 1, 0.2126f * tgt.x + 0.7152f * tgt.y + 0.0722f * tgt.z);
        atomicAdd(ts + 2, 1.0f);
      }
      *chunk_at(G, row, 0) = make_uint4(pack_h2(g[0], g[1]), pack_h2(g[2], 0.0f), 0u, 0u);
    } else {
      *chunk_at(G, row, 2 * part) = make_uint4(0u, 0u, 0u, 0u);
    }
    *chunk_at(G, row, 2 * part + 1) = make_uint4(0u, 0u, 0u, 0u);
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    // ---- backward: layer 5 (output) down to 0
    for (int l = kLayers - 1; l >= 0; --l) {
      if (threadIdx.x == 0) {
        tc::fence_after_sync();
        const uint32_t x_in = x_s + l * kTileBytes;  // this layer's input
        const uint32_t dw = tmem + 64u + 64u * (uint32_t)l;
#pragma unroll
        for (uint32_t kk = 0; kk < 4; ++kk)  // K = 64 outputs of this layer
          tc::mma_f16(tmem, tc::desc_k(g_s, kk), tc::desc_mn(w_s + l * kWBytes, kk, kWBytes), kIdescBwd, kk);
#pragma unroll
        for (uint32_t kk = 0; kk < 8; ++kk)  // K = 128 samples
          tc::mma_f16(dw, tc::desc_mn(g_s, kk, kTileBytes), tc::desc_mn(x_in, kk, kTileBytes), kIdescWgrad,
                      (tiles > 0 || kk > 0) ? 1u : 0u);
        tc::mma_commit(bar);
      }
      const bool ok = tc::mbar_wait(bar, phase, v.wait_cycles);
      tc::fence_after_sync();
      uint32_t acc[16];  // dX_l: this part's 16 columns; of layer 0 the 16 that hold its four levels' 8
      tc::tmem_ld16(lane_addr + (l > 0 ? 16u * part : 16u * (part >> 1)), acc);
      tc::tmem_wait_ld();
      tc::fence_before_sync();
      if (l > 0) {
        // G_{l-1} = dH_l * (H_l > 0)
        uint8_t* H = X + l * kTileBytes;
        const uint4 ha = *chunk_at(H, row, 2 * part), hb = *chunk_at(H, row, 2 * part + 1);
        const uint32_t h[8] = {ha.x, ha.y, ha.z, ha.w, hb.x, hb.y, hb.z, hb.w};
        uint32_t p[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float2 hv = unpack_h2(h[k]);
          const float a0 = hv.x > 0.0f ? __uint_as_float(acc[2 * k]) : 0.0f;
          const float a1 = hv.y > 0.0f ? __uint_as_float(acc[2 * k + 1]) : 0.0f;
          p[k] = pack_h2(fminf(65504.0f, fmaxf(-65504.0f, a0)), fminf(65504.0f, fmaxf(-65504.0f, a1)));
        }
        *chunk_at(G, row, 2 * part) = make_uint4(p[0], p[1], p[2], p[3]);
        *chunk_at(G, row, 2 * part + 1) = make_uint4(p[4], p[5], p[6], p[7]);
        tc::fence_async_smem();
      }
      if (__syncthreads_or(!ok)) { failed = true; break; }
      phase ^= 1u;
      if (l == 0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float g0 = __uint_as_float((part & 1u) ? acc[8 + 2 * q] : acc[2 * q]) * inv_n;
          const float g1 = __uint_as_float((part & 1u) ? acc[9 + 2 * q] : acc[2 * q + 1]) * inv_n;
          scatter_level(v, 4 * (int)part + q, point, valid ? g0 : 0.0f, valid ? g1 : 0.0f);
        }
      }
    }
  }
  if (failed) {
    fail_and_drain(v, bar, phase);
  } else if (tiles > 0 && (warp & 3u) < 2u) {
    // weight gradients: rows 0..63 of each dW accumulator (TMEM lanes 0..63), 16 columns per part
    tc::fence_after_sync();
    for (int l = 0; l < kLayers; ++l) {
      uint32_t acc[16];
      tc::tmem_ld16(lane_addr + 64u + 64u * (uint32_t)l + 16u * part, acc);
      tc::tmem_wait_ld();
      float4* gw = reinterpret_cast<float4*>(v.grad_w + (size_t)l * kWidth * kWidth + (size_t)row * kWidth + 16u * part);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        atomicAdd(gw + k, make_float4(__uint_as_float(acc[4 * k]) * inv_n, __uint_as_float(acc[4 * k + 1]) * inv_n,
                                      __uint_as_float(acc[4 * k + 2]) * inv_n, __uint_as_float(acc[4 * k + 3]) * inv_n));
    }
  }
  // loss: warp reduce then one atomic per warp (part 0 holds it)
  if (part == 0) {
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xFFFFFFFFu, loss, o);
    if ((threadIdx.x & 31u) == 0 && v.loss) atomicAdd(v.loss, loss * inv_n);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, 512);
}

// ---------------------------------------------------------------- Adam
__device__ __forceinline__ bool fin(float x) { return x == x && fabsf(x) <= 3.402823e38f; }

// ibc1 / ibc2: 1 / (1 - beta^t), rounded once on the host (a product per value instead of two divisions)
__device__ __forceinline__ float adam_one(float cur, float& m, float& vv, float g, float lr, float b1, float b2,
                                          float eps, float ibc1, float ibc2, int* diag) {
  if (!fin(cur) || !fin(m) || !fin(vv) || vv < 0.0f) {
    m = 0.0f;
    vv = 0.0f;
    if (diag) atomicAdd(diag, 1);
    return fin(cur) ? cur : 0.0f;
  }
  if (!fin(g)) {
    if (diag) atomicAdd(diag, 1);
    return cur;
  }
  const float mi = b1 * m + (1.0f - b1) * g;
  const float vi = b2 * vv + (1.0f - b2) * g * g;
  const float mh = mi * ibc1, vh = vi * ibc2;
  const float up = cur - lr * mh / (sqrtf(vh) + eps);
  if (!fin(up) || !fin(mi) || !fin(vi)) {
    if (diag) atomicAdd(diag, 1);
    return cur;
  }
  m = mi;
  vv = vi;
  return fminf(65504.0f, fmaxf(-65504.0f, up));
}

// One parameter array as pairs: f32 master, moments and gradient, fp16 copy.
struct AdamPairs {
  float2 *master, *m, *v, *grad;
  __half2* out16;
  size_t pairs;
  float lr;
};

__device__ __forceinline__ void adam_pairs(const AdamPairs& a, size_t first, size_t step, float b1, float b2, float eps,
                                           float ibc1, float ibc2, int* diag) {
  float2 *__restrict__ master = a.master, *__restrict__ pm = a.m, *__restrict__ pv = a.v, *__restrict__ grad = a.grad;
  __half2* __restrict__ out16 = a.out16;
  for (size_t i = first; i < a.pairs; i += step) {
    float2 w = master[i], mm = pm[i], vv = pv[i];
    const float2 g = grad[i];
    w.x = adam_one(w.x, mm.x, vv.x, g.x, a.lr, b1, b2, eps, ibc1, ibc2, diag);
    w.y = adam_one(w.y, mm.y, vv.y, g.y, a.lr, b1, b2, eps, ibc1, ibc2, diag);
    master[i] = w;
    pm[i] = mm;
    pv[i] = vv;
    grad[i] = make_float2(0.0f, 0.0f);
    out16[i] = __floats2half2_rn(w.x, w.y);
  }
}

// Adam over the table and, in the last `weight_ctas` CTAs, the weights (a launch
// of their own cost 4 us of every step); clears the gradients and writes the
// fp16 copies in the same pass.  Bound by memory: 76 bytes a pair.
__global__ void __launch_bounds__(256) k_nrc_adam(AdamPairs table, AdamPairs weights, unsigned weight_ctas, float b1,
                                                  float b2, float eps, float ibc1, float ibc2, int* diag) {
  const unsigned table_ctas = gridDim.x - weight_ctas;
  if (blockIdx.x < table_ctas)
    adam_pairs(table, (size_t)blockIdx.x * 256 + threadIdx.x, (size_t)table_ctas * 256, b1, b2, eps, ibc1, ibc2, diag);
  else
    adam_pairs(weights, (size_t)(blockIdx.x - table_ctas) * 256 + threadIdx.x, (size_t)weight_ctas * 256, b1, b2, eps,
               ibc1, ibc2, diag);
}

constexpr size_t kInferSmem = kLayers * kWBytes + 64 + 1024;
constexpr size_t kTrainSmem = kLayers * kWBytes + (1 + kLayers) * kTileBytes + 64 + 1024;

int sm_count() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms > 0 ? sms : 1;
}

}  // namespace

void level_resolutions(const Config& c, float* out) {
  for (int l = 0; l < kMaxLevels; ++l) out[l] = (float)std::floor((double)c.base_resolution * std::pow((double)c.growth, l));
}

template <int T>
void launch_infer_t(const View& v, const float4* records, uint32_t rec_stride_f4, const uint32_t* n_dev, uint32_t n,
                    float* rgb_out, float4* radiance, cudaStream_t s) {
  static PerDevice<int> resident;
  const int per_sm = resident.get(current_device(), [] {
    int ctas = 0;
    VT_CUDA(cudaFuncSetAttribute(k_nrc_infer<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kInferSmem));
    VT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, k_nrc_infer<T>, 128 * T, kInferSmem));
    return std::max(1, std::min(ctas, 512 / (int)infer_cols(T)));  // TMEM: 512 columns per SM
  });
  const uint32_t tiles = (n + kTile - 1) / kTile;
  const uint32_t ctas = (tiles + T - 1) / T;
  const uint32_t cap = (uint32_t)(per_sm * sm_count());
  k_nrc_infer<T><<<ctas < cap ? ctas : cap, 128 * T, kInferSmem, s>>>(v, records, rec_stride_f4, n_dev, n, rgb_out,
                                                                          radiance);
}

void launch_infer(const View& v, const float4* records, uint32_t rec_stride_f4, const uint32_t* n_dev, uint32_t n,
                  float* rgb_out, float4* radiance, int tiles_per_cta, cudaStream_t s) {
  if (n == 0) return;
  // a batch of fewer tiles than SMs x T gets fewer tiles per CTA instead of idle SMs
  // (1,000 to 18,944 queries: 31 -> 17 us; 40,000: 33 -> 24 us)
  const uint32_t tiles = (n + kTile - 1) / kTile, sms = (uint32_t)sm_count();
  tiles_per_cta = (int)std::min<uint32_t>((uint32_t)tiles_per_cta, (tiles + sms - 1) / sms);
  // tiles in flight per CTA: 1 to 4.  The registers and TMEM of four tiles fill an SM
  if (tiles_per_cta >= 4) launch_infer_t<4>(v, records, rec_stride_f4, n_dev, n, rgb_out, radiance, s);
  else if (tiles_per_cta == 3) launch_infer_t<3>(v, records, rec_stride_f4, n_dev, n, rgb_out, radiance, s);
  else if (tiles_per_cta == 2) launch_infer_t<2>(v, records, rec_stride_f4, n_dev, n, rgb_out, radiance, s);
  else launch_infer_t<1>(v, records, rec_stride_f4, n_dev, n, rgb_out, radiance, s);
}

void launch_train(const View& v, const float4* samples, uint32_t n, cudaStream_t s) {
  if (n == 0) return;
  static PerDevice<bool> opted_in;
  opted_in.get(current_device(), [] {
    VT_CUDA(cudaFuncSetAttribute(k_nrc_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrainSmem));
    return true;
  });
  const uint32_t tiles = (n + kTile - 1) / kTile;
  const uint32_t grid = tiles < (uint32_t)sm_count() ? tiles : (uint32_t)sm_count();
  k_nrc_train<<<grid, 128 * kTrainGroups, kTrainSmem, s>>>(v, samples, n);
}

void launch_adam(const AdamArrays& table, const AdamArrays& weights, float beta1, float beta2, float eps, float bc1,
                 float bc2, int* diag, cudaStream_t s) {
  auto pairs = [](const AdamArrays& a) {
    return AdamPairs{reinterpret_cast<float2*>(a.master), reinterpret_cast<float2*>(a.m),
                     reinterpret_cast<float2*>(a.v), reinterpret_cast<float2*>(a.grad),
                     reinterpret_cast<__half2*>(a.out16), a.count / 2, a.lr};
  };
  const size_t g = (table.count / 2 + 255) / 256;
  const unsigned table_ctas = (unsigned)(g < 148 * 16 ? g : 148 * 16), weight_ctas = 16;
  k_nrc_adam<<<table_ctas + weight_ctas, 256, 0, s>>>(pairs(table), pairs(weights), weight_ctas, beta1, beta2, eps,
                                                      1.0f / bc1, 1.0f / bc2, diag);
}

}  // namespace nrc
}  // namespace vt
