// Elementwise tails of a DiT block either side of the attention path (HBM-bound streams):
//
//   layernorm_affine_kernel   out = LayerNorm(x) * mul + add   -> 16 bit
//       the modulated input of the self-attention and of the FFN, LayerNorm(x) * (1 + scale) + shift,
//       and the affine LayerNorm in front of the cross-attention: one pass over the residual
//       stream instead of the reference's LayerNorm + float() + multiply + add kernels
//   gate_residual_kernel      x += y * gate                    (residual stream in place, 16-bit branch output)
//
// The residual stream is fp32 (Wan) or 16-bit (Flux).  Algorithmic bytes per element with an fp32
// stream: LayerNorm 4 read + 2 written; gated residual 4 + 2 read, 4 written.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "elementwise.cuh"

namespace chitu {

constexpr int kLnThreads = 256;
constexpr int kLnMaxVec = 8;  // float4 per thread: rows of up to 8192 channels

struct LayerNormParams {
  const void* x;         // [rows, C] residual stream: fp32, or 16-bit (x_dtype 0 bf16, 1 fp16, 2 fp32)
  int x_dtype;
  void* out;             // [rows, C] bf16 / fp16
  const float* mul;      // [B or 1, C] fp32, or nullptr (= 1)
  const float* add;      // [B or 1, C] fp32, or nullptr (= 0)
  long long mul_batch_stride, add_batch_stride;  // elements between batches (0: one vector for all)
  long long rows, rows_per_batch;
  int C;
  int add_one;           // multiply by (1 + mul) instead of mul
  int out_fp16;
  float eps;
};

// four consecutive stream elements as floats / back (dtype 0 bf16, 1 fp16, 2 fp32)
__device__ __forceinline__ float4 stream_ld4(const void* p, int dtype, size_t vec) {
  if (dtype == 2) return __ldcs(reinterpret_cast<const float4*>(p) + vec);
  const uint2 raw = __ldcs(reinterpret_cast<const uint2*>(p) + vec);
  float2 a, b;
  if (dtype == 0) {
    a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  } else {
    a = __half22float2(*reinterpret_cast<const __half2*>(&raw.x));
    b = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
  }
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void stream_st4(void* p, int dtype, size_t vec, float4 v) {
  if (dtype == 2) {
    reinterpret_cast<float4*>(p)[vec] = v;
    return;
  }
  uint2 o;
  if (dtype == 0) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    o.x = *reinterpret_cast<const uint32_t*>(&lo);
    o.y = *reinterpret_cast<const uint32_t*>(&hi);
  } else {
    const __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
    o.x = *reinterpret_cast<const uint32_t*>(&lo);
    o.y = *reinterpret_cast<const uint32_t*>(&hi);
  }
  reinterpret_cast<uint2*>(p)[vec] = o;
}

__device__ __forceinline__ float ln_block_sum(float v, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int warp = threadIdx.x >> 5;
  __syncthreads();  // red[] may still be read from the previous reduction
  if ((threadIdx.x & 31) == 0) red[warp] = v;
  __syncthreads();
  float s = 0.f;
#pragma unroll
  for (int w = 0; w < kLnThreads / 32; ++w) s += red[w];
  return s;
}

// One CTA per row at a time (grid-stride over rows); the row lives in registers between the two
// reductions (mean, then the centred sum of squares).
__global__ void __launch_bounds__(kLnThreads)
layernorm_affine_kernel(const LayerNormParams p) {
  __shared__ float red[kLnThreads / 32];
  const int n_vec = p.C >> 2;
  for (long long row = blockIdx.x; row < p.rows; row += gridDim.x) {
    const size_t row_vec0 = static_cast<size_t>(row) * n_vec;
    float4 v[kLnMaxVec];
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < kLnMaxVec; ++i) {
      const int idx = threadIdx.x + i * kLnThreads;
      if (idx < n_vec) {
        v[i] = stream_ld4(p.x, p.x_dtype, row_vec0 + idx);  // streamed once
        sum += (v[i].x + v[i].y) + (v[i].z + v[i].w);
      }
    }
    const float mean = ln_block_sum(sum, red) / static_cast<float>(p.C);
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < kLnMaxVec; ++i) {
      const int idx = threadIdx.x + i * kLnThreads;
      if (idx < n_vec) {
        v[i].x -= mean; v[i].y -= mean; v[i].z -= mean; v[i].w -= mean;
        sq += (v[i].x * v[i].x + v[i].y * v[i].y) + (v[i].z * v[i].z + v[i].w * v[i].w);
      }
    }
    const float rstd = rsqrtf(ln_block_sum(sq, red) / static_cast<float>(p.C) + p.eps);
    const long long b = row / p.rows_per_batch;
    const float4* mul = p.mul ? reinterpret_cast<const float4*>(p.mul + b * p.mul_batch_stride) : nullptr;
    const float4* add = p.add ? reinterpret_cast<const float4*>(p.add + b * p.add_batch_stride) : nullptr;
    uint2* dst = reinterpret_cast<uint2*>(static_cast<uint16_t*>(p.out) + row * p.C);
    const float one = p.add_one ? 1.f : 0.f;
#pragma unroll
    for (int i = 0; i < kLnMaxVec; ++i) {
      const int idx = threadIdx.x + i * kLnThreads;
      if (idx < n_vec) {
        float4 m = mul ? __ldg(mul + idx) : make_float4(1.f, 1.f, 1.f, 1.f);
        const float4 a = add ? __ldg(add + idx) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (mul) { m.x += one; m.y += one; m.z += one; m.w += one; }
        const float r0 = fmaf(v[i].x * rstd, m.x, a.x), r1 = fmaf(v[i].y * rstd, m.y, a.y);
        const float r2 = fmaf(v[i].z * rstd, m.z, a.z), r3 = fmaf(v[i].w * rstd, m.w, a.w);
        uint2 o;
        if (p.out_fp16) {
          const __half2 lo = __floats2half2_rn(r0, r1), hi = __floats2half2_rn(r2, r3);
          o.x = *reinterpret_cast<const uint32_t*>(&lo);
          o.y = *reinterpret_cast<const uint32_t*>(&hi);
        } else {
          const __nv_bfloat162 lo = __floats2bfloat162_rn(r0, r1), hi = __floats2bfloat162_rn(r2, r3);
          o.x = *reinterpret_cast<const uint32_t*>(&lo);
          o.y = *reinterpret_cast<const uint32_t*>(&hi);
        }
        dst[idx] = o;
      }
    }
  }
}

template <int kXDtype>
__device__ __forceinline__ void ln_unpack(const uint4 raw, float (&f)[8]) {
  // 16 bytes of the stream: 8 values when 16-bit, 4 when fp32 (f[4..7] unused)
  if constexpr (kXDtype == 2) {
    f[0] = __uint_as_float(raw.x); f[1] = __uint_as_float(raw.y);
    f[2] = __uint_as_float(raw.z); f[3] = __uint_as_float(raw.w);
    f[4] = f[5] = f[6] = f[7] = 0.f;
  } else {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if constexpr (kXDtype == 0) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
      } else {
        const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
        f[2 * i] = h.x;
        f[2 * i + 1] = h.y;
      }
    }
  }
}

// 16-bit pairs of the output type
__device__ __forceinline__ uint32_t ln_pack(float lo, float hi, int fp16) {
  if (fp16) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// Warp-per-row form for rows of at most 8 KiB: the row sits in registers as raw 16-byte vectors (up to 16
// per lane, all loads in flight at once), the two reductions are warp shuffles, and nothing waits at a block
// barrier.  Lane l owns vectors l, l + 32, ...  Bound by the modulation vectors, which every row loads anew from
// cache (four times the bytes of a 16-bit stream), so it serves the shapes that have few of them per row or too few rows
// per batch for the column form below (the dispatch states where, with both sides' times).
constexpr int kLnWarpMaxVec = 16;

template <int kXDtype>
__global__ void __launch_bounds__(256) layernorm_affine_warp_kernel(const LayerNormParams p) {
  constexpr int kPer = kXDtype == 2 ? 4 : 8;  // channels per 16-byte vector
  const int lane = threadIdx.x & 31;
  const int n_vec = p.C / kPer;               // vectors per row (a multiple of 32: checked by the host)
  const int per_lane = n_vec >> 5;
  const long long warps = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  const float inv_c = 1.0f / static_cast<float>(p.C);
  const float one = p.add_one ? 1.f : 0.f;
  for (long long row = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); row < p.rows;
       row += warps) {
    const uint4* src = reinterpret_cast<const uint4*>(p.x) + static_cast<size_t>(row) * n_vec;
    uint4 raw[kLnWarpMaxVec];
#pragma unroll
    for (int i = 0; i < kLnWarpMaxVec; ++i)
      if (i < per_lane) raw[i] = __ldcs(src + lane + i * 32);
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < kLnWarpMaxVec; ++i)
      if (i < per_lane) {
        float f[8];
        ln_unpack<kXDtype>(raw[i], f);
#pragma unroll
        for (int e = 0; e < kPer; ++e) sum += f[e];
      }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float mean = sum * inv_c;
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < kLnWarpMaxVec; ++i)
      if (i < per_lane) {
        float f[8];
        ln_unpack<kXDtype>(raw[i], f);
#pragma unroll
        for (int e = 0; e < kPer; ++e) sq = fmaf(f[e] - mean, f[e] - mean, sq);
      }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    const float rstd = rsqrtf(sq * inv_c + p.eps);
    const long long b = row / p.rows_per_batch;
    const float* mul = p.mul ? p.mul + b * p.mul_batch_stride : nullptr;
    const float* add = p.add ? p.add + b * p.add_batch_stride : nullptr;
    uint16_t* dst = static_cast<uint16_t*>(p.out) + static_cast<size_t>(row) * p.C;
#pragma unroll
    for (int i = 0; i < kLnWarpMaxVec; ++i)
      if (i < per_lane) {
        const int c0 = (lane + i * 32) * kPer;
        float f[8], r[8];
        ln_unpack<kXDtype>(raw[i], f);
#pragma unroll
        for (int q = 0; q < kPer; q += 4) {
          float4 m = mul ? __ldg(reinterpret_cast<const float4*>(mul + c0 + q)) : make_float4(1.f, 1.f, 1.f, 1.f);
          const float4 a = add ? __ldg(reinterpret_cast<const float4*>(add + c0 + q)) : make_float4(0.f, 0.f, 0.f, 0.f);
          if (mul) { m.x += one; m.y += one; m.z += one; m.w += one; }
          r[q] = fmaf((f[q] - mean) * rstd, m.x, a.x);
          r[q + 1] = fmaf((f[q + 1] - mean) * rstd, m.y, a.y);
          r[q + 2] = fmaf((f[q + 2] - mean) * rstd, m.z, a.z);
          r[q + 3] = fmaf((f[q + 3] - mean) * rstd, m.w, a.w);
        }
        uint32_t o[4];
#pragma unroll
        for (int q = 0; q < kPer / 2; ++q) {
          if (p.out_fp16) {
            const __half2 h = __floats2half2_rn(r[2 * q], r[2 * q + 1]);
            o[q] = *reinterpret_cast<const uint32_t*>(&h);
          } else {
            const __nv_bfloat162 h = __floats2bfloat162_rn(r[2 * q], r[2 * q + 1]);
            o[q] = *reinterpret_cast<const uint32_t*>(&h);
          }
        }
        if constexpr (kPer == 8)
          *reinterpret_cast<uint4*>(dst + c0) = make_uint4(o[0], o[1], o[2], o[3]);
        else
          *reinterpret_cast<uint2*>(dst + c0) = make_uint2(o[0], o[1]);
      }
  }
}

// Column form: thread t of a CTA owns the 16-byte vectors t, t + blockDim.x, ... (kVec of them) of every row the CTA
// visits, so mul and add sit in registers (as 24 KB of loads per row they were four times the stream itself), and
// kRows rows go through the two block reductions (mean, then the centred sum of squares) together, with the
// next kRows in flight.  blockIdx.y is the batch.  HBM bound; us at 4096 / 6889 x 3072 bf16, 32760 x 1536 and 2000 x 5120
// fp32 (cold L2, 6 us of launch and event included): 24.6, 31.6, 65.5, 33.8 with a warp (5120: a block) per row, so
// 18.5, 24.6, 65.4, 22.6.
// Up to 384 threads run two (fp32, whose rows hold half as many channels per thread: three) CTAs per SM, wider rows
// with 64 registers and half as many rows in flight (two CTAs up to 512 threads).
template <int kXDtype, int kVec, int kMaxThreads>
__global__ void __launch_bounds__(kMaxThreads, kMaxThreads > 384 ? 1 : kXDtype == 2 ? 3 : 2) layernorm_affine_rows_kernel(const LayerNormParams p) {
  constexpr int kLnRows = kMaxThreads <= 384 ? 4 : 2;
  constexpr int kPer = kXDtype == 2 ? 4 : 8;  // channels per 16-byte vector
  __shared__ float red[2][kLnRows][32];
  const int n_vec = p.C / kPer;
  const int n_warps = blockDim.x >> 5;
  const float inv_c = 1.0f / static_cast<float>(p.C);
  const long long batch = blockIdx.y;
  const long long row_end = p.rows_per_batch;
  const uint4* x = static_cast<const uint4*>(p.x) + batch * p.rows_per_batch * n_vec;
  uint16_t* out = static_cast<uint16_t*>(p.out) + batch * p.rows_per_batch * p.C;

  float m[kVec][kPer], a[kVec][kPer];
#pragma unroll
  for (int v = 0; v < kVec; ++v) {
    const int vec = threadIdx.x + v * blockDim.x;
#pragma unroll
    for (int e = 0; e < kPer; e += 4) {
      float4 mv = make_float4(1.f, 1.f, 1.f, 1.f), av = make_float4(0.f, 0.f, 0.f, 0.f);
      if (vec < n_vec && p.mul) {
        mv = __ldg(reinterpret_cast<const float4*>(p.mul + batch * p.mul_batch_stride + vec * kPer + e));
        if (p.add_one) { mv.x += 1.f; mv.y += 1.f; mv.z += 1.f; mv.w += 1.f; }
      }
      if (vec < n_vec && p.add)
        av = __ldg(reinterpret_cast<const float4*>(p.add + batch * p.add_batch_stride + vec * kPer + e));
      m[v][e] = mv.x; m[v][e + 1] = mv.y; m[v][e + 2] = mv.z; m[v][e + 3] = mv.w;
      a[v][e] = av.x; a[v][e + 1] = av.y; a[v][e + 2] = av.z; a[v][e + 3] = av.w;
    }
  }
  const long long step = static_cast<long long>(gridDim.x) * kLnRows;
  long long row = static_cast<long long>(blockIdx.x) * kLnRows;
  uint4 cur[kLnRows][kVec], nxt[kLnRows][kVec];
  auto load = [&](uint4 (&buf)[kLnRows][kVec], long long row0) {
#pragma unroll
    for (int r = 0; r < kLnRows; ++r)
#pragma unroll
      for (int v = 0; v < kVec; ++v) {
        const int vec = threadIdx.x + v * blockDim.x;
        buf[r][v] = make_uint4(0u, 0u, 0u, 0u);
        if (vec < n_vec && row0 + r < row_end) buf[r][v] = __ldcs(x + (row0 + r) * n_vec + vec);
      }
  };
  load(cur, row);
  for (; row < row_end; row += step) {
    load(nxt, row + step);
    float s[kLnRows], mean[kLnRows];
#pragma unroll
    for (int r = 0; r < kLnRows; ++r) {
      s[r] = 0.f;
#pragma unroll
      for (int v = 0; v < kVec; ++v) {
        float f[8];
        ln_unpack<kXDtype>(cur[r][v], f);
#pragma unroll
        for (int e = 0; e < kPer; ++e) s[r] += f[e];
      }
    }
    block_sums<kLnRows, kLnRows == 4 || kVec == 2>(s, red[0], n_warps);
#pragma unroll
    for (int r = 0; r < kLnRows; ++r) {
      mean[r] = s[r] * inv_c;
      s[r] = 0.f;
#pragma unroll
      for (int v = 0; v < kVec; ++v) {
        if (static_cast<int>(threadIdx.x + v * blockDim.x) >= n_vec) continue;
        float f[8];
        ln_unpack<kXDtype>(cur[r][v], f);
#pragma unroll
        for (int e = 0; e < kPer; ++e) s[r] = fmaf(f[e] - mean[r], f[e] - mean[r], s[r]);
      }
    }
    block_sums<kLnRows, kLnRows == 4 || kVec == 2>(s, red[1], n_warps);
#pragma unroll
    for (int r = 0; r < kLnRows; ++r) {
      const float rstd = rsqrtf(s[r] * inv_c + p.eps);
#pragma unroll
      for (int v = 0; v < kVec; ++v) {
        const int vec = threadIdx.x + v * blockDim.x;
        if (vec >= n_vec || row + r >= row_end) continue;
        float f[8], y[kPer];
        ln_unpack<kXDtype>(cur[r][v], f);
#pragma unroll
        for (int e = 0; e < kPer; ++e) y[e] = fmaf((f[e] - mean[r]) * rstd, m[v][e], a[v][e]);
        uint16_t* dst = out + (row + r) * p.C + vec * kPer;
        if constexpr (kPer == 8)
          *reinterpret_cast<uint4*>(dst) = make_uint4(ln_pack(y[0], y[1], p.out_fp16), ln_pack(y[2], y[3], p.out_fp16),
                                                      ln_pack(y[4], y[5], p.out_fp16), ln_pack(y[6], y[7], p.out_fp16));
        else
          *reinterpret_cast<uint2*>(dst) = make_uint2(ln_pack(y[0], y[1], p.out_fp16), ln_pack(y[2], y[3], p.out_fp16));
      }
    }
#pragma unroll
    for (int r = 0; r < kLnRows; ++r)
#pragma unroll
      for (int v = 0; v < kVec; ++v) cur[r][v] = nxt[r][v];
  }
}

struct GateResidualParams {
  void* x;               // [rows, C] residual stream (x_dtype 0 bf16, 1 fp16, 2 fp32), updated in place
  int x_dtype;
  const void* y;         // [rows, C] bf16 / fp16 branch output
  const float* gate;     // [B or 1, C] fp32, or nullptr (= 1)
  long long gate_batch_stride;
  long long rows, rows_per_batch;
  int C;
  int y_fp16;
};

__global__ void __launch_bounds__(256)
gate_residual_kernel(const GateResidualParams p) {
  const int n_vec = p.C >> 2;
  const long long total = p.rows * n_vec;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride) {
    const long long row = i / n_vec;
    const int idx = static_cast<int>(i - row * n_vec);
    float4 xv = stream_ld4(p.x, p.x_dtype, static_cast<size_t>(i));
    const uint2 raw = __ldcs(reinterpret_cast<const uint2*>(p.y) + i);
    float2 y0, y1;
    if (p.y_fp16) {
      y0 = __half22float2(*reinterpret_cast<const __half2*>(&raw.x));
      y1 = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
    } else {
      y0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
      y1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    }
    float4 g = make_float4(1.f, 1.f, 1.f, 1.f);
    if (p.gate) g = __ldg(reinterpret_cast<const float4*>(p.gate + (row / p.rows_per_batch) * p.gate_batch_stride) + idx);
    xv.x = fmaf(y0.x, g.x, xv.x);
    xv.y = fmaf(y0.y, g.y, xv.y);
    xv.z = fmaf(y1.x, g.z, xv.z);
    xv.w = fmaf(y1.y, g.w, xv.w);
    stream_st4(p.x, p.x_dtype, static_cast<size_t>(i), xv);
  }
}

// Column form of the same update: a thread owns eight channels (its gate sits in registers) of every row its CTA
// visits, four rows in flight.  The CTA's threads are rows_par rows side by side, blockIdx.y is the batch.  (The
// general kernel divides 64-bit indices for every 4 elements and reads the gate each time.)  HBM bound; us at
// 4096 x 3072 bf16, 1024 x 3072 and 32760 x 1536 fp32 (inputs larger than L2, launches in a graph): 31.2, 8.4, 104.6 ->
// 14.3, 8.3, 80.5 (5.3, 4.5 and 6.2 TB/s).
template <int kXDtype, bool kYFp16, int kMaxThreads>
__global__ void __launch_bounds__(kMaxThreads) gate_residual_rows_kernel(const GateResidualParams p, int rows_par) {
  constexpr int kGateRows = kMaxThreads <= 512 ? 4 : 2;
  const int n_vec = p.C >> 3;
  const int sub = threadIdx.x / n_vec;
  const int vec = threadIdx.x - sub * n_vec;
  const long long batch = blockIdx.y;
  float g[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) g[e] = 1.f;
  if (p.gate) {
    const float4* gp = reinterpret_cast<const float4*>(p.gate + batch * p.gate_batch_stride) + vec * 2;
    const float4 g0 = __ldg(gp), g1 = __ldg(gp + 1);
    g[0] = g0.x; g[1] = g0.y; g[2] = g0.z; g[3] = g0.w;
    g[4] = g1.x; g[5] = g1.y; g[6] = g1.z; g[7] = g1.w;
  }
  constexpr int kXVecs = kXDtype == 2 ? 2 : 1;  // 16-byte vectors of eight stream channels
  uint4* x = static_cast<uint4*>(p.x) + (batch * p.rows_per_batch * n_vec + vec) * kXVecs;
  const uint4* y = static_cast<const uint4*>(p.y) + batch * p.rows_per_batch * n_vec + vec;
  const long long step = static_cast<long long>(gridDim.x) * rows_par;
  for (long long row0 = static_cast<long long>(blockIdx.x) * rows_par + sub; row0 < p.rows_per_batch; row0 += step * kGateRows) {
    uint4 yv[kGateRows], xv[kGateRows][kXVecs];
#pragma unroll
    for (int r = 0; r < kGateRows; ++r) {
      const long long row = row0 + r * step;
      if (row < p.rows_per_batch) {
        yv[r] = __ldcs(y + row * n_vec);
#pragma unroll
        for (int i = 0; i < kXVecs; ++i) xv[r][i] = __ldcs(x + row * n_vec * kXVecs + i);
      }
    }
#pragma unroll
    for (int r = 0; r < kGateRows; ++r) {
      const long long row = row0 + r * step;
      if (row >= p.rows_per_batch) continue;
      float fy[8], fx[8];
      ln_unpack<kYFp16 ? 1 : 0>(yv[r], fy);
      if constexpr (kXDtype == 2) {
        const uint4 lo = xv[r][0], hi = xv[r][1];
        fx[0] = __uint_as_float(lo.x); fx[1] = __uint_as_float(lo.y); fx[2] = __uint_as_float(lo.z); fx[3] = __uint_as_float(lo.w);
        fx[4] = __uint_as_float(hi.x); fx[5] = __uint_as_float(hi.y); fx[6] = __uint_as_float(hi.z); fx[7] = __uint_as_float(hi.w);
      } else {
        ln_unpack<kXDtype>(xv[r][0], fx);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) fx[e] = fmaf(fy[e], g[e], fx[e]);
      uint4* dst = x + row * n_vec * kXVecs;
      if constexpr (kXDtype == 2) {
        dst[0] = make_uint4(__float_as_uint(fx[0]), __float_as_uint(fx[1]), __float_as_uint(fx[2]), __float_as_uint(fx[3]));
        dst[1] = make_uint4(__float_as_uint(fx[4]), __float_as_uint(fx[5]), __float_as_uint(fx[6]), __float_as_uint(fx[7]));
      } else {
        dst[0] = make_uint4(ln_pack(fx[0], fx[1], kXDtype), ln_pack(fx[2], fx[3], kXDtype), ln_pack(fx[4], fx[5], kXDtype),
                            ln_pack(fx[6], fx[7], kXDtype));
      }
    }
  }
}

// ----------------------------------------------------------------------------
// Classifier-free guidance: out = uncond + scale * (cond - uncond), optionally rescaled row by row to
// the norm of the conditional prediction (out *= ||cond|| / ||out|| over the last dim).  One warp per
// row, three passes over registers-sized chunks are avoided by keeping the row sums in two
// accumulators and re-reading the (L1 / L2 resident) row for the rescaled store.
// ----------------------------------------------------------------------------
struct CfgCombineParams {
  const void* cond;
  const void* uncond;
  void* out;
  long long rows;
  int C;
  int dtype;       // kBF16 / kFP16 / kFP32 of all three tensors
  int rescale;
  float scale;
};

__device__ __forceinline__ float cfg_ld(const void* p, int dtype, size_t i) {
  if (dtype == 2) return static_cast<const float*>(p)[i];
  if (dtype == 0) return __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]);
  return __half2float(static_cast<const __half*>(p)[i]);
}
__device__ __forceinline__ void cfg_st(void* p, int dtype, size_t i, float v) {
  if (dtype == 2) static_cast<float*>(p)[i] = v;
  else if (dtype == 0) static_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v);
  else static_cast<__half*>(p)[i] = __float2half_rn(v);
}

__global__ void __launch_bounds__(256) cfg_combine_kernel(const CfgCombineParams p) {
  const int lane = threadIdx.x & 31;
  const long long warps = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  for (long long row = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); row < p.rows;
       row += warps) {
    const size_t base = static_cast<size_t>(row) * p.C;
    float factor = 1.f;
    if (p.rescale) {
      float nc = 0.f, no = 0.f;
      for (int c = lane; c < p.C; c += 32) {
        const float a = cfg_ld(p.cond, p.dtype, base + c), b = cfg_ld(p.uncond, p.dtype, base + c);
        // the reference forms `combined` in the tensors' dtype before taking its norm
        float o = b + p.scale * (a - b);
        if (p.dtype == 0) o = __bfloat162float(__float2bfloat16_rn(o));
        else if (p.dtype == 1) o = __half2float(__float2half_rn(o));
        nc = fmaf(a, a, nc);
        no = fmaf(o, o, no);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        nc += __shfl_xor_sync(0xffffffffu, nc, o);
        no += __shfl_xor_sync(0xffffffffu, no, o);
      }
      factor = sqrtf(nc) / sqrtf(no);
    }
    for (int c = lane; c < p.C; c += 32) {
      const float a = cfg_ld(p.cond, p.dtype, base + c), b = cfg_ld(p.uncond, p.dtype, base + c);
      cfg_st(p.out, p.dtype, base + c, (b + p.scale * (a - b)) * factor);
    }
  }
}

}  // namespace chitu
