// What follows a mixer that reads a memory out head by head (bfloat16): every head's float32 read-out divided by its own root mean
// square, times a weight, times a gate's sigmoid or SiLU.
//
//   out[t, h, :] = y / sqrt(mean(y^2) + eps) * w * act(gate[t, h, :])
//
// Dv / 8 neighbouring lanes (a power of two, at most 32) take a head, eight channels each: two 16-byte loads of y, one of the gate
// and one store a thread, the sum by shuffles.  What bounds it: bytes (2048 tokens of 32 heads of 64: 33 MB).  A warp per head with
// four-byte and two-byte accesses, y read twice, took 23 to 25 us; this takes 9.
#pragma once

#include "common.cuh"

__device__ __forceinline__ void unpack_bf16x8(uint4 u, float* x) {
  const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) { x[2 * e] = __uint_as_float(w[e] << 16); x[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u); }
}
__device__ __forceinline__ uint4 pack_bf16x8(const float* x) {
  unsigned w[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(x[2 * e], x[2 * e + 1]);
    w[e] = *reinterpret_cast<const unsigned*>(&v);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// weight [Dv], or [width] with per_head.  The launch has a whole warp for every 256 channels: lanes behind the last one take part in
// the shuffles.
__global__ void __launch_bounds__(256)
head_finish_bf16x8_kernel(const float* __restrict__ y, const __nv_bfloat16* __restrict__ gate, int ld_gate,
                          const float* __restrict__ weight, int per_head, __nv_bfloat16* __restrict__ out, int ld_out, int T_,
                          int width, int Dv, float eps, int silu) {
  pdl_trigger();
  pdl_wait();
  const int vecs = width >> 3, lanes = Dv >> 3;
  const long long unit = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = unit < (long long)T_ * vecs;
  const int t = live ? (int)(unit / vecs) : 0, c = live ? (int)(unit - (long long)t * vecs) * 8 : 0;
  float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, g[8];
  if (live) {
    const float4 a = *reinterpret_cast<const float4*>(y + (size_t)t * width + c);
    const float4 b = *reinterpret_cast<const float4*>(y + (size_t)t * width + c + 4);
    unpack_bf16x8(*reinterpret_cast<const uint4*>(gate + (size_t)t * ld_gate + c), g);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
  float ss = 0.f;
#pragma unroll
  for (int e = 0; e < 8; ++e) ss = fmaf(v[e], v[e], ss);
  for (int o = lanes >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if (!live) return;
  const float r = 1.0f / sqrtf(ss / (float)Dv + eps);
  const float* w = weight + (per_head ? c : c % Dv);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float s = 1.0f / (1.0f + expf(-g[e]));
    v[e] = v[e] * r * w[e] * (silu ? g[e] * s : s);
  }
  *reinterpret_cast<uint4*>(out + (size_t)t * ld_out + c) = pack_bf16x8(v);
}

// Whether the sizes and addresses allow it; if so, launches.
static inline bool head_finish_bf16x8(const float* y, const void* gate, int ld_gate, const float* weight, int per_head, void* out,
                                      int ld_out, int T_, int heads, int Dv, float eps, int silu, cudaStream_t stream) {
  const int lanes = Dv / 8;
  if (Dv % 8 || lanes < 1 || lanes > 32 || (lanes & (lanes - 1)) || ld_gate % 8 || ld_out % 8) return false;
  if ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(out)) & 15) return false;
  const long long units = (long long)T_ * heads * lanes;
  if ((units + 255) / 256 > 0x7fffffffLL) return false;
  kvb_launch(head_finish_bf16x8_kernel, dim3((unsigned)((units + 255) / 256)), dim3(256), 0, stream, y, (const __nv_bfloat16*)gate,
             ld_gate, weight, per_head, (__nv_bfloat16*)out, ld_out, T_, heads * Dv, Dv, eps, silu);
  return true;
}
