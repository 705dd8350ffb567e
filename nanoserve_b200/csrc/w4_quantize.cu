// Round-to-nearest symmetric 4-bit group quantizer (cold path: runs once per weight matrix).
//
// Same arithmetic, bit for bit, as the reference's quantize_w4_kernel (kernels/quant/w4a16.cuh:274-297):
//   per (row, group): mx = max|w|;  s = bf16_rn(mx > 0 ? mx / 7 : 1);  q = clamp(rint_even(w / float(s)) + 8, 0, 15)
// with IEEE fp32 division.  The reference walks a group with one thread; here each lane converts whole 8-element
// words from 16-byte loads, and the maximum is a shuffle reduction (max is order-independent, so the result is
// identical).
//
// Groups of 32, 64, 128 and 256 (a group is a power-of-two run of lanes) run w4_quantize_fast_kernel, bound by the 2.5
// bytes per weight it moves; other groups run w4_quantize_kernel, a warp per group and an IEEE division per weight.
#include <algorithm>

#include "ptx.cuh"
#include "w4_internal.h"

namespace b2 {
namespace {

__global__ void __launch_bounds__(256) w4_quantize_kernel(const __nv_bfloat16* __restrict__ W,
                                                          uint32_t* __restrict__ Wq,
                                                          __nv_bfloat16* __restrict__ S, int N, int K, int G) {
  const int KG = K / G;
  const int lane = threadIdx.x & 31;
  const size_t total = (size_t)N * KG;
  const size_t warps = ((size_t)gridDim.x * blockDim.x) >> 5;
  for (size_t idx = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; idx < total; idx += warps) {
    const size_t n = idx / KG;
    const int g = (int)(idx - n * KG);
    const __nv_bfloat16* w = W + n * K + (size_t)g * G;
    const int words = G / 8;
    float mx = 0.f;
    for (int j = lane; j < words; j += 32) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(w) + j);
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(h[i]);
        mx = fmaxf(mx, fmaxf(fabsf(f.x), fabsf(f.y)));
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const __nv_bfloat16 sb = __float2bfloat16(mx > 0.f ? __fdiv_rn(mx, 7.f) : 1.f);
    const float sf = __bfloat162float(sb);
    if (lane == 0) S[idx] = sb;
    for (int j = lane; j < words; j += 32) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(w) + j);
      const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&v);
      uint32_t word = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int q = min(15, max(0, __float2int_rn(__fdiv_rn(__bfloat162float(e[i]), sf)) + 8));
        word |= static_cast<uint32_t>(q) << (4 * i);
      }
      Wq[n * (K / 8) + (size_t)g * words + j] = word;
    }
  }
}

// |w| as bf16 bits order like their values: the largest of a lane's eight.
__device__ __forceinline__ uint32_t abs_max_bits(const uint4& v) {
  const uint32_t m = __vmaxu2(__vmaxu2(v.x & 0x7FFF7FFFu, v.y & 0x7FFF7FFFu),
                              __vmaxu2(v.z & 0x7FFF7FFFu, v.w & 0x7FFF7FFFu));
  return max(m & 0xFFFFu, m >> 16);
}

// LPG lanes per group, a lane two of its words (G = 16 LPG), half a group apart: a warp's load covers whole lines or sectors.  Groups
// tile W without gaps (K % G == 0): a warp takes kUnroll times 32 / LPG consecutive groups, all their loads in flight before
// the first is used.  The scale and its reciprocal are then computed once for sixteen weights of a lane, and the arithmetic takes
// two weights per instruction: with one word per lane the kernel was bound by its 75 instructions per word as much as by memory.
//
// The division is replaced without changing a bit.  w and s have 8-bit significands, so w / s is either exactly halfway
// between two integers or at least 2^-10 from it (the numerator of w / s - (k + 1/2) is a multiple of the smaller unit
// of the two).  u = fma(w, rn(1 / s), 1536) rounds w / s to a multiple of 2^-13 with an error below 2^-13: a halfway
// case lands on the half exactly and no other does.  The second addition rounds that to an integer, half to even like
// rint, and leaves q = rint(w / s) + 8 in the low mantissa bits; |w / s| <= 7.03, so no clamp.  This needs a finite,
// normal s with a normal reciprocal; a group that has none, or an inf or a nan, is divided as before.
//
// 18944 x 3584 at G = 128: 27.0 us (6.3 TB/s of bf16 in, words and scales out; a copy's rate), one word per lane 35.0, with a
// division per weight and half of the lanes idle 162.
constexpr int kUnroll = 2, kThreads = 128;  // 1, 2, 3, 4 at 256 threads: 30.4, 27.3, 27.8, 28.8 us; 2 at 128 and 512: 27.0, 28.8
template <int LPG>
__global__ void __launch_bounds__(kThreads) w4_quantize_fast_kernel(const uint4* __restrict__ W, uint32_t* __restrict__ Wq,
                                                               __nv_bfloat16* __restrict__ S, size_t groups) {
  constexpr int kGroups = 32 / LPG;  // of a warp at a time
  const int lane = threadIdx.x & 31, r = lane % LPG;
  const size_t g0 = (((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * (kGroups * kUnroll) + lane / LPG;
  uint4 v[kUnroll][2];
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const size_t g = g0 + u * kGroups;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      v[u][h] = make_uint4(0u, 0u, 0u, 0u);
      if (g < groups) v[u][h] = __ldcs(W + g * (2 * LPG) + h * LPG + r);
    }
  }
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    uint32_t mx = max(abs_max_bits(v[u][0]), abs_max_bits(v[u][1]));
#pragma unroll
    for (int o = LPG / 2; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    __nv_bfloat16 sb = __float2bfloat16(mx ? __fdiv_rn(__uint_as_float(mx << 16), 7.f) : 1.f);
    float sf = __bfloat162float(sb);
    uint32_t word[2] = {0u, 0u};
    // s outside [2^-100, 2^100] (or of an infinite or nan maximum): the quotient itself
    const bool plain = mx < 0x7F80u && sf >= 0x1p-100f && sf <= 0x1p100f;
    if (__all_sync(0xffffffffu, plain)) {
      const float rc = __frcp_rn(sf);
      const float2 rc2 = make_float2(rc, rc), half2 = make_float2(1536.f, 1536.f);
      const float to_int = 12582912.f - 1536.f + 8.f;  // 1.5 * 2^23 + 8: q in the low mantissa bits
      const float2 to_int2 = make_float2(to_int, to_int);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t e[4] = {v[u][h].x, v[u][h].y, v[u][h].z, v[u][h].w};
#pragma unroll
        for (int i = 3; i >= 0; --i) {
          const float2 w2 = make_float2(__uint_as_float(e[i] << 16), __uint_as_float(e[i] & 0xFFFF0000u));
          const float2 q = add_f32x2(fma_f32x2(w2, rc2, half2), to_int2);
          word[h] = word[h] * 16u + __float_as_uint(q.y);
          word[h] = word[h] * 16u + __float_as_uint(q.x);
        }
        word[h] -= 0x4B400000u * 0x11111111u;  // what the eight exponents left (modulo 2^32)
      }
    } else {
      float m = 0.f;  // the maximum leaves nans out, like fmaxf
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t e[4] = {v[u][h].x, v[u][h].y, v[u][h].z, v[u][h].w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
          m = fmaxf(m, fmaxf(fabsf(__uint_as_float(e[i] << 16)), fabsf(__uint_as_float(e[i] & 0xFFFF0000u))));
      }
#pragma unroll
      for (int o = LPG / 2; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      sb = __float2bfloat16(m > 0.f ? __fdiv_rn(m, 7.f) : 1.f);
      sf = __bfloat162float(sb);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t e[4] = {v[u][h].x, v[u][h].y, v[u][h].z, v[u][h].w};
#pragma unroll 1
        for (int i = 0; i < 8; ++i) {
          const uint32_t pair = i < 2 ? e[0] : i < 4 ? e[1] : i < 6 ? e[2] : e[3];
          const float w = __uint_as_float(i & 1 ? pair & 0xFFFF0000u : pair << 16);
          word[h] |= static_cast<uint32_t>(min(15, max(0, __float2int_rn(__fdiv_rn(w, sf)) + 8))) << (4 * i);
        }
      }
    }
    const size_t g = g0 + u * kGroups;
    if (g < groups) {
      __stcs(Wq + g * (2 * LPG) + r, word[0]);
      __stcs(Wq + g * (2 * LPG) + LPG + r, word[1]);
      if (r == 0) S[g] = sb;
    }
  }
}

template <int LPG>
void launch_fast(const void* W, void* Wq, void* S, size_t groups, cudaStream_t stream) {
  const size_t per_cta = (kThreads / 32) * (32 / LPG) * kUnroll;
  w4_quantize_fast_kernel<LPG><<<(unsigned)((groups + per_cta - 1) / per_cta), kThreads, 0, stream>>>(
      static_cast<const uint4*>(W), static_cast<uint32_t*>(Wq), static_cast<__nv_bfloat16*>(S), groups);
}

}  // namespace

int quantize_launch(const void* W, void* Wq, void* S, int N, int K, int G, cudaStream_t stream) {
  if (G <= 0 || K <= 0 || N <= 0 || K % G || G % 32) return kErrBadShape;
  if (!W || !Wq || !S) return kErrBadPointer;
  // 16-byte loads of W need 16-byte aligned rows and groups: K % 8 == 0 follows from G % 32 == 0
  if (reinterpret_cast<uintptr_t>(W) & 15) return kErrBadPointer;
  const size_t groups = (size_t)N * (K / G);
  if (G == 32 || G == 64 || G == 128 || G == 256) {
    switch (G) {
      case 32: launch_fast<2>(W, Wq, S, groups, stream); break;
      case 64: launch_fast<4>(W, Wq, S, groups, stream); break;
      case 128: launch_fast<8>(W, Wq, S, groups, stream); break;
      default: launch_fast<16>(W, Wq, S, groups, stream); break;
    }
    return (int)cudaGetLastError();
  }
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
    return kErrDevice;
  const size_t blocks = std::min<size_t>((groups + 7) / 8, (size_t)sms * 32);  // grid-stride: 32 CTAs per SM at most
  w4_quantize_kernel<<<(unsigned)blocks, 256, 0, stream>>>(static_cast<const __nv_bfloat16*>(W),
                                                          static_cast<uint32_t*>(Wq),
                                                          static_cast<__nv_bfloat16*>(S), N, K, G);
  return (int)cudaGetLastError();
}

}  // namespace b2
