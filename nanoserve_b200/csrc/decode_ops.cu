// Small kernels that sit between the quantized linears of a batch-1 decode step and read the current
// position from device memory, so that one captured CUDA graph serves every step:
//   b2_rope_kv_store     bias add + rotary embedding on q and k of the new token, k/v appended to the cache
//   b2_decode_attention  one query token against the cached keys/values (grouped-query attention)
//   b2_greedy_next       argmax over the logits, position += 1, embedding row of the chosen token
// The reference does these steps with PyTorch ops and a Python-side position (python/nanoserve/qwen.py:119-133,
// 147-151, 174-177: bias add, rope, _store_kv, SDPA over the cache, argmax); a host-side position would force one
// graph per step.  Arithmetic follows the reference's conventions: bf16 storage, fp32 math, rotate-half RoPE with
// angle = pos * inv_freq[i] (kernels/fused/rope.cuh:14-43), softmax scale 1/sqrt(D).
#include <atomic>
#include <cfloat>
#include <cstdint>
#include <cuda_bf16.h>

#include "../../include/nanoserve_b200.h"
#include "ptx.cuh"
#include "w4_common.cuh"
#include "w4_internal.h"

namespace {

using bf16 = __nv_bfloat16;

// The small kernels of a decode step are launched with programmatic stream serialization, like the GEMVs around them:
// they become resident while the previous kernel drains and start the moment it has completed, which takes the
// launch latency off the step's critical path.  Under such a launch the SM's L1 is not invalidated between the
// producer of the inputs and the loads, so everything a previous kernel may have written is read with
// ld.global.cg (L2), never through the non-coherent path.
__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ float ld_bf16(const bf16* p) {
  return __bfloat162float(__ushort_as_bfloat16(__ldcg(reinterpret_cast<const unsigned short*>(p))));
}
// E (2 or 4) consecutive bf16 as floats with one L2 load.
template <int E>
__device__ __forceinline__ void ld_row(const bf16* p, float (&f)[E]) {
  static_assert(E == 2 || E == 4, "head dimension 64 or 128");
  if constexpr (E == 4) {
    const uint2 v = __ldcg(reinterpret_cast<const uint2*>(p));
    f[0] = __uint_as_float(v.x << 16);
    f[1] = __uint_as_float(v.x & 0xFFFF0000u);
    f[2] = __uint_as_float(v.y << 16);
    f[3] = __uint_as_float(v.y & 0xFFFF0000u);
  } else {
    const unsigned v = __ldcg(reinterpret_cast<const unsigned*>(p));
    f[0] = __uint_as_float(v << 16);
    f[1] = __uint_as_float(v & 0xFFFF0000u);
  }
}
// The rotation of the pair (a, b) of a key, and of the element x of a query whose partner D/2 away is `other`.  Which product is
// rounded before the addition is written out: left to the compiler it differed between kernels, and one in 2 * 10^5 of the
// appended key elements with it (one in 250 where the products cancel).
__device__ __forceinline__ void rotate_pair(float& a, float& b, float sn, float cs) {
  const float ra = __fmaf_rn(a, cs, -__fmul_rn(b, sn)), rb = __fmaf_rn(b, cs, __fmul_rn(a, sn));
  a = ra;
  b = rb;
}
__device__ __forceinline__ float rotate_query(float x, float other, float sn, float cs, bool first_half) {
  return first_half ? __fmaf_rn(x, cs, -__fmul_rn(other, sn)) : __fmaf_rn(other, sn, __fmul_rn(x, cs));
}
template <typename... Args>
cudaError_t launch_pdl(void (*kernel)(Args...), dim3 grid, dim3 block, cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = 0;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// grid: Hq + 2*Hk blocks (one per head of the fused qkv row), block: D/2 threads.
// With wait_sig set, qkv is the gathered output of a tensor-parallel GEMV (b2_w4_linear_tp): every block first waits
// (bounded) until all producing CTAs of all ranks have counted themselves in, then reads qkv from L2.
__global__ void rope_kv_store_kernel(bf16* qkv, const bf16* __restrict__ bias,
                                     const float* __restrict__ inv_freq, const int* __restrict__ pos_ptr,
                                     bf16* __restrict__ cache_k, bf16* __restrict__ cache_v, int Hq, int Hk, int D,
                                     int max_len, const unsigned* wait_sig, const int* epoch, unsigned wait_per_epoch,
                                     int* status) {
  const int h = blockIdx.x, i = threadIdx.x, half = D / 2;
  pdl_begin();
  if (wait_sig != nullptr) {
    if (i == 0) {
      const unsigned target = ((unsigned)*reinterpret_cast<const volatile int*>(epoch) + 1u) * wait_per_epoch;
      const long long t0 = clock64();
      for (;;) {
        unsigned v;
        asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(wait_sig) : "memory");
        if ((int)(v - target) >= 0) break;
        if (clock64() - t0 > 1000000000LL) {  // about half a second: report and go on with what is there
          if (status != nullptr) atomicCAS(status, 0, b2::kStatusGemvTimeout);
          break;
        }
        __nanosleep(40);
      }
    }
    __syncthreads();
  }
  const int pos = __ldcg(pos_ptr);
  bf16* x = qkv + (size_t)h * D;
  float a = __bfloat162float(__ushort_as_bfloat16(__ldcg(reinterpret_cast<const unsigned short*>(x) + i)));
  float b = __bfloat162float(__ushort_as_bfloat16(__ldcg(reinterpret_cast<const unsigned short*>(x) + i + half)));
  if (bias != nullptr) {  // the projection output is stored in bf16, then the bias is added in bf16 (q += bq)
    a = __bfloat162float(__float2bfloat16(a + __bfloat162float(bias[(size_t)h * D + i])));
    b = __bfloat162float(__float2bfloat16(b + __bfloat162float(bias[(size_t)h * D + i + half])));
  }
  if (h < Hq + Hk) {  // q and k heads rotate, v heads do not
    float sn, cs;
    sincosf((float)pos * inv_freq[i], &sn, &cs);
    rotate_pair(a, b, sn, cs);
  }
  const bf16 oa = __float2bfloat16(a), ob = __float2bfloat16(b);
  x[i] = oa;
  x[i + half] = ob;
  if (h >= Hq && pos < max_len) {
    const int kh = h - Hq;
    bf16* dst = (kh < Hk ? cache_k + ((size_t)kh * max_len + pos) * D
                         : cache_v + ((size_t)(kh - Hk) * max_len + pos) * D);
    dst[i] = oa;
    dst[i + half] = ob;
  }
}

// Decode attention in two launches.  Pass 1, grid (Hk, kSplits): a CTA takes one KV head and one slice of the
// cached positions; it first copies the slice's K and V rows into shared memory with 16-byte loads that are all in
// flight together (one L2 round trip for the whole slice; a loop of dependent-looking 8-byte loads per position
// cost a round trip per position: 16 us per layer at 600 positions), then warp w serves query head w of the group
// (Hq / Hk <= 8 heads share a KV head); lanes split the head dimension; online softmax per warp.  It writes
// un-normalised partials (max, sum, acc[D]) per (query head, split).  Pass 2, grid Hq: merges the splits, all of
// its loads issued before the first use.  With 4 KV heads x 32 splits the first pass fills 128 SMs however long
// the cache is.
constexpr int kSplits = 32;
constexpr int kTileRows = 32;  // positions staged in shared memory at a time

template <int D>
__global__ void __launch_bounds__(256) decode_attention_partial_kernel(
    const bf16* q, const bf16* cache_k, const bf16* cache_v, const int* pos_ptr, float* part, int Hq, int Hk,
    int max_len, float scale) {
  constexpr int E = D / 32;        // elements per lane
  constexpr int kRowU4 = D / 8;    // 16-byte units per row
  __shared__ __align__(16) bf16 s_k[kTileRows * D];
  __shared__ __align__(16) bf16 s_v[kTileRows * D];
  const int kh = blockIdx.x, sp = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rep = Hq / Hk;
  pdl_begin();
  const int h = kh * rep + min(warp, rep - 1);
  const int n = min(__ldcg(pos_ptr) + 1, max_len);
  const int per = (n + kSplits - 1) / kSplits;
  const int j0 = sp * per, j1 = min(n, j0 + per);
  const uint4* kbase = reinterpret_cast<const uint4*>(cache_k + (size_t)kh * max_len * D);
  const uint4* vbase = reinterpret_cast<const uint4*>(cache_v + (size_t)kh * max_len * D);
  float qf[E];
  ld_row<E>(q + (size_t)h * D + lane * E, qf);
#pragma unroll
  for (int e = 0; e < E; ++e) qf[e] *= scale;
  float m = -FLT_MAX, l = 0.f, acc[E];
#pragma unroll
  for (int e = 0; e < E; ++e) acc[e] = 0.f;
  for (int t0 = j0; t0 < j1; t0 += kTileRows) {
    const int rows = min(kTileRows, j1 - t0);
    const int units = rows * kRowU4;
    if (t0 > j0) __syncthreads();  // everybody is done with the previous tile
    // all loads first, then all stores: one round trip for the tile
    constexpr int kPerThread = (kTileRows * kRowU4 + 255) / 256;
    uint4 kv[kPerThread], vv[kPerThread];
#pragma unroll
    for (int i = 0; i < kPerThread; ++i) {
      const int u = threadIdx.x + i * 256;
      if (u < units) {
        kv[i] = __ldcg(kbase + (size_t)t0 * kRowU4 + u);
        vv[i] = __ldcg(vbase + (size_t)t0 * kRowU4 + u);
      }
    }
#pragma unroll
    for (int i = 0; i < kPerThread; ++i) {
      const int u = threadIdx.x + i * 256;
      if (u < units) {
        reinterpret_cast<uint4*>(s_k)[u] = kv[i];
        reinterpret_cast<uint4*>(s_v)[u] = vv[i];
      }
    }
    __syncthreads();
    if (warp < rep) {
      for (int r = 0; r < rows; ++r) {
        float s = 0.f, kf[E], vf[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
          kf[e] = __bfloat162float(s_k[r * D + lane * E + e]);
          vf[e] = __bfloat162float(s_v[r * D + lane * E + e]);
        }
#pragma unroll
        for (int e = 0; e < E; ++e) s += qf[e] * kf[e];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const float mn = fmaxf(m, s);
        const float corr = __expf(m - mn), pj = __expf(s - mn);
        l = l * corr + pj;
#pragma unroll
        for (int e = 0; e < E; ++e) acc[e] = acc[e] * corr + pj * vf[e];
        m = mn;
      }
    }
  }
  if (warp >= rep) return;
  float* out = part + ((size_t)h * kSplits + sp) * (D + 2);
  if (lane == 0) {
    out[0] = m;
    out[1] = l;
  }
#pragma unroll
  for (int e = 0; e < E; ++e) out[2 + lane * E + e] = acc[e];
}

template <int D>
__global__ void decode_attention_merge_kernel(const float* part, bf16* out) {
  const int h = blockIdx.x, d = threadIdx.x;  // block: D threads
  pdl_begin();
  const float* p = part + (size_t)h * kSplits * (D + 2);
  // every load of the merge is issued before the first use: one L2 round trip, not one per split
  float ms[kSplits], ls[kSplits], as[kSplits];
#pragma unroll
  for (int s = 0; s < kSplits; ++s) {
    ms[s] = __ldcg(p + s * (D + 2));
    ls[s] = __ldcg(p + s * (D + 2) + 1);
    as[s] = __ldcg(p + s * (D + 2) + 2 + d);
  }
  float mm = -FLT_MAX;
#pragma unroll
  for (int s = 0; s < kSplits; ++s) mm = fmaxf(mm, ms[s]);
  float num = 0.f, den = 0.f;
#pragma unroll
  for (int s = 0; s < kSplits; ++s) {
    const float f = ms[s] == -FLT_MAX ? 0.f : __expf(ms[s] - mm);
    num += f * as[s];
    den += f * ls[s];
  }
  out[(size_t)h * D + d] = __float2bfloat16(den > 0.f ? num / den : 0.f);
}

// The attention of one decode step in ONE launch: bias add + RoPE on q and k of the new token, the new k/v row
// appended to the cache, the partial pass over the cache, and the merge.  Same grid and tile loop as the two-launch
// form above.  Every warp prepares its own query head in registers (bias, rotation, rounding to bf16 as
// b2_rope_kv_store stores it).  The CTA whose slice holds the new position computes the new k and v rows, stores them
// to the cache and serves them to its own tile loop from shared memory.  The last CTA of a KV head to have written
// its partials (an arrival counter per KV head; nobody waits) merges the splits of that head's query heads.
// (Tensor-parallel calls and the form with a counter; the others run decode_attention_cluster_kernel below.)
template <int D>
__global__ void __launch_bounds__(256) decode_attention_fused_kernel(
    const bf16* qkv, const bf16* __restrict__ bias, const float* __restrict__ inv_freq, const int* pos_ptr,
    bf16* cache_k, bf16* cache_v, float* part, int* counters, bf16* out, int Hq, int Hk, int max_len, float scale,
    const unsigned* wait_sig, const int* epoch, unsigned wait_per_epoch, int* status, const b2::GemvTp ann,
    int early) {
  constexpr int E = D / 32;        // elements per lane
  constexpr int kRowU4 = D / 8;    // 16-byte units per row
  constexpr int half = D / 2;
  __shared__ __align__(16) bf16 s_k[kTileRows * D];
  __shared__ __align__(16) bf16 s_v[kTileRows * D];
  __shared__ __align__(16) bf16 s_newk[D];
  __shared__ __align__(16) bf16 s_newv[D];
  __shared__ float s_f[8 * kSplits];   // merge: weight of every (query head of the group, split)
  __shared__ float s_den[8];
  __shared__ int s_last;
  const int kh = blockIdx.x, sp = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rep = Hq / Hk;
  const uint4* kbase = reinterpret_cast<const uint4*>(cache_k + (size_t)kh * max_len * D);
  const uint4* vbase = reinterpret_cast<const uint4*>(cache_v + (size_t)kh * max_len * D);
  constexpr int kPerThread = (kTileRows * kRowU4 + 255) / 256;
  uint4 kv[kPerThread], vv[kPerThread];
  int pos = 0, n = 0, per = 0, j0 = 0, j1 = 0;
  auto slice = [&]() {
    pos = __ldcg(pos_ptr);
    n = min(pos + 1, max_len);
    per = (n + kSplits - 1) / kSplits;
    j0 = sp * per;
    j1 = min(n, j0 + per);
  };
  auto request = [&](int t0) {
    const int units = min(kTileRows, j1 - t0) * kRowU4;
#pragma unroll
    for (int i = 0; i < kPerThread; ++i) {
      const int u = tid + i * 256;
      if (u < units && t0 + u / kRowU4 != pos) {  // the row this launch appends is not in the cache yet
        kv[i] = __ldcg(kbase + (size_t)t0 * kRowU4 + u);
        vv[i] = __ldcg(vbase + (size_t)t0 * kRowU4 + u);
      }
    }
  };
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // `early`: the position and the cached rows below it were written by earlier steps, not by the kernel in front of
  // this one (which produces qkv): the first tile's rows are requested while that kernel still runs
  if (early) {
    slice();
    if (j0 < j1) request(j0);
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // deferred signal of the tensor-parallel GEMV in front of this kernel (it has completed)
  if (ann.announce_world && blockIdx.x == 0 && blockIdx.y == 0 && tid < ann.announce_world)
    asm volatile("red.release.sys.global.add.u32 [%0], 1;" ::"l"(ann.announce_peer[tid]) : "memory");
  if (wait_sig != nullptr) {
    if (tid == 0) {
      const unsigned target = ((unsigned)*reinterpret_cast<const volatile int*>(epoch) + 1u) * wait_per_epoch;
      const long long t0 = clock64();
      for (;;) {
        unsigned v;
        asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(wait_sig) : "memory");
        if ((int)(v - target) >= 0) break;
        if (clock64() - t0 > 1000000000LL) {  // about half a second: report and go on with what is there
          if (status != nullptr) atomicCAS(status, 0, b2::kStatusGemvTimeout);
          break;
        }
        __nanosleep(40);
      }
    }
    __syncthreads();
  }
  if (!early) {
    slice();
    if (j0 < j1) request(j0);
  }
  const bool owner = pos < max_len && pos >= j0 && pos < j1;  // this CTA's slice holds the new position

  // ---- the new k and v rows (owner only): thread i < D/2 rotates the pair (i, i + D/2) of k, the next D/2 threads
  // add the bias to a pair of v
  if (owner && tid < D) {
    const bool is_v = tid >= half;
    const int i = is_v ? tid - half : tid;
    const int hh = Hq + (is_v ? Hk : 0) + kh;
    const bf16* x = qkv + (size_t)hh * D;
    float a = ld_bf16(x + i), b = ld_bf16(x + i + half);
    if (bias != nullptr) {
      a = __bfloat162float(__float2bfloat16(a + __bfloat162float(bias[(size_t)hh * D + i])));
      b = __bfloat162float(__float2bfloat16(b + __bfloat162float(bias[(size_t)hh * D + i + half])));
    }
    if (!is_v) {
      float sn, cs;
      sincosf((float)pos * inv_freq[i], &sn, &cs);
      rotate_pair(a, b, sn, cs);
    }
    const bf16 oa = __float2bfloat16(a), ob = __float2bfloat16(b);
    bf16* sm = is_v ? s_newv : s_newk;
    sm[i] = oa;
    sm[i + half] = ob;
    bf16* dst = (is_v ? cache_v : cache_k) + ((size_t)kh * max_len + pos) * D;
    dst[i] = oa;
    dst[i + half] = ob;
  }

  // ---- this warp's query head: bias, rotation, bf16 rounding, softmax scale
  const int h = kh * rep + min(warp, rep - 1);
  float qf[E];
  {
    ld_row<E>(qkv + (size_t)h * D + lane * E, qf);
    if (bias != nullptr) {
#pragma unroll
      for (int e = 0; e < E; ++e)
        qf[e] = __bfloat162float(__float2bfloat16(qf[e] + __bfloat162float(bias[(size_t)h * D + lane * E + e])));
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const float other = __shfl_xor_sync(0xffffffffu, qf[e], 16);  // the element D/2 away
      float sn, cs;
      sincosf((float)pos * inv_freq[(lane * E + e) % half], &sn, &cs);
      qf[e] = __bfloat162float(__float2bfloat16(rotate_query(qf[e], other, sn, cs, lane < 16))) * scale;
    }
  }

  float m = -FLT_MAX, l = 0.f, acc[E];
#pragma unroll
  for (int e = 0; e < E; ++e) acc[e] = 0.f;
  for (int t0 = j0; t0 < j1; t0 += kTileRows) {
    const int rows = min(kTileRows, j1 - t0);
    const int units = rows * kRowU4;
    if (t0 > j0) request(t0);
    __syncthreads();  // everybody is done with the previous tile; the new rows are in shared memory
#pragma unroll
    for (int i = 0; i < kPerThread; ++i) {
      const int u = tid + i * 256;
      if (u < units) {
        const bool fresh = t0 + u / kRowU4 == pos;
        reinterpret_cast<uint4*>(s_k)[u] = fresh ? reinterpret_cast<const uint4*>(s_newk)[u % kRowU4] : kv[i];
        reinterpret_cast<uint4*>(s_v)[u] = fresh ? reinterpret_cast<const uint4*>(s_newv)[u % kRowU4] : vv[i];
      }
    }
    __syncthreads();
    if (warp < rep) {
      for (int r = 0; r < rows; ++r) {
        float s = 0.f, kf[E], vf[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
          kf[e] = __bfloat162float(s_k[r * D + lane * E + e]);
          vf[e] = __bfloat162float(s_v[r * D + lane * E + e]);
        }
#pragma unroll
        for (int e = 0; e < E; ++e) s += qf[e] * kf[e];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const float mn = fmaxf(m, s);
        const float corr = __expf(m - mn), pj = __expf(s - mn);
        l = l * corr + pj;
#pragma unroll
        for (int e = 0; e < E; ++e) acc[e] = acc[e] * corr + pj * vf[e];
        m = mn;
      }
    }
  }
  if (warp < rep) {
    float* o = part + ((size_t)h * kSplits + sp) * (D + 2);
    if (lane == 0) {
      __stcg(o, m);
      __stcg(o + 1, l);
    }
#pragma unroll
    for (int e = 0; e < E; ++e) __stcg(o + 2 + lane * E + e, acc[e]);
  }

  if (counters == nullptr) return;  // a merge launch follows
  // ---- the last CTA of this KV head to arrive merges the splits
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    const int old = atomicAdd(counters + kh, 1);
    const int last = old == kSplits - 1;
    if (last) counters[kh] = 0;  // ready for the next launch (launches that share the counters are stream-ordered)
    s_last = last;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // weight of every (query head, split): exp(m - max m), and the denominator of every head
  if (warp < rep) {
    const int hq = kh * rep + warp;
    const float* pp = part + ((size_t)hq * kSplits + lane) * (D + 2);  // kSplits == 32: one split per lane
    const float ms = __ldcg(pp), ls = __ldcg(pp + 1);
    float mm = ms;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, o));
    const float f = ms == -FLT_MAX ? 0.f : __expf(ms - mm);
    float den = f * ls;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
    s_f[warp * kSplits + lane] = f;
    if (lane == 0) s_den[warp] = den;
  }
  __syncthreads();
  for (int item = tid; item < rep * D; item += 256) {
    const int w = item / D, d = item - w * D;
    const int hq = kh * rep + w;
    const float* pp = part + (size_t)hq * kSplits * (D + 2) + 2 + d;
    float as[kSplits];
#pragma unroll
    for (int sidx = 0; sidx < kSplits; ++sidx) as[sidx] = __ldcg(pp + sidx * (D + 2));
    float num = 0.f;
#pragma unroll
    for (int sidx = 0; sidx < kSplits; ++sidx) num += s_f[w * kSplits + sidx] * as[sidx];
    const float den = s_den[w];
    out[(size_t)hq * D + d] = __float2bfloat16(den > 0.f ? num / den : 0.f);
  }
}

// The same in one launch without a last CTA to wait for: the sixteen CTAs of a KV head are a cluster and send their partials to
// the CTA that merges them (st.async, counted on a barrier of that CTA; CTA r merges dimensions [r D/16, (r + 1) D/16) of every
// head).  A CTA holds two of the 32 slices, a warp one (query head, slice); every sum is taken over the same values in the same
// order as in the pass and the merge launch of the two-launch form, so the results are that form's to the bit.
// What bounds it is latency: 0.6 us until the kernel in front is seen complete, 0.6 for q's load and the rotation, 2 for the rows of a
// slice, one way through the cluster 0.5, the merge 0.5.  A layer's attention at 560 positions, alone in a chain: 8.6 us in two
// launches, 5.6 in this one; a decode step of 28 layers 1.567 -> 1.490 ms.  On the way: eight CTAs of 28 warps found no place beside a
// GEMV's CTA and started late (1.620 ms); a butterfly per row and an exponential per row and warp took 270 cycles a row.
// With many positions it is a warp's chain over its rows, 32 to a pass: the next pass's rows are on their way meanwhile, into a second
// stage (loaded behind the pass they cost 28 query and 4 KV heads 21.6 us at 4096 positions, now 19.0, and made long contexts of
// few heads slower than the two launches: 7 and 1 head at 32768 154 us, now 126, there 141; 1 and 1 152, now 121, there 129).
constexpr int kAttnCtas = 16, kSlicesPerCta = kSplits / kAttnCtas;
template <int D>
struct AttnSmem {  // offsets of the dynamic shared memory
  static constexpr int kTile = kSlicesPerCta * kTileRows * D * 2;  // K or V rows of a pass
  static constexpr int kStage = 2 * kTile;                         // both; the next pass's are loaded beside them
  static constexpr int kNew = 2 * kStage;                          // the new k and v row
  static constexpr int kMaxSum = kNew + 4 * D;                     // [head][slice] maximum and sum
  static constexpr int kPart = kMaxSum + 8 * kSplits * 8;          // [head][slice][D / 16] un-normalised
  static constexpr int kRot = kPart + 8 * kSplits * (D / kAttnCtas) * 4;  // sine and cosine of the new position
  // More than half of an SM, so that no SM takes two of these CTAs while others have none, and less than a CTA of the streaming
  // GEMV, a decode step's other kernel (112 KB), leaves: it is there early, and the next kernel's beside it.  (1.513 -> 1.490 ms per
  // token.  The half-SM CTAs of the other GEMVs, 113 KB, find no place beside it: two halves and no more make a whole.)
  static constexpr int kBytes = 116224;
  static_assert(kRot + D / 2 * 8 <= kBytes, "shared memory");
};
// E (2 or 4) consecutive bf16 of shared memory as floats.
template <int E>
__device__ __forceinline__ void lds_row(const bf16* p, float (&f)[E]) {
  if constexpr (E == 4) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    f[0] = __uint_as_float(v.x << 16);
    f[1] = __uint_as_float(v.x & 0xFFFF0000u);
    f[2] = __uint_as_float(v.y << 16);
    f[3] = __uint_as_float(v.y & 0xFFFF0000u);
  } else {
    const unsigned v = *reinterpret_cast<const unsigned*>(p);
    f[0] = __uint_as_float(v << 16);
    f[1] = __uint_as_float(v & 0xFFFF0000u);
  }
}
template <int E>
__device__ __forceinline__ void send_part(uint32_t addr, uint32_t bar, uint32_t rank, const float (&a)[E]) {
  if constexpr (E == 4) b2::st_async_f4(addr, bar, rank, a[0], a[1], a[2], a[3]);
  else b2::st_async_f2(addr, bar, rank, a[0], a[1]);
}

template <int D>
__global__ void __launch_bounds__(512, 2) decode_attention_cluster_kernel(
    const bf16* qkv, const bf16* __restrict__ bias, const float* __restrict__ inv_freq, const int* pos_ptr,
    bf16* cache_k, bf16* cache_v, bf16* out, int Hq, int Hk, int max_len, float scale, int early, int* status) {
  constexpr int E = D / 32;        // elements per lane
  constexpr int kRowU4 = D / 8;    // 16-byte units per row
  constexpr int half = D / 2, kMine = D / kAttnCtas;
  using S = AttnSmem<D>;
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ __align__(8) unsigned long long s_bar;
  __shared__ int s_abort;
  const uint32_t base = b2::smem_u32(sm), bar = b2::smem_u32(&s_bar);
  bf16* s_newk = reinterpret_cast<bf16*>(sm + S::kNew);
  bf16* s_newv = s_newk + D;
  const int crank = (int)b2::cluster_rank(), kh = blockIdx.x / kAttnCtas;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rep = Hq / Hk;
  const int slice = warp / rep, w = warp - slice * rep, sp = crank * kSlicesPerCta + slice;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (tid == 0) {
    s_abort = 0;
    b2::mbar_init(bar, 1);
    b2::mbar_arrive_expect_tx(bar, (uint32_t)(rep * kSplits) * (kMine * 4 + 8));
    b2::fence_mbar_init();
  }
  __syncthreads();
  b2::cluster_arrive();  // (waited for before the first store into a peer: its barrier is set up)

  const uint4* kbase = reinterpret_cast<const uint4*>(cache_k + (size_t)kh * max_len * D);
  const uint4* vbase = reinterpret_cast<const uint4*>(cache_v + (size_t)kh * max_len * D);
  int pos = 0, n = 0, per = 0;
  auto find = [&]() {
    pos = __ldcg(pos_ptr);
    n = min(pos + 1, max_len);
    per = (n + kSplits - 1) / kSplits;
  };
  // rows [t0, t0 + kTileRows) of each of the CTA's slices, copied past the registers; the row that this launch appends is not in
  // the cache yet
  auto request = [&](int t0, int stage) {
    const int rows = min(kTileRows, per - t0), units = kSlicesPerCta * rows * kRowU4;
    for (int u = tid; u < units; u += blockDim.x) {
      static_assert(kSlicesPerCta == 2, "no division");
      const int c = u % kRowU4, r = u / kRowU4, sl = r >= rows, j = (crank * kSlicesPerCta + sl) * per + t0 + (r - sl * rows);
      if (j < n && j != pos) {
        const uint32_t dst = base + stage * S::kStage + ((sl * kTileRows + (r - sl * rows)) * kRowU4 + c) * 16;
        b2::cp_async_cg16(dst, kbase + (size_t)j * kRowU4 + c);
        b2::cp_async_cg16(dst + S::kTile, vbase + (size_t)j * kRowU4 + c);
      }
    }
  };
  // `early`: the position and the cached rows below it were written by earlier steps, not by the kernel in front of this one
  if (early) {
    find();
    request(0, 0);
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (!early) {
    find();
    request(0, 0);
  }
  const int j0 = sp * per, j1 = min(n, j0 + per);

  // ---- this warp's query head; the rotation's sines and cosines once per CTA
  const int h = kh * rep + w;
  float2* s_rot = reinterpret_cast<float2*>(sm + S::kRot);
  float qf[E], qb[E];
  ld_row<E>(qkv + (size_t)h * D + lane * E, qf);
#pragma unroll
  for (int e = 0; e < E; ++e) qb[e] = bias != nullptr ? __bfloat162float(bias[(size_t)h * D + lane * E + e]) : 0.f;
  for (int i = tid; i < half; i += blockDim.x) {
    float sn, cs;
    sincosf((float)pos * inv_freq[i], &sn, &cs);
    s_rot[i] = make_float2(sn, cs);
  }
  __syncthreads();
  // ---- the new k and v rows, in the CTA whose slices hold the new position: i < D/2 rotates the pair (i, i + D/2) of k, the
  // next D/2 add the bias to a pair of v
  for (int t = tid; pos < max_len && pos / per / kSlicesPerCta == crank && t < D; t += blockDim.x) {
    const bool is_v = t >= half;
    const int i = is_v ? t - half : t;
    const int hh = Hq + (is_v ? Hk : 0) + kh;
    const bf16* x = qkv + (size_t)hh * D;
    float a = ld_bf16(x + i), b = ld_bf16(x + i + half);
    if (bias != nullptr) {
      a = __bfloat162float(__float2bfloat16(a + __bfloat162float(bias[(size_t)hh * D + i])));
      b = __bfloat162float(__float2bfloat16(b + __bfloat162float(bias[(size_t)hh * D + i + half])));
    }
    if (!is_v) {
      rotate_pair(a, b, s_rot[i].x, s_rot[i].y);
    }
    const bf16 oa = __float2bfloat16(a), ob = __float2bfloat16(b);
    bf16* row = is_v ? s_newv : s_newk;
    row[i] = oa;
    row[i + half] = ob;
    bf16* dst = (is_v ? cache_v : cache_k) + ((size_t)kh * max_len + pos) * D;
    dst[i] = oa;
    dst[i + half] = ob;
  }
  // ---- bias, rotation, bf16 rounding, softmax scale
  if (bias != nullptr) {
#pragma unroll
    for (int e = 0; e < E; ++e) qf[e] = __bfloat162float(__float2bfloat16(qf[e] + qb[e]));
  }
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const float other = __shfl_xor_sync(0xffffffffu, qf[e], 16);  // the element D/2 away
    const float2 rot = s_rot[(lane * E + e) % half];
    qf[e] = __bfloat162float(__float2bfloat16(rotate_query(qf[e], other, rot.x, rot.y, lane < 16))) * scale;
  }

  float m = -FLT_MAX, l = 0.f, acc[E];
#pragma unroll
  for (int e = 0; e < E; ++e) acc[e] = 0.f;
  for (int t0 = 0, stage = 0; t0 < per; t0 += kTileRows, stage ^= 1) {
    b2::cp_async_wait_all();
    __syncthreads();  // the pass's rows are there, and everybody is done with those of the last one
    if (t0 + kTileRows < per) request(t0 + kTileRows, stage ^ 1);
    unsigned char* tile = sm + stage * S::kStage;
    // the new row into its place in the pass that holds it
    if (const int r = pos - t0 - (crank * kSlicesPerCta + pos / per % kSlicesPerCta) * per;
        pos < max_len && pos / per / kSlicesPerCta == crank && r >= 0 && r < kTileRows) {
      const int at = (pos / per % kSlicesPerCta * kTileRows + r) * kRowU4;
      for (int u = tid; u < 2 * kRowU4; u += blockDim.x)
        *reinterpret_cast<uint4*>(tile + (u < kRowU4 ? 0 : S::kTile) + (at + u % kRowU4) * 16) =
            reinterpret_cast<const uint4*>(s_newk)[u];
      __syncthreads();
    }
    const int rows = min(kTileRows, j1 - j0 - t0);
    const bf16* tk = reinterpret_cast<const bf16*>(tile) + slice * kTileRows * D + lane * E;
    const bf16* tv = tk + S::kTile / 2;
    // Eight rows at a time.  A row's parts are added over the lanes as one tree, as a butterfly would; each of its first three steps
    // halves the rows that a lane goes on with (9 exchanges for the 40 of eight butterflies), and row q ends in lanes 4 q to
    // 4 q + 3.  There the running maxima are a scan and the exponentials of all rows one instruction; only the products and sums
    // that depend on one another go row by row.
    for (int r0 = 0; r0 < rows; r0 += 8, tk += 8 * D, tv += 8 * D) {
      float x[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {  // (what rows behind the slice's end hold is not used)
        float kf[E];
        lds_row<E>(tk + q * D, kf);
        x[q] = 0.f;
#pragma unroll
        for (int e = 0; e < E; ++e) x[q] += qf[e] * kf[e];
      }
#pragma unroll
      for (int o = 16, k = 4; o >= 4; o >>= 1, k >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int q = 0; q < k; ++q) {
          const float give = up ? x[q] : x[q + k], keep = up ? x[q + k] : x[q];
          x[q] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
      }
      float sq = x[0];
      sq += __shfl_xor_sync(0xffffffffu, sq, 2);
      sq += __shfl_xor_sync(0xffffffffu, sq, 1);
      float mn = sq;
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) {
        const float before = __shfl_up_sync(0xffffffffu, mn, o);
        if (lane >= o) mn = fmaxf(before, mn);
      }
      mn = fmaxf(m, mn);
      const float last = __shfl_up_sync(0xffffffffu, mn, 4), mp = lane < 4 ? m : last;
      const float corr = __expf(mp - mn), pj = __expf(sq - mn);
      const int count = min(8, rows - r0);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (q >= count) break;
        const float c = __shfl_sync(0xffffffffu, corr, q * 4), pq = __shfl_sync(0xffffffffu, pj, q * 4);
        float vf[E];
        lds_row<E>(tv + q * D, vf);
        l = l * c + pq;
#pragma unroll
        for (int e = 0; e < E; ++e) acc[e] = acc[e] * c + pq * vf[e];
      }
      m = __shfl_sync(0xffffffffu, mn, (count - 1) * 4);
    }
  }

  // ---- partials to the CTAs that merge them: lanes 2 r and 2 r + 1 hold the dimensions of CTA r
  b2::cluster_wait();
  send_part<E>(base + S::kPart + ((w * kSplits + sp) * kMine + lane % (32 / kAttnCtas) * E) * 4, bar, lane / (32 / kAttnCtas), acc);
  if (lane < kAttnCtas) b2::st_async_f2(base + S::kMaxSum + (w * kSplits + sp) * 8, bar, lane, m, l);
  if (warp < rep) {  // a warp merges a head: a lane a slice's weight, then a lane a dimension
    b2::mbar_wait(bar, 0, &s_abort);
    __syncwarp();
    float2* ml = reinterpret_cast<float2*>(sm + S::kMaxSum) + warp * kSplits;
    const float* as = reinterpret_cast<const float*>(sm + S::kPart) + warp * kSplits * kMine + lane % kMine;
    const float2 mine = ml[lane];
    float mm = mine.x;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, o));
    ml[lane].x = mine.x == -FLT_MAX ? 0.f : __expf(mine.x - mm);
    __syncwarp();
    float num = 0.f, den = 0.f;
#pragma unroll 16
    for (int z = 0; z < kSplits; ++z) {
      const float2 f = ml[z];
      num += f.x * as[z * kMine];
      den += f.x * f.y;
    }
    if (lane < kMine) out[(size_t)(kh * rep + warp) * D + crank * kMine + lane] = __float2bfloat16(den > 0.f ? num / den : 0.f);
  }
  __syncthreads();
  if (s_abort) {  // a peer never sent: nothing may come in after this CTA has left
    b2::cluster_arrive();
    b2::cluster_wait();
    if (tid == 0) atomicCAS(status, 0, b2::kStatusGemvTimeout);
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
  }
}

// Greedy choice in two launches.  Pass 1, kArgBlocks CTAs: each scans a slice of the logits and writes its best
// (value, index).  Pass 2, one CTA: picks the best of those (lowest index on ties, as torch.argmax returns the
// first occurrence), records the token, advances step and position, and copies the token's embedding row.
constexpr int kArgBlocks = 148;

__device__ __forceinline__ void argmax_merge(float& best, int& bi, float ov, int oi) {
  if (ov > best || (ov == best && oi < bi)) {
    best = ov;
    bi = oi;
  }
}

__global__ void __launch_bounds__(256) argmax_partial_kernel(const bf16* __restrict__ logits, int V,
                                                             float* __restrict__ pv, int* __restrict__ pi) {
  __shared__ float s_v[8];
  __shared__ int s_i[8];
  float best = -FLT_MAX;
  int bi = 0x7fffffff;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < V; i += gridDim.x * blockDim.x) {
    const float v = __bfloat162float(logits[i]);
    if (v > best) {  // indices ascend within a thread, so the first occurrence is kept
      best = v;
      bi = i;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    argmax_merge(best, bi, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, bi, o));
  if ((threadIdx.x & 31) == 0) {
    s_v[threadIdx.x >> 5] = best;
    s_i[threadIdx.x >> 5] = bi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) argmax_merge(best, bi, s_v[w], s_i[w]);
    pv[blockIdx.x] = best;
    pi[blockIdx.x] = bi;
  }
}

// One CTA, between the vocabulary projection and the next step's first kernel, so its latencies are the step's: as many threads as
// parts, the embedding row in 16-byte pieces, launched programmatically (10.7 -> 4.9 us after 1188 parts).
constexpr int kFinishThreads = 1024;
__global__ void __launch_bounds__(kFinishThreads) greedy_finish_kernel(const float* pv, const int* pi, int nparts, int V,
                                                                       const bf16* embed, int H, int* pos_ptr,
                                                                       long long* out_tokens, int* step_ptr, bf16* x_next) {
  constexpr int kWarps = kFinishThreads / 32;
  __shared__ float s_v[kWarps];
  __shared__ int s_i[kWarps];
  __shared__ int s_tok;
  float best = -FLT_MAX;
  int bi = 0x7fffffff, step = 0, pos = 0;
  // (its dependents start when it has ended: the attention of the next step, behind a kernel that lets its own start at once, reads
  // the position without a wait)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (threadIdx.x == 0) {
    step = __ldcg(step_ptr);
    pos = __ldcg(pos_ptr);
  }
  for (int i = threadIdx.x; i < nparts; i += kFinishThreads) argmax_merge(best, bi, __ldcg(pv + i), __ldcg(pi + i));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    argmax_merge(best, bi, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, bi, o));
  if ((threadIdx.x & 31) == 0) {
    s_v[threadIdx.x >> 5] = best;
    s_i[threadIdx.x >> 5] = bi;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    best = s_v[threadIdx.x];
    bi = s_i[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      argmax_merge(best, bi, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, bi, o));
    if (threadIdx.x == 0) {
      if (bi < 0 || bi >= V) bi = 0;
      s_tok = bi;
      out_tokens[step] = bi;
      *step_ptr = step + 1;
      *pos_ptr = pos + 1;
    }
  }
  __syncthreads();
  const bf16* row = embed + (size_t)s_tok * H;
  if (((reinterpret_cast<uintptr_t>(embed) | reinterpret_cast<uintptr_t>(x_next)) & 15) == 0 && H % 8 == 0) {
    for (int i = threadIdx.x; i < H / 8; i += kFinishThreads)
      reinterpret_cast<uint4*>(x_next)[i] = __ldcg(reinterpret_cast<const uint4*>(row) + i);
  } else {
    for (int i = threadIdx.x; i < H; i += kFinishThreads)
      reinterpret_cast<unsigned short*>(x_next)[i] = __ldcg(reinterpret_cast<const unsigned short*>(row) + i);
  }
}

}  // namespace

// One thread waits (bounded) for an arrival counter of a fused all-gather: kernels that follow on the stream may then
// read the gathered rows without a wait of their own.
__global__ void tp_wait_kernel(const unsigned* wait_sig, int* epoch, unsigned wait_per_epoch, int* status,
                               const b2::GemvTp ann, int advance_epoch) {
  // deferred signal of the kernel in front of this one (complete: plain stream order), one thread per rank
  if (threadIdx.x < ann.announce_world)
    asm volatile("red.release.sys.global.add.u32 [%0], 1;" ::"l"(ann.announce_peer[threadIdx.x]) : "memory");
  if (threadIdx.x != 0) return;
  const unsigned target = ((unsigned)*reinterpret_cast<const volatile int*>(epoch) + 1u) * wait_per_epoch;
  const long long t0 = clock64();
  for (;;) {
    unsigned v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(wait_sig) : "memory");
    if ((int)(v - target) >= 0) break;
    if (clock64() - t0 > 1000000000LL) {
      if (status != nullptr) atomicCAS(status, 0, b2::kStatusGemvTimeout);
      break;
    }
    __nanosleep(40);
  }
  if (advance_epoch) *epoch += 1;  // the use of the counters that this wait closes is over
}

namespace b2 {
int tp_wait_launch(const void* wait_sig, const void* epoch, unsigned wait_per_epoch, int* status, cudaStream_t stream,
                   const GemvTp* announce, int advance_epoch) {
  if (!wait_sig || !epoch) return kErrBadPointer;
  GemvTp ann;
  if (announce != nullptr) ann = *announce;
  tp_wait_kernel<<<1, 32, 0, stream>>>(static_cast<const unsigned*>(wait_sig),
                                       static_cast<int*>(const_cast<void*>(epoch)), wait_per_epoch, status, ann,
                                       advance_epoch);
  return (int)cudaGetLastError();
}
int rope_kv_store_launch(void* qkv, const void* bias, const void* inv_freq, const void* pos, void* cache_k,
                         void* cache_v, int Hq, int Hk, int D, int max_len, const void* wait_sig, const void* epoch,
                         unsigned wait_per_epoch, int* status, cudaStream_t stream) {
  if (Hq < 1 || Hk < 1 || D < 2 || D % 2 || D / 2 > 1024 || max_len < 1) return kErrBadShape;
  if (!qkv || !inv_freq || !pos || !cache_k || !cache_v) return kErrBadPointer;
  if (wait_sig != nullptr && !epoch) return kErrBadPointer;
  // the kernel moves bf16 pairs: 4-byte alignment of the activations, the bias and the caches
  if ((reinterpret_cast<uintptr_t>(qkv) & 3) || (reinterpret_cast<uintptr_t>(bias) & 3) ||
      (reinterpret_cast<uintptr_t>(cache_k) & 3) || (reinterpret_cast<uintptr_t>(cache_v) & 3) ||
      (reinterpret_cast<uintptr_t>(inv_freq) & 3) || (reinterpret_cast<uintptr_t>(pos) & 3))
    return kErrBadPointer;
  const cudaError_t e = launch_pdl(rope_kv_store_kernel, dim3(Hq + 2 * Hk), dim3(D / 2), stream,
                                   static_cast<bf16*>(qkv), static_cast<const bf16*>(bias),
                                   static_cast<const float*>(inv_freq), static_cast<const int*>(pos),
                                   static_cast<bf16*>(cache_k), static_cast<bf16*>(cache_v), Hq, Hk, D, max_len,
                                   static_cast<const unsigned*>(wait_sig), static_cast<const int*>(epoch),
                                   wait_per_epoch, status);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}
}  // namespace b2

namespace b2 {
int decode_attention_fused_launch(const void* qkv, const void* bias, const void* inv_freq, const void* pos,
                                  void* cache_k, void* cache_v, void* out, void* workspace, int Hq, int Hk, int D,
                                  int max_len, const GemvTp* tp, int flags, int* status, cudaStream_t stream) {
  static_assert(kSplits == 32, "the merge takes one split per lane");
  if (Hq < 1 || Hk < 1 || Hq % Hk || Hq / Hk > 8 || max_len < 1) return b2::kErrBadShape;
  if (D != 128 && D != 64) return b2::kErrNotImplemented;
  if (!qkv || !inv_freq || !cache_k || !cache_v || !pos || !out || !workspace) return b2::kErrBadPointer;
  GemvTp ann;
  if (tp != nullptr) ann = *tp;
  const void* wait_sig = ann.wait_sig;
  const void* epoch = ann.epoch;
  const unsigned wait_per_epoch = ann.wait_per_epoch;
  if (wait_sig != nullptr && !epoch) return b2::kErrBadPointer;
  // 8-byte loads of q, 16-byte loads and stores of cache rows, float partials and counters in the workspace
  if ((reinterpret_cast<uintptr_t>(qkv) & 7) || (reinterpret_cast<uintptr_t>(bias) & 3) ||
      (reinterpret_cast<uintptr_t>(cache_k) & 15) || (reinterpret_cast<uintptr_t>(cache_v) & 15) ||
      (reinterpret_cast<uintptr_t>(out) & 1) || (reinterpret_cast<uintptr_t>(workspace) & 3) ||
      (reinterpret_cast<uintptr_t>(pos) & 3) || (reinterpret_cast<uintptr_t>(inv_freq) & 3))
    return b2::kErrBadPointer;
  const float scale = 1.f / sqrtf((float)D);
  float* part = static_cast<float*>(workspace);
  const bool one_launch = (flags & 1) != 0;
  int* counters = one_launch ? reinterpret_cast<int*>(part + (size_t)Hq * kSplits * (D + 2)) : nullptr;
  const dim3 grid(Hk, kSplits);
  // The cluster form where all of the call's clusters run at once: a CTA takes an SM, so that a second wave costs as much as the
  // first, where the two launches keep several small CTAs to an SM.  The line is the device's count of clusters of sixteen (seven on
  // a B200; none on a slice of one).  us per layer in a chain, this form and in brackets the two launches, 512 / 4096 positions,
  // heads of 128: 28 query and 4 KV heads 5.8 / 19.0 (8.2 / 34.7), 28 and 7 5.7 / 16.5 (7.4 / 24.7); with two waves and more, a
  // pass's rows loaded behind the last pass, 32 and 8 10.1 / 36.4 (7.2 / 23.5), 32 and 32 27.7 / 108 (11.9 / 41.0).
  // Its waits for the peers are bounded, so it needs the device's status word; the two launches wait for nobody, and run where the
  // word does not exist yet (a first call, under capture perhaps, where it could not be made).
  int* const word = tp == nullptr ? device_status_word_if_ready() : nullptr;
  if (!one_launch && word != nullptr && (flags & 4) == 0) {
    static std::atomic<int> clusters_on[2][64];  // one more than their number: asked once
    int dev = -1;
    if (const cudaError_t e = cudaGetDevice(&dev); e != cudaSuccess) return (int)e;
    auto cluster = [&](auto kernel, int smem, bool* fits) {
      cudaLaunchConfig_t cfg{};
      cfg.dynamicSmemBytes = smem;
      cfg.stream = stream;
      cudaLaunchAttribute attr[2];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = kAttnCtas;
      attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
      attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[1].val.programmaticStreamSerializationAllowed = 1;
      cfg.attrs = attr;
      const bool cached = dev >= 0 && dev < 64;
      int known = cached ? clusters_on[D == 128][dev].load(std::memory_order_acquire) : 0;
      if (known == 0) {
        int clusters = 0;
        cfg.numAttrs = 1;
        cfg.gridDim = dim3(kAttnCtas);
        cfg.blockDim = dim3(8 * kSlicesPerCta * 32);  // the most heads that share a KV head
        const bool asked = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess &&
                           cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                           cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess;
        if (!asked) (void)cudaGetLastError();
        known = asked ? clusters + 1 : 1;
        if (cached) clusters_on[D == 128][dev].store(known, std::memory_order_release);
      }
      *fits = Hk < known;
      if (!*fits) return cudaSuccess;
      cfg.gridDim = dim3(Hk * kAttnCtas);
      cfg.blockDim = dim3(Hq / Hk * kSlicesPerCta * 32);
      cfg.numAttrs = 2;
      return cudaLaunchKernelEx(&cfg, kernel, static_cast<const bf16*>(qkv), static_cast<const bf16*>(bias),
                                static_cast<const float*>(inv_freq), static_cast<const int*>(pos),
                                static_cast<bf16*>(cache_k), static_cast<bf16*>(cache_v), static_cast<bf16*>(out), Hq, Hk,
                                max_len, scale, (flags & 2) ? 1 : 0, word);
    };
    bool fits = false;
    const cudaError_t e = D == 128 ? cluster(decode_attention_cluster_kernel<128>, AttnSmem<128>::kBytes, &fits)
                                   : cluster(decode_attention_cluster_kernel<64>, AttnSmem<64>::kBytes, &fits);
    if (e != cudaSuccess || fits) return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
  }
  auto go = [&](auto kernel) {
    return launch_pdl(kernel, grid, dim3(256), stream, static_cast<const bf16*>(qkv),
                      static_cast<const bf16*>(bias), static_cast<const float*>(inv_freq),
                      static_cast<const int*>(pos), static_cast<bf16*>(cache_k), static_cast<bf16*>(cache_v), part,
                      counters, static_cast<bf16*>(out), Hq, Hk, max_len, scale,
                      static_cast<const unsigned*>(wait_sig), static_cast<const int*>(epoch), wait_per_epoch, status,
                      ann, (flags & 2) ? 1 : 0);
  };
  cudaError_t e = D == 128 ? go(decode_attention_fused_kernel<128>) : go(decode_attention_fused_kernel<64>);
  if (e == cudaSuccess && !one_launch) {
    e = D == 128 ? launch_pdl(decode_attention_merge_kernel<128>, dim3(Hq), dim3(128), stream,
                              static_cast<const float*>(part), static_cast<bf16*>(out))
                 : launch_pdl(decode_attention_merge_kernel<64>, dim3(Hq), dim3(64), stream,
                              static_cast<const float*>(part), static_cast<bf16*>(out));
  }
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}
}  // namespace b2

extern "C" {

int b2_rope_kv_store(void* qkv, const void* bias, const void* inv_freq, const void* pos, void* cache_k, void* cache_v,
                     int Hq, int Hk, int D, int max_len, void* stream) {
  return b2::rope_kv_store_launch(qkv, bias, inv_freq, pos, cache_k, cache_v, Hq, Hk, D, max_len, nullptr, nullptr, 0,
                                  nullptr, static_cast<cudaStream_t>(stream));
}

size_t b2_decode_workspace_bytes(int Hq, int D) {
  const size_t attn = (size_t)Hq * kSplits * (D + 2) * sizeof(float);
  const size_t arg = (size_t)kArgBlocks * (sizeof(float) + sizeof(int));
  return attn > arg ? attn : arg;
}

int b2_decode_attention(const void* q, const void* cache_k, const void* cache_v, const void* pos, void* out,
                        void* workspace, int Hq, int Hk, int D, int max_len, void* stream) {
  if (Hq < 1 || Hk < 1 || Hq % Hk || Hq / Hk > 8 || max_len < 1) return b2::kErrBadShape;
  if (D != 128 && D != 64) return b2::kErrNotImplemented;
  if (!q || !cache_k || !cache_v || !pos || !out || !workspace) return b2::kErrBadPointer;
  // 8-byte loads of q, 16-byte loads of the cache rows, float partials in the workspace
  if ((reinterpret_cast<uintptr_t>(q) & 7) || (reinterpret_cast<uintptr_t>(cache_k) & 15) ||
      (reinterpret_cast<uintptr_t>(cache_v) & 15) || (reinterpret_cast<uintptr_t>(out) & 1) ||
      (reinterpret_cast<uintptr_t>(workspace) & 3) || (reinterpret_cast<uintptr_t>(pos) & 3))
    return b2::kErrBadPointer;
  const float scale = 1.f / sqrtf((float)D);
  const auto st = static_cast<cudaStream_t>(stream);
  float* part = static_cast<float*>(workspace);
  const dim3 grid(Hk, kSplits);
  if (D == 128) {
    launch_pdl(decode_attention_partial_kernel<128>, grid, dim3(256), st, static_cast<const bf16*>(q),
               static_cast<const bf16*>(cache_k), static_cast<const bf16*>(cache_v), static_cast<const int*>(pos), part,
               Hq, Hk, max_len, scale);
    launch_pdl(decode_attention_merge_kernel<128>, dim3(Hq), dim3(128), st, static_cast<const float*>(part),
               static_cast<bf16*>(out));
  } else {
    launch_pdl(decode_attention_partial_kernel<64>, grid, dim3(256), st, static_cast<const bf16*>(q),
               static_cast<const bf16*>(cache_k), static_cast<const bf16*>(cache_v), static_cast<const int*>(pos), part,
               Hq, Hk, max_len, scale);
    launch_pdl(decode_attention_merge_kernel<64>, dim3(Hq), dim3(64), st, static_cast<const float*>(part),
               static_cast<bf16*>(out));
  }
  return (int)cudaGetLastError();
}

size_t b2_decode_attention_fused_workspace_bytes(int Hq, int Hk, int D) {
  return (size_t)Hq * kSplits * (D + 2) * sizeof(float) + (size_t)Hk * sizeof(int);
}

int b2_greedy_next(const void* logits, int V, const void* embed, int H, void* pos, void* out_tokens, void* step,
                   void* x_next, void* workspace, void* stream) {
  if (V < 1 || H < 1) return b2::kErrBadShape;
  if (!logits || !embed || !pos || !out_tokens || !step || !x_next || !workspace) return b2::kErrBadPointer;
  const auto st = static_cast<cudaStream_t>(stream);
  float* pv = static_cast<float*>(workspace);
  int* pi = reinterpret_cast<int*>(pv + kArgBlocks);
  argmax_partial_kernel<<<kArgBlocks, 256, 0, st>>>(static_cast<const bf16*>(logits), V, pv, pi);
  const cudaError_t e = launch_pdl(greedy_finish_kernel, dim3(1), dim3(kFinishThreads), st, static_cast<const float*>(pv),
                                   static_cast<const int*>(pi), (int)kArgBlocks, V, static_cast<const bf16*>(embed), H,
                                   static_cast<int*>(pos), static_cast<long long*>(out_tokens), static_cast<int*>(step),
                                   static_cast<bf16*>(x_next));
  if (e != cudaSuccess) return (int)e;
  return (int)cudaGetLastError();
}

// Second half of b2_greedy_next for callers whose logits kernel already reduced blocks of the vocabulary
// (b2_lm_head): picks the largest of `nparts` (value, index) pairs, lowest index on ties, then does what
// b2_greedy_next does with the token.
int b2_greedy_pick(const void* part_max, const void* part_idx, int nparts, int V, const void* embed, int H, void* pos,
                   void* out_tokens, void* step, void* x_next, void* stream) {
  if (V < 1 || H < 1 || nparts < 1) return b2::kErrBadShape;
  if (!part_max || !part_idx || !embed || !pos || !out_tokens || !step || !x_next) return b2::kErrBadPointer;
  const cudaError_t e = launch_pdl(greedy_finish_kernel, dim3(1), dim3(kFinishThreads), static_cast<cudaStream_t>(stream),
                                   static_cast<const float*>(part_max), static_cast<const int*>(part_idx), nparts, V,
                                   static_cast<const bf16*>(embed), H, static_cast<int*>(pos),
                                   static_cast<long long*>(out_tokens), static_cast<int*>(step), static_cast<bf16*>(x_next));
  if (e != cudaSuccess) return (int)e;
  return (int)cudaGetLastError();
}

}  // extern "C"
