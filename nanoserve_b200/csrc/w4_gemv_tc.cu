// W4A16 decode GEMV on the fifth-generation tensor cores, nine to sixteen tokens, groups of 128:
// Y[M,N] (bf16) = X[M,K] (bf16) . dequant(Wq, S)^T with exact weights.
//
// The arithmetic is that of w4_gemv_mid.cu: nibbles as signed bytes 16 (q - 8), X as block fixed point per (token,
// 128-chunk) in an unsigned low and a signed high byte plane, integer products, one conversion to float and one fused
// multiply-add per (row, token, chunk).  There the products run on mma.sync and the loop is bound by shared-memory reads of
// X's fragments and by issue slots.  Here they run on tcgen05.mma (kind::i8) in the frame of w4_gemm_narrow.cu:
//   * 128 weight rows are the M side; the bytes go from registers to tensor memory (three instructions per eight
//     weights; a thread owns a row) and the MMA reads them there.  The byte order the nibble masks give is the order X is
//     stored in: the contraction index is a dummy;
//   * the planes of the CTA's K range stay in shared memory as the N side, 16 token columns each, read by the tensor core
//     only;
//   * a step is one chunk.  Its integer sums start at zero and a group of warps converts and scales them while the next
//     step's products run: the wait for its buffer of bytes is also the wait for the sums of that buffer's last use;
//   * K is cut over a cluster and summed through distributed shared memory in rank order (no second launch).
// Measured at 13 tokens against the mma.sync kernel, weights from HBM, us: 37888 x 3584 21.7 (25.9), 3584 x 18944 18.1
// (20.8), 3584 x 3584 7.8 (9.4), 10240 x 8192 19.2 (24.6), 14336 x 4096 14.6 (17.6).  What bounds it: about 0.6 us per step
// of 256 rows, the chain of a group's waits, TMEM stores and loads and 16 int-to-float conversions per row.  One product
// instruction for both planes (the high one offset to unsigned, corrected by the rows' weight sums) was 5 % slower.
// Every wait is bounded; a CTA that gives up records a status, still takes part in the cluster barriers and frees its TMEM.
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <cstdio>

#include "ptx.cuh"
#include "tensor_map.h"
#include "w4_common.cuh"
#include "w4_internal.h"

namespace b2 {
namespace {

constexpr int kStepK = 128;
constexpr int kMaxSlots = 8;
constexpr int kTokens = 16;
constexpr int kHeaderBytes = 1024;
constexpr int kXStep = 2 * kTokens * 128;   // bytes of a step's two planes
constexpr int kInfoStep = kTokens * 4;      // and of its factors
constexpr int kSmemHalf = 115712, kSmemFull = 232448;
constexpr int kBufs = 2;      // bytes and sums of two steps in TMEM, one per group of warps (two each were no faster)

struct TcParams {
  const __nv_bfloat16* S;
  const __nv_bfloat16* X;
  __nv_bfloat16* Y;
  int* status;
  int M, N, K, KG;
  int nkb;      // steps of 128
  int ks;       // CTAs of a cluster, each with its share of the steps
  int sw;       // ring slots of packed words (K = 256 each)
  int off_x;    // planes, then factors, behind the ring
  int off_info;
};

__device__ __forceinline__ void umma_i8_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// kind::i8, s32 result: bits [4,6) 2 = s32, [7,10) and [10,13) A and B: 0 = u8, 1 = s8; N and M as for kind::f16.
__host__ __device__ constexpr uint32_t umma_idesc_s8(int b_signed, int M, int N) {
  return (2u << 4) | (1u << 7) | (static_cast<uint32_t>(b_signed) << 10) | (static_cast<uint32_t>(N >> 3) << 17) |
         (static_cast<uint32_t>(M >> 4) << 24);
}

// MB: blocks of 128 weight rows per tile.  DW: conversion warps, two groups of 4 MB that take the steps in turn.
// SV: scales per load.
template <int MB, int DW, int MINB, int SV>
__global__ void __launch_bounds__(128 + DW * 32, MINB)
    w4_gemv_tc_kernel(const __grid_constant__ CUtensorMap tmap_w, const TcParams p) {
  constexpr int kRows = MB * 128, kWSlot = kRows * 128, kThreads = DW * 32;
  constexpr int kTmemCols = 256;  // 128 or 256 used; see the launch
  static_assert(DW == 8 * MB, "two groups of warps");
  extern __shared__ unsigned char smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bar_w_full = base, bar_w_empty = base + 8 * kMaxSlots, bar_a_full = base + 16 * kMaxSlots;
  const uint32_t bar_a_empty = bar_a_full + 8 * kBufs, bar_acc = bar_a_empty + 8 * kBufs, bar_x = bar_acc + 8;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + 512);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen + 516);
  const uint32_t ring_w = base + kHeaderBytes, xs = base + p.off_x, info = base + p.off_info;

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int crank = p.ks > 1 ? (int)cluster_rank() : 0;
  const int n0 = (blockIdx.x / p.ks) * kRows;
  const int kb0 = (int)((long)crank * p.nkb / p.ks), nkb = (int)((long)(crank + 1) * p.nkb / p.ks) - kb0;

  if (tid == 0) {
    *abort_flag = 0;
    for (int s = 0; s < kMaxSlots; ++s) {
      mbar_init(bar_w_full + 8 * s, 1);
      mbar_init(bar_w_empty + 8 * s, DW);
    }
    for (int b = 0; b < kBufs; ++b) {
      mbar_init(bar_a_full + 8 * b, 4 * MB);
      mbar_init(bar_a_empty + 8 * b, 1);
    }
    mbar_init(bar_acc, 1);
    mbar_init(bar_x, 1);
    fence_mbar_init();
    tma_prefetch_desc(&tmap_w);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  pdl_launch_dependents();
  const uint32_t tmem_d = __shfl_sync(0xffffffffu, *tmem_slot, 0);  // [buffer][block][low 16 | high 16] columns
  const uint32_t tmem_a = tmem_d + kBufs * MB * 32;                   // [buffer][block][32] columns
  const bool poisoned = *reinterpret_cast<volatile int*>(p.status) != 0;

  if (!poisoned) {
    if (warp == 0) {
      if (lane == 0) {
        // The kernel in front may be the one that writes the weights: until it has finished they are only brought into
        // L2 (two slots; sixteen launches of a decoder stack at 13 tokens, us: 226, one slot 227, the whole ring 229,
        // nothing 231, the ring filled before the wait 224).
        for (int i = 0; i < nkb && i < 4; i += 2) tma_prefetch_2d(&tmap_w, (kb0 + i) * (kStepK / 8), n0);
        pdl_wait_prior_grid();
        int s = 0;
        uint32_t ph = 1;
        for (int i = 0; i < nkb; i += 2) {
          mbar_wait(bar_w_empty + 8 * s, ph, abort_flag);
          mbar_arrive_expect_tx(bar_w_full + 8 * s, kWSlot);
          tma_load_2d(ring_w + s * kWSlot, &tmap_w, (kb0 + i) * (kStepK / 8), n0, bar_w_full + 8 * s);
          if (++s == p.sw) { s = 0; ph ^= 1; }
        }
      }
      __syncwarp();
    } else if (warp == 1) {
      constexpr uint32_t id_lo = umma_idesc_s8(0, 128, kTokens), id_hi = umma_idesc_s8(1, 128, kTokens);
      const uint64_t desc0 = umma_desc_k128(xs);
      pdl_wait_prior_grid();  // the kernel in front may run longer than a bounded wait for X
      mbar_wait(bar_x, 0, abort_flag);
      for (int i = 0; i < nkb; ++i) {
        const int buf = i % kBufs;
        mbar_wait(bar_a_full + 8 * buf, (i / kBufs) & 1, abort_flag);
        __syncwarp();
        tc_fence_after_sync();
        const uint64_t db = desc0 + i * (kXStep >> 4);
        const uint32_t a = tmem_a + buf * MB * 32, d = tmem_d + buf * MB * 32;
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
#pragma unroll
            for (int mb = 0; mb < MB; ++mb) {
              umma_i8_ts(d + mb * 32, a + mb * 32 + kk * 8, db + kk * 2, id_lo, kk > 0 ? 1u : 0u);
              umma_i8_ts(d + mb * 32 + 16, a + mb * 32 + kk * 8, db + (kTokens * 128 >> 4) + kk * 2, id_hi,
                         kk > 0 ? 1u : 0u);
            }
          }
          umma_commit(bar_a_empty + 8 * buf);
          if (i + 1 == nkb) umma_commit(bar_acc);
        }
        __syncwarp();
      }
    } else if (warp >= 4) {
      const int dw = warp - 4, quad = warp & 3;  // the quarter of the TMEM lanes this warp may touch
      const int mb = (dw >> 2) % MB, grp = dw / (4 * MB);
      const int row = mb * 128 + quad * 32 + lane, n = n0 + row, ct = tid - 128;
      const bool live = n < p.N;
      const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
      const __nv_bfloat16* s_row = p.S + (size_t)(live ? n : 0) * p.KG;
      auto load_sv = [&](int v) {
        uint2 r = make_uint2(0u, 0u);
        if (live && v * SV < p.KG) {
          if (SV == 4) r = __ldcg(reinterpret_cast<const uint2*>(s_row + v * SV));
          else r.x = __ldcg(reinterpret_cast<const uint32_t*>(s_row + v * SV));
        }
        return r;
      };
      int g = kb0 + grp;
      if (live && g < p.KG) prefetch_l2(s_row + g);
      pdl_wait_prior_grid();
      uint2 cur = load_sv(g / SV), nxt = load_sv(g / SV + 1);
      const uint32_t pick = g & 1 ? 0x7632 : 0x5410;  // the odd or the even scale of a pair, as the high half of a float

      // ---- X: 16 consecutive k of a token per item, the eight items of a chunk in eight consecutive lanes; the largest
      // magnitude of a (token, chunk) is scaled to below 2^15, its values are rounded to 16-bit integers (the low mantissa
      // bits of x * 2^.. + 1.5 * 2^23) and split into bytes, in the order the nibble masks produce.
      {
        constexpr int UN = 4;
        const int per_tok = nkb * 8, items = kTokens * per_tok;
        for (int it0 = ct; it0 < items; it0 += kThreads * UN) {  // (items and threads: multiples of 32)
          uint4 va[UN], vb[UN];
#pragma unroll
          for (int u = 0; u < UN; ++u) {
            const int it = it0 + u * kThreads, m = it / per_tok, r = it - m * per_tok;
            va[u] = vb[u] = make_uint4(0u, 0u, 0u, 0u);
            if (it < items && m < p.M) {
              const uint4* src = reinterpret_cast<const uint4*>(p.X + (size_t)m * p.K + (size_t)kb0 * kStepK + r * 16);
              va[u] = __ldcg(src);
              vb[u] = __ldcg(src + 1);
            }
          }
#pragma unroll
          for (int u = 0; u < UN; ++u) {
            const int it = it0 + u * kThreads, m = it / per_tok, r = it - m * per_tok;
            if (it < items) {  // (warp-uniform)
              const uint32_t w[8] = {va[u].x, va[u].y, va[u].z, va[u].w, vb[u].x, vb[u].y, vb[u].z, vb[u].w};
              uint32_t mx2 = 0;
#pragma unroll
              for (int i = 0; i < 8; ++i) mx2 = __vmaxu2(mx2, w[i] & 0x7FFF7FFFu);
              uint32_t mx = max(mx2 & 0xFFFFu, mx2 >> 16);
              mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
              mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
              mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
              uint32_t eb = mx >> 7;
              const bool bad = eb == 255u;
              eb = min(254u, max(40u, eb));
              const float down = __uint_as_float((uint32_t)(16 + 252 - (int)eb) << 23);
              uint32_t v[16];
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                v[2 * i] = __float_as_uint(fmaf(__uint_as_float(w[i] << 16), down, 12582912.f));
                v[2 * i + 1] = __float_as_uint(fmaf(__uint_as_float(w[i] & 0xFFFF0000u), down, 12582912.f));
              }
              const uint32_t at = xs + (r >> 3) * kXStep + m * 128 + (((uint32_t)r ^ (uint32_t)m) & 7u) * 16;
#pragma unroll
              for (int pl = 0; pl < 2; ++pl) {
                uint32_t o[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const int b = (j & 1) * 8 + (j >> 1);  // first k of the word: 0, 8, 1, 9; then every second one
                  const uint32_t t0 = __byte_perm(v[b], v[b + 2], 0x5140), t1 = __byte_perm(v[b + 4], v[b + 6], 0x5140);
                  o[j] = __byte_perm(t0, t1, pl ? 0x7632 : 0x5410);
                }
                sts128(at + pl * kTokens * 128, make_uint4(o[0], o[1], o[2], o[3]));
              }
              if ((r & 7) == 0)
                asm volatile("st.shared.b32 [%0], %1;" ::"r"(info + (r >> 3) * kInfoStep + m * 4),
                             "r"(bad ? 0x7FC00000u : (uint32_t)((int)eb - 18) << 23)
                             : "memory");
            }
          }
        }
      }
      fence_proxy_async_smem();
      asm volatile("bar.sync 1, %0;" ::"r"(kThreads) : "memory");
      if (ct == 0) mbar_arrive(bar_x);

      // ---- steps
      const uint32_t src_row = ring_w + row * 128, swz = (uint32_t)row & 7u;
      uint32_t src_off[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) src_off[j] = src_row + (((uint32_t)(grp * 4 + j) ^ swz) << 4);
      const uint32_t a_dst = tmem_a + lane_off + mb * 32, d_src = tmem_d + lane_off + mb * 32;
      float acc[kTokens];
#pragma unroll
      for (int e = 0; e < kTokens; ++e) acc[e] = 0.f;
      // the sums of step i: lo + 256 hi exactly, then scale times the token's factor
      uint32_t d[32];
      auto add_step = [&](int i, float scale) {
#pragma unroll
        for (int q = 0; q < kTokens / 4; ++q) {
          const uint4 f = lds128(info + i * kInfoStep + q * 16);
          const float ff[4] = {__uint_as_float(f.x), __uint_as_float(f.y), __uint_as_float(f.z), __uint_as_float(f.w)};
#pragma unroll
          for (int e = 0; e < 4; ++e)
            acc[4 * q + e] = fmaf(scale * ff[e], (float)((int)d[4 * q + e] + ((int)d[16 + 4 * q + e] << 8)), acc[4 * q + e]);
        }
      };
      float s_prev = 0.f;
      int s = 0;
      uint32_t ph = 0;
      for (int i = grp; i < nkb; i += 2) {
        const float scale = __uint_as_float(__byte_perm(0, SV == 4 && (g & 2) ? cur.y : cur.x, pick) & 0xFFFF0000u);
        if (SV == 2 || (g & 2)) {
          cur = nxt;
          nxt = load_sv(g / SV + 2);
        }
        g += 2;
        mbar_wait(bar_w_full + 8 * s, ph, abort_flag);
        uint32_t v[32];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 w4 = lds128(src_off[j] + s * kWSlot);
          const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
          for (int h = 0; h < 2; ++h) {  // two words: their even nibbles, their odd nibbles
            v[8 * j + 4 * h] = ((w[2 * h] << 4) & 0xF0F0F0F0u) ^ 0x80808080u;
            v[8 * j + 4 * h + 1] = ((w[2 * h + 1] << 4) & 0xF0F0F0F0u) ^ 0x80808080u;
            v[8 * j + 4 * h + 2] = (w[2 * h] & 0xF0F0F0F0u) ^ 0x80808080u;
            v[8 * j + 4 * h + 3] = (w[2 * h + 1] & 0xF0F0F0F0u) ^ 0x80808080u;
          }
        }
        const int buf = i % kBufs;
        mbar_wait(bar_a_empty + 8 * buf, ((i / kBufs) & 1) ^ 1, abort_flag);
        __syncwarp();
        tc_fence_after_sync();
        tmem_st_32x32(a_dst + buf * (MB * 32), v);
        tmem_st_wait();
        if (i >= kBufs) {
          tmem_ld_32x32(d_src + buf * (MB * 32), d);
          tmem_ld_wait();
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(bar_a_full + 8 * buf);
          mbar_arrive(bar_w_empty + 8 * s);
        }
        if (i >= kBufs) add_step(i - kBufs, s_prev);
        s_prev = scale;
        if (++s == p.sw) { s = 0; ph ^= 1; }
      }
      mbar_wait(bar_acc, 0, abort_flag);
      __syncwarp();
      tc_fence_after_sync();
      const int last = nkb - 1 - ((nkb - 1 - grp) & 1);  // the group's last step (below zero: none)
      if (last >= 0) {
        tmem_ld_32x32(d_src + (last % kBufs) * (MB * 32), d);
        tmem_ld_wait();
        add_step(last, s_prev);
      }
      // [group][token][row], over the ring: every copy has landed
#pragma unroll
      for (int e = 0; e < kTokens; ++e)
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(ring_w + (uint32_t)((grp * kTokens + e) * kRows + row) * 4), "f"(acc[e])
                     : "memory");
    }
  }
  tc_fence_before_sync();
  __syncwarp();
  if (p.ks > 1)
    cluster_barrier();
  else
    __syncthreads();
  // every CTA adds up its share of the tile, four rows of a token per thread, in rank and group order
  if (warp >= 4 && !poisoned) {
    const int units = p.M * (kRows / 4), u1 = (int)((long)(crank + 1) * units / p.ks);
    for (int u = (int)((long)crank * units / p.ks) + tid - 128; u < u1; u += kThreads) {
      const int tok = u / (kRows / 4), r = (u % (kRows / 4)) * 4, n = n0 + r;
      const uint32_t at = ring_w + (uint32_t)(tok * kRows + r) * 4;
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int z = 0; z < 8; ++z)
        if (z < p.ks) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float4 b = ld_cluster_f4(at + h * kTokens * kRows * 4, z);
            a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
          }
        }
      __nv_bfloat16* y = p.Y + (size_t)tok * p.N + n;
      if (n + 4 <= p.N && (p.N & 3) == 0) {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(a.x, a.y), hi = __floats2bfloat162_rn(a.z, a.w);
        *reinterpret_cast<uint2*>(y) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo),
                                                  *reinterpret_cast<const uint32_t*>(&hi));
      } else {
        const float f[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (n + e < p.N) y[e] = __float2bfloat16(f[e]);
      }
    }
  }
  __syncwarp();
  if (p.ks > 1) cluster_barrier();  // the peers have read this CTA's part
  __syncthreads();
  if (*abort_flag) {
    if (tid == 0) atomicCAS(p.status, kStatusOk, kStatusGemvTimeout);
    for (int i = 0; i < 64; ++i) __nanosleep(2000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_d, kTmemCols);
  }
}

using TcKernel = void (*)(const CUtensorMap, const TcParams);

struct TcPlan {
  int form = 0, ks = 1, sw = 0, steps = 0;  // form 0: 128 rows, two CTAs per SM; 1: 256 rows, one
  double us = 0;
};

// Estimated time (us, fitted to 512 to 57344 x 2048 to 28672): waves of CTAs, 4.6 each for start, X and the exchange, 0.62
// per step of a 256-row CTA; a 128-row one takes 0.5 alone on its SM and twice that with a neighbour, and up to 2 more to
// start and sum up where K is cut into single steps and the chip is full (5097 x 768 in clusters of six: 6.3).  A CTA's steps
// are limited by the planes of X beside two ring slots.  wanted_*: 0 = any.
bool tc_plan(int N, int K, int sm_count, int wanted_form, int wanted_ks, TcPlan* out) {
  const int nkb = K / kStepK;
  bool any = false;
  for (int form = 0; form < 2; ++form) {
    if (wanted_form && form != wanted_form - 1) continue;
    const int rows = form ? 256 : 128, room = (form ? kSmemFull : kSmemHalf) - 1024 - kHeaderBytes;
    const long tiles = (N + rows - 1) / rows;
    for (int ks = 1; ks <= 8 && ks <= nkb; ++ks) {
      if (wanted_ks && ks != std::min({wanted_ks, 8, nkb})) continue;
      const int steps = (nkb + ks - 1) / ks;
      TcPlan pl;
      pl.form = form;
      pl.ks = ks;
      pl.steps = steps;
      pl.sw = std::min(kMaxSlots, (room - steps * (kXStep + kInfoStep)) / (rows * 128));
      if (pl.sw < 2) continue;
      // clusters leave some SMs of a GPC out
      const long cap = (form ? 1 : 2) * (ks == 1 ? sm_count : ks == 7 ? sm_count * 0.7 : ks == 8 ? sm_count * 0.8 : sm_count * 0.87);
      const long ctas = tiles * ks, waves = (ctas + cap - 1) / cap;
      const double busy = std::min(1.0, (double)ctas / waves / (2.0 * sm_count));
      pl.us = waves * (form ? 4.6 + 0.62 * steps : 3.8 + (0.5 + 0.5 * busy) * steps + (steps == 1 ? 2.0 * busy : 0.0));
      if (!any || pl.us < out->us) *out = pl;
      any = true;
    }
  }
  return any;
}

}  // namespace

// Nine to sixteen tokens and groups of 128, where the estimate is below what the mma.sync kernel takes: 6 + 0.145 w + 3 K /
// 1e4 us (w = millions of weights; 57344 x 8192 stays, 88 us against 96, and 8192 x 28672, 50 against 57).  Fewer tokens: the
// mma.sync kernel pads to eight and is as fast or faster (37888 x 3584 at eight 20.0 against 21.0).  The estimate is 4 %
// short over 200 shapes, 10 % where a 128-row CTA has nine steps and more (1500 x 11008: 13.9 us against 11.0, estimated at
// 11.1 and 11.7).  Two chunks of K on few rows are all start-up, of which this kernel has more (700 x 256: 3.9 to 4.1 us against
// 3.3; 6000 x 256 level).  Over 110 shapes the pick takes 1.006 times the shorter one's time in the geometric mean.
// (Pointers: null = "assume aligned", for the queries that have no operands.)
bool gemv_tc_applies(const void* X, const void* Wq, const void* S, const void* Y, int M, int N, int K, int G, int flags,
                     int sm_count) {
  if (G != kStepK || K < 2 * kStepK || K % (2 * kStepK) || N < 1 || M < 1 || M > kTokens) return false;
  if (((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(Wq)) & 15) || (reinterpret_cast<uintptr_t>(Y) & 7) ||
      (reinterpret_cast<uintptr_t>(S) & 3))
    return false;
  TcPlan pl;
  if (flags < 0) return tc_plan(N, K, sm_count, (flags >> 24) & 3, (flags >> 20) & 15, &pl);
  if ((flags & ~kFlagNoPdl) != 0 || M <= 8 || (K <= 256 && N < 5000) || !tc_plan(N, K, sm_count, 0, 0, &pl)) return false;
  const double longer = pl.form == 0 && pl.steps >= 9 ? 1.1 : 1.04;
  return longer * pl.us < 6.0 + 0.145e-6 * ((double)N * K) + 3e-4 * K;
}

int gemv_tc_describe(int N, int K, int flags, int sm_count, char* buf, int buflen) {
  const bool forced = flags < 0;
  TcPlan pl;
  if (!tc_plan(N, K, sm_count, forced ? (flags >> 24) & 3 : 0, forced ? (flags >> 20) & 15 : 0, &pl)) return 0;
  const int rows = pl.form ? 256 : 128;
  return snprintf(buf, buflen,
                  "tcgen05 GEMV: %d CTAs (%d per SM), tiles of %d rows x %d tokens, clusters of %d along K, 2 planes (16-bit X), "
                  "%d ring slots",
                  (N + rows - 1) / rows * pl.ks, pl.form ? 1 : 2, rows, kTokens, pl.ks, pl.sw);
}

// flags: bits 20-23 CTAs per cluster, bits 24-25 tile (1: 128 rows, two CTAs per SM; 2: 256 rows, one), 0 = the rule.
int gemv_tc_launch(const void* X, const void* Wq, const void* S, void* Y, int M, int N, int K, const Workspace& ws,
                   int flags, int sm_count, cudaStream_t stream) {
  TcParams p{};
  p.S = static_cast<const __nv_bfloat16*>(S);
  p.X = static_cast<const __nv_bfloat16*>(X);
  p.Y = static_cast<__nv_bfloat16*>(Y);
  p.status = ws.status;
  p.M = M; p.N = N; p.K = K;
  p.KG = K / kStepK;
  p.nkb = K / kStepK;
  const bool forced = flags < 0;
  TcPlan pl;
  if (!tc_plan(N, K, sm_count, forced ? (flags >> 24) & 3 : 0, forced ? (flags >> 20) & 15 : 0, &pl)) return kErrTooLarge;
  const int form = pl.form, rows = form ? 256 : 128, slot = rows * 128, steps = (p.nkb + pl.ks - 1) / pl.ks;
  p.ks = pl.ks;
  p.sw = pl.sw;
  p.off_x = kHeaderBytes + p.sw * slot;
  p.off_info = p.off_x + steps * kXStep;
  CUtensorMap tw;
  if (!make_tensor_map_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, Wq, (uint64_t)N, (uint64_t)K / 8, rows, 32,
                          CU_TENSOR_MAP_SWIZZLE_128B))
    return kErrDevice;
  static constexpr TcKernel kKernels[2][2] = {{w4_gemv_tc_kernel<1, 8, 2, 2>, w4_gemv_tc_kernel<1, 8, 2, 4>},
                                              {w4_gemv_tc_kernel<2, 16, 1, 2>, w4_gemv_tc_kernel<2, 16, 1, 4>}};
  const int sv4 = p.KG % 4 == 0 && reinterpret_cast<uintptr_t>(S) % 8 == 0;
  const TcKernel kernel = kKernels[form][sv4];
  const int smem = form ? kSmemFull : kSmemHalf;  // all of it: at most 512 columns' worth of CTAs fit on an SM
  static std::atomic<bool> done[64][2][2];
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev >= 64 || !done[dev][form][sv4].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    if (dev < 64) done[dev][form][sv4].store(true, std::memory_order_release);
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((N + rows - 1) / rows * p.ks);
  cfg.blockDim = dim3(form ? 640 : 384);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (p.ks > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = p.ks;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
  }
  if ((flags & kFlagNoPdl) == 0) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  e = cudaLaunchKernelEx(&cfg, kernel, tw, p);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

}  // namespace b2
