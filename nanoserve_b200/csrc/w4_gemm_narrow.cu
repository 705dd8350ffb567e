// W4A16 GEMM for sm_100a where the tokens are few:  Y[M,N] (bf16) = X[M,K] (bf16) . dequant(Wq, S)^T: the token counts of
// batched decoding and short prompts (M > 16), and at most 16 tokens where the quantization group is finer than the
// GEMVs' exact integer arithmetic serves.  Same operands and numerics as w4_gemm.cu: each weight is RN_bf16((q - 8) * s),
// products accumulate in fp32, one rounding at the store.
//
// What bounds it: the packed weights' way from HBM (0.5 bytes per weight), and next to it the conversion of every
// weight (eleven instructions per eight, six of them on the ALU pipe at two cycles).  w4_gemm.cu gives the tokens the 128-row
// side of the MMA and writes the converted weights to shared memory: with 48 tokens it pads the MMA to 128, sends every weight through shared memory twice and
// has one CTA per 256 weight rows with no way to fill the chip but fp32 part-tiles in global memory.  Here
//   * the WEIGHTS are the M side of tcgen05.mma (128 rows per block) and the tokens its N side (16 to 128 columns, a
//     multiple of 16): the MMA's work follows the token count;
//   * converted weights go from registers to TENSOR MEMORY (tcgen05.st; a thread owns a weight row = a TMEM lane) and
//     the MMA takes its A operand from there.  Shared memory carries the packed words once and the X tile;
//   * K is cut over the CTAs of a CLUSTER (up to eight), which add their fp32 accumulators up through distributed shared
//     memory in rank order: no scratch in global memory, no counters, the result does not depend on timing;
//   * launched programmatically: the first slots of packed words are brought into L2 ahead of everything else, the first scales
//     before the wait for the kernel in front.  All reads and writes come after it has finished, so it may be the kernel that
//     writes the weights.
// Measured, weights from HBM, one launch behind the other on one card, us at 48 tokens, in brackets this kernel with 17 instructions
// per eight weights and fetched parts, and w4_gemm.cu: 4608 x 3584 8.8 (9.5, 24), 37888 x 3584 21.7 (24.9, 45), 3584 x 18944 16.3 (18.4, 49),
// 8192 x 28672 40.0 (44.8, 103), 3584 x 3584 6.9 (8.8, 23.5); 128 x 37888 x 3584 35.0 (39.2, 51), 777 x 5000 x 4096 in groups of 64 30.9
// (33.6), 512 x 3584 x 18944 71.9 (77.4).  What moved them: weights converted in eleven instructions, the questions to the
// barriers ahead of the last products of a step, parts of a cut K sent instead of fetched, tensor memory freed beside the last
// sums.  What bounds it: at 48 tokens the sixteen products of a step take 590 cycles (37 each, whatever the tokens up to 64: the
// weights' way out of tensor memory) and the conversion 980 per step of either group; a step takes 0.60 us (37888 x 14336 less
// 37888 x 3584), 1170 cycles at 1965 MHz, so neither hides the other whole; 11 of the 21.7 us are HBM's.  At 112 columns the products take
// 57 cycles each, 912 a step, and a step 0.82 us, 1610 cycles: nearly one behind the other.  A third group of
// conversion warps (24 in all, three buffers) changed nothing.
// Warps: 0 packed words (TMA), 1 MMA issue and TMEM, 2 X tiles (TMA), 3 idle, then DW conversion warps, which also do
// the epilogue.  All rings run on mbarriers with bounded waits; a CTA that gives up records a status, still takes part in
// the cluster barriers, frees its TMEM and returns.
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

constexpr int kKB = 128;              // K per step and per X slot: two 128-byte rows of X per token
constexpr int kMaxSlots = 10;
constexpr int kHeaderBytes = 1024;    // barriers and flags
constexpr int kSmemHalf = 115712;     // two CTAs per SM: (228 KB / 2) - 1 KB
constexpr int kSmemFull = 232448;
constexpr uint32_t kUnitBytes = 16 * 32 * 4;  // fp32 sums of 16 tokens x 32 rows
constexpr int kAhead = 3;  // slots of packed words brought into L2 ahead of the wait for the kernel in front

struct NarrowParams {
  const __nv_bfloat16* S;
  __nv_bfloat16* Y;
  int* status;
  int M, N, K, G, KG;
  int nkb;        // K blocks of 128
  int ks;         // CTAs of a cluster, each with its share of the K blocks
  int nt;         // token columns of a tile (multiple of 16)
  int t_tiles;    // token tiles (fastest in the tile order: neighbours read the same weights)
  int sw, sx;     // ring slots of packed words, of X
  int sv;         // scales per load: 4, 2 or 1, by the alignment of a row of S
  int tmem_cols;  // power of two
  int red;        // offset of the parts of a cut K, sent there as they are ready; 0: none, they lie over the rings and are fetched
};

// D[tmem] (+)= A[tmem] * B[smem desc]: A is 128 lanes x 8 columns of bf16 pairs per K = 16.
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// MB: blocks of 128 weight rows per tile (each X tile is then read by MB MMAs).  DW: conversion warps, in DW / (4 MB)
// groups that take the K blocks in turn; the converted weights of two K blocks fit in TMEM.  MINB: CTAs per SM.
// MODE: 4 or 2: groups of 128 (a scale per row and step), read that many at a time; 64, 32: groups of 64 or 32 and whole
// steps, a step's two or four scales per read; 0: any group, any K.  RED: the parts of a cut K are sent (p.red); a kernel of its
// own, since its code made short launches of the others up to 6 % longer.  AHEAD: scales are brought into L2 a sector ahead, by the rows'
// warps (1) or the one that issues the products (2), see narrow_form_ahead.
template <int MB, int DW, int MINB, int MODE, bool RED, int AHEAD = 0>
__global__ void __launch_bounds__(128 + DW * 32, MINB)
    w4_gemm_narrow_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                          const NarrowParams p) {
  constexpr int kRows = MB * 128, kGroups = DW / (4 * MB), kWSlot = kRows * 128;  // a slot of packed words: K = 256
  static_assert(kGroups == 2, "a slot of packed words holds a step for either group");
  [[maybe_unused]] constexpr int kSectorSteps = 16 * MODE / 128;  // steps whose scales fill a sector of 32 bytes (MODE 64, 32)
  constexpr bool G128 = MODE == 2 || MODE == 4;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;  // swizzled tiles
  unsigned char* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bar_w_full = base, bar_w_empty = base + 8 * kMaxSlots;
  const uint32_t bar_x_full = base + 16 * kMaxSlots, bar_x_empty = base + 24 * kMaxSlots;
  const uint32_t bar_a_full = base + 32 * kMaxSlots, bar_a_empty = bar_a_full + 16;
  const uint32_t bar_acc = bar_a_empty + 16, bar_red = bar_acc + 8;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + 512);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen + 516);
  volatile int* status_seen = reinterpret_cast<volatile int*>(gen + 520);
  const uint32_t ring_w = base + kHeaderBytes, ring_x = ring_w + p.sw * kWSlot;
  const uint32_t x_slot = (uint32_t)p.nt * 256;

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int crank = p.ks > 1 ? (int)cluster_rank() : 0;
  const int tile = blockIdx.x / p.ks;
  const int m0 = (tile % p.t_tiles) * p.nt, n0 = (tile / p.t_tiles) * kRows;
  const int kb0 = (int)((long)crank * p.nkb / p.ks), nkb = (int)((long)(crank + 1) * p.nkb / p.ks) - kb0;

  // Units of 16 tokens x 32 rows, in the order (tokens, rows): the parts of a cut K are added by unit, and this CTA adds those from
  // first_unit(crank) to first_unit(crank + 1).
  const int rt = min(p.nt, p.M - m0), units = (rt + 15) / 16 * (kRows / 32);
  auto first_unit = [&](int rank) { return (rank * units + p.ks - 1) / p.ks; };

  // (only brought into L2: the kernel in front may be the one that writes them)
  if (tid == 64)
    for (int i = 0; i < nkb && i < 2 * kAhead; i += 2) tma_prefetch_2d(&tmap_w, (kb0 + i) * (kKB / 8), n0);
  if (tid == 0) {
    *abort_flag = 0;
    for (int s = 0; s < kMaxSlots; ++s) {
      mbar_init(bar_w_full + 8 * s, 1);
      mbar_init(bar_w_empty + 8 * s, DW);
      mbar_init(bar_x_full + 8 * s, 1);
      mbar_init(bar_x_empty + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_a_full + 8 * b, 4 * MB);
      mbar_init(bar_a_empty + 8 * b, 1);
    }
    mbar_init(bar_acc, 1);
    mbar_init(bar_red, 1);
    if constexpr (RED) mbar_arrive_expect_tx(bar_red, (uint32_t)((first_unit(crank + 1) - first_unit(crank)) * p.ks) * kUnitBytes);
    fence_mbar_init();
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
  }
  if (tid == 64) *status_seen = *reinterpret_cast<volatile int*>(p.status);  // (one answer for all warps of the CTA)
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), p.tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  pdl_launch_dependents();
  if constexpr (RED) cluster_arrive();  // (waited for before the first store into a peer: its barrier is set up)
  const uint32_t tmem_d = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const uint32_t tmem_a = tmem_d + ((MB * p.nt + 31) & ~31);
  const bool poisoned = *status_seen != 0;
  // Behind this the conversion warps leave tensor memory alone: the warp that allocated it frees it while they add up and store.
  // (Where the parts are fetched it does so behind the cluster barrier: ahead of it all would wait.)
  const bool fetched = !RED && p.ks > 1;
  auto rows_done = [&] {
    if (!fetched) asm volatile("bar.arrive 1, %0;" ::"n"(DW * 32 + 32) : "memory");
  };

  if (!poisoned) {
    if (warp == 0) {
      if (lane == 0) {
        pdl_wait_prior_grid();  // it may be the kernel that writes the weights
        int s = 0;
        uint32_t ph = 1;
        for (int i = 0; i < nkb; i += 2) {  // (128-byte rows: the copy engine's rate counts rows, not bytes)
          mbar_wait(bar_w_empty + 8 * s, ph, abort_flag);
          mbar_arrive_expect_tx(bar_w_full + 8 * s, kWSlot);
          tma_load_2d(ring_w + s * kWSlot, &tmap_w, (kb0 + i) * (kKB / 8), n0, bar_w_full + 8 * s);
          if (++s == p.sw) { s = 0; ph ^= 1; }
        }
      }
      __syncwarp();
    } else if (warp == 2) {
      if (lane == 0) {
        pdl_wait_prior_grid();
        int s = 0;
        uint32_t ph = 1;
        for (int i = 0; i < nkb; ++i) {
          mbar_wait(bar_x_empty + 8 * s, ph, abort_flag);
          mbar_arrive_expect_tx(bar_x_full + 8 * s, x_slot);
          const uint32_t dst = ring_x + s * x_slot;
          tma_load_2d(dst, &tmap_x, (kb0 + i) * kKB, m0, bar_x_full + 8 * s);
          tma_load_2d(dst + x_slot / 2, &tmap_x, (kb0 + i) * kKB + 64, m0, bar_x_full + 8 * s);
          if (++s == p.sx) { s = 0; ph ^= 1; }
        }
      }
      __syncwarp();
    } else if (warp == 1) {
      // The whole warp runs the loop and one elected lane issues: with everything the instructions take the same in all
      // lanes the descriptors stay in uniform registers.  (Under `if (lane == 0)` an issue took 176 cycles, whatever the
      // tile, and bounded the kernel.)
      const uint32_t idesc = umma_idesc_bf16(128, p.nt);
      const uint64_t desc0 = umma_desc_k128(ring_x);
      int xs = 0;
      uint32_t xph = 0;
      pdl_wait_prior_grid();  // the kernel in front may run longer than a bounded wait for X
      // An answer of a barrier takes some 130 cycles: the questions of the next step go in ahead of the last products of this one,
      // which the tensor core takes as long to get through (128 tokens, 37888 x 3584: 37.1 -> 36.2 us; 48: 24.7 -> 24.1).
      bool ready = false;
      for (int i = 0; i < nkb; ++i) {
        const int buf = i & 1, xs_this = xs;
        if (!ready) {
          if (!__all_sync(0xffffffffu, mbar_try_wait2(bar_x_full + 8 * xs, xph, bar_a_full + 8 * buf, (i >> 1) & 1))) {
            mbar_wait(bar_x_full + 8 * xs, xph, abort_flag);
            mbar_wait(bar_a_full + 8 * buf, (i >> 1) & 1, abort_flag);
            __syncwarp();
          }
        }
        tc_fence_after_sync();
        const uint64_t db = desc0 + ((xs * x_slot) >> 4);
        const uint32_t a = tmem_a + buf * MB * 64;
        if (++xs == p.sx) { xs = 0; xph ^= 1; }
        bool next = false;
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {
            if (kk == 7)  // (of no meaning behind the last step)
              next = mbar_test_wait2(bar_x_full + 8 * xs, xph, bar_a_full + 8 * (buf ^ 1), ((i + 1) >> 1) & 1);
            const uint64_t d = db + (kk & 3) * 2 + (kk >> 2) * (x_slot >> 5);
#pragma unroll
            for (int mb = 0; mb < MB; ++mb)
              umma_f16_ts(tmem_d + mb * p.nt, a + mb * 64 + kk * 8, d, idesc, (i > 0 || kk > 0) ? 1u : 0u);
          }
          umma_commit(bar_a_empty + 8 * buf);
          umma_commit(bar_x_empty + 8 * xs_this);
          if (i + 1 == nkb) umma_commit(bar_acc);
        }
        ready = __any_sync(0xffffffffu, next);
        __syncwarp();
        if constexpr (AHEAD == 2) {
          if (i % kSectorSteps == 0 && i + kSectorSteps < nkb) {
#pragma unroll
            for (int r = 0; r < 4 * MB; ++r) {
              const int n = n0 + r * 32 + lane;
              if (n < p.N) prefetch_l2(p.S + (size_t)n * p.KG + (kb0 + i + kSectorSteps) * (128 / MODE));
            }
          }
        }
      }
    }
  }
  if (warp >= 4) {
    const int dw = warp - 4, quad = warp & 3;       // the quarter of the TMEM lanes this warp may touch
    const int mb = (dw >> 2) % MB, grp = dw / (4 * MB);
    const int row = mb * 128 + quad * 32 + lane;    // weight row of the tile
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    if (!poisoned) {
      const int n = n0 + row;
      const bool live = n < p.N;
      const __nv_bfloat16* s_row = p.S + (size_t)(live ? n : 0) * p.KG;
      // Scales, p.sv of them per load (a thread reads along its own row, so every load touches 32 lines), the next load
      // in flight while one is used.  General groups: (g, kin) is the group of the current K position and the position
      // inside it, vi the load that group is in.
      const int sv = G128 ? MODE : MODE == 64 ? 2 : MODE == 32 ? 4 : p.sv;
      auto load_sv = [&](int v) {
        uint2 r = make_uint2(0u, 0u);
        const int g = v * sv;
        if (live && g < p.KG) {
          if (sv == 4) r = __ldcg(reinterpret_cast<const uint2*>(s_row + g));
          else if (sv == 2) r.x = __ldcg(reinterpret_cast<const uint32_t*>(s_row + g));
          else r.x = __ldcg(reinterpret_cast<const unsigned short*>(s_row + g));
        }
        return r;
      };
      int k = (kb0 + grp) * kKB;
      int g = MODE ? kb0 + grp : k / p.G, kin = MODE ? 0 : k - g * p.G;  // MODE: g counts steps
      int vi = G128 || MODE == 0 ? g / sv : g;
      if (const int first = MODE >= 32 ? g * sv : g; live && first < p.KG) prefetch_l2(s_row + first);
      pdl_wait_prior_grid();
      uint2 cur = load_sv(vi), nxt = load_sv(MODE >= 32 ? vi + 2 : vi + 1);
      auto scale2 = [&]() {  // the pair (s, s) of the current position
        const int e = g - vi * sv;
        return __byte_perm(e & 2 ? cur.y : cur.x, 0, e & 1 ? 0x3232 : 0x1010);
      };
      auto advance = [&](int by) {
        kin += by;
        while (kin >= p.G) {
          kin -= p.G;
          ++g;
        }
        while (g >= (vi + 1) * sv) {
          ++vi;
          cur = nxt;
          nxt = load_sv(vi + 1);
        }
      };
      [[maybe_unused]] const uint32_t pick = (kb0 + grp) & 1 ? 0x3232 : 0x1010;
      const uint32_t src_row = ring_w + row * 128, swz = (uint32_t)row & 7u;
      uint32_t src_off[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) src_off[j] = src_row + (((uint32_t)(grp * 4 + j) ^ swz) << 4);
      const uint32_t a_dst = tmem_a + lane_off + (grp * MB + mb) * 64;
      int s = 0;
      uint32_t ph = 0, aph = 1;
      for (int i = grp; i < nkb; i += 2) {
        uint32_t sc[4];
        if constexpr (G128) {
          sc[0] = sc[1] = sc[2] = sc[3] = __byte_perm(MODE == 4 && (g & 2) ? cur.y : cur.x, 0, pick);
          if (MODE == 2 || (g & 2)) {
            cur = nxt;
            nxt = load_sv(g / MODE + 2);
          }
          g += 2;
        } else if constexpr (MODE == 64 || MODE == 32) {
          sc[0] = __byte_perm(cur.x, 0, 0x1010);
          sc[1] = MODE == 64 ? sc[0] : __byte_perm(cur.x, 0, 0x3232);
          sc[2] = __byte_perm(MODE == 64 ? cur.x : cur.y, 0, MODE == 64 ? 0x3232 : 0x1010);
          sc[3] = MODE == 64 ? sc[2] : __byte_perm(cur.y, 0, 0x3232);
          cur = nxt;
          nxt = load_sv(g + 4);
          g += 2;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            sc[j] = k + 32 * j < p.K ? scale2() : 0u;  // behind the end of K: zero weights
            advance(j < 3 ? 32 : 32 + kKB);
          }
          k += 2 * kKB;
        }
        if constexpr (AHEAD == 1) {
          const int ahead = (kb0 + i + kSectorSteps) * (128 / MODE);
          if (i % kSectorSteps == 0 && i + kSectorSteps < nkb && live && ahead < p.KG) prefetch_l2(s_row + ahead);
        }
        bool plain = dequant_scale_plain(sc[0]);
        if constexpr (!G128) {
#pragma unroll
          for (int j = 1; j < 4; ++j) plain = plain && dequant_scale_plain(sc[j]);
        }
        plain = __all_sync(0xffffffffu, plain);
        mbar_wait(bar_w_full + 8 * s, ph, abort_flag);
        uint4 w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = lds128(src_off[j] + s * kWSlot);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t v[32];
          if (plain) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const uint4 q = w[2 * half + j];
              const DequantScale ds = dequant_scale(sc[2 * half + j]);
              dequant_word(q.x, ds, v + 16 * j);
              dequant_word(q.y, ds, v + 16 * j + 4);
              dequant_word(q.z, ds, v + 16 * j + 8);
              dequant_word(q.w, ds, v + 16 * j + 12);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const uint4 q = w[2 * half + j];
              dequant_word_any(q.x, sc[2 * half + j], v + 16 * j);
              dequant_word_any(q.y, sc[2 * half + j], v + 16 * j + 4);
              dequant_word_any(q.z, sc[2 * half + j], v + 16 * j + 8);
              dequant_word_any(q.w, sc[2 * half + j], v + 16 * j + 12);
            }
          }
          if (half == 0) {
            mbar_wait(bar_a_empty + 8 * grp, aph, abort_flag);
            __syncwarp();
            tc_fence_after_sync();
          }
          tmem_st_32x32(a_dst + half * 32, v);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(bar_a_full + 8 * grp);
          mbar_arrive(bar_w_empty + 8 * s);  // the slot's words went into the conversion above
        }
        aph ^= 1;
        if (++s == p.sw) { s = 0; ph ^= 1; }
      }
      mbar_wait(bar_acc, 0, abort_flag);
      __syncwarp();
      tc_fence_after_sync();

      // ---- the accumulator columns (tokens) of the warp's 32 rows; two groups of warps take alternate 16 columns
      if constexpr (RED) cluster_wait();
      for (int c0 = 16 * grp; c0 < rt; c0 += 16 * kGroups) {
        uint32_t v[16];
        tmem_ld_32x16(tmem_d + lane_off + mb * p.nt + c0, v);
        tmem_ld_wait();
        if constexpr (RED) {
          // a unit's parts go to the CTA that adds them, in the order of ranks: [unit][rank][four tokens][row]
          const int u = c0 / 16 * (kRows / 32) + (row >> 5), owner = u * p.ks / units;
          const uint32_t at = base + p.red + (uint32_t)((u - first_unit(owner)) * p.ks + crank) * kUnitBytes + lane * 16;
#pragma unroll
          for (int q = 0; q < 4; ++q)
            st_async_f4(at + q * 512, bar_red, owner, __uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]),
                        __uint_as_float(v[4 * q + 2]), __uint_as_float(v[4 * q + 3]));
        } else if (p.ks == 1) {
          __nv_bfloat16* y = p.Y + (size_t)(m0 + c0) * p.N + n;
#pragma unroll
          for (int e = 0; e < 16; ++e)
            if (live && c0 + e < rt) y[(size_t)e * p.N] = __float2bfloat16(__uint_as_float(v[e]));
        } else {  // [token][row], over the rings: every copy has landed and every MMA has read its operands
#pragma unroll
          for (int e = 0; e < 16; ++e)
            asm volatile("st.shared.b32 [%0], %1;" ::"r"(ring_w + (uint32_t)((c0 + e) * kRows + row) * 4), "r"(v[e])
                         : "memory");
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      rows_done();
      if constexpr (RED) {
        const int u0 = first_unit(crank), n_units = first_unit(crank + 1) - u0;
        if (dw < n_units) {
          mbar_wait(bar_red, 0, abort_flag);
          __syncwarp();
          for (int b = dw; b < n_units; b += DW) {
            const int u = u0 + b, c0 = u / (kRows / 32) * 16, ny = n0 + u % (kRows / 32) * 32 + lane;
            const uint32_t part = base + p.red + (uint32_t)(b * p.ks) * kUnitBytes + lane * 16;
            __nv_bfloat16* y = p.Y + (size_t)(m0 + c0) * p.N + ny;
#pragma unroll 1
            for (int q = 0; q < 4; ++q) {
              float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
              for (int z = 0; z < 8; ++z)
                if (z < p.ks) {
                  const uint4 f = lds128(part + z * kUnitBytes + q * 512);
                  sum[0] += __uint_as_float(f.x);
                  sum[1] += __uint_as_float(f.y);
                  sum[2] += __uint_as_float(f.z);
                  sum[3] += __uint_as_float(f.w);
                }
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (ny < p.N && c0 + 4 * q + e < rt)
                  y[(size_t)(4 * q + e) * p.N] = __float2bfloat16(sum[e]);
            }
          }
        }
      }
    } else {  // (this barrier has no limit)
      rows_done();
    }
  }
  __syncwarp();
  bool freed = false;
  auto free_early = [&] {
    if (!poisoned && !__any_sync(0xffffffffu, *abort_flag != 0)) {  // (every product has been waited for)
      tc_fence_after_sync();
      tmem_dealloc(tmem_d, p.tmem_cols);
      freed = true;
    }
  };
  if (warp == 1 && !fetched) {
    asm volatile("bar.sync 1, %0;" ::"n"(DW * 32 + 32) : "memory");
    free_early();
  }
  if constexpr (RED) {
    if (warp < 4 || poisoned) cluster_wait();
  } else if (fetched) {
    cluster_barrier();
    if (warp == 1) free_early();
    // every CTA adds up its share of the tile, four rows of a token per thread, in rank order
    if (warp >= 4 && !poisoned) {
      const int quads = rt * (kRows / 4);
      const int u1 = (int)((long)(crank + 1) * quads / p.ks);
      for (int u = (int)((long)crank * quads / p.ks) + tid - 128; u < u1; u += DW * 32) {
        const int tok = u / (kRows / 4), r = (u % (kRows / 4)) * 4, n = n0 + r;
        const uint32_t at = ring_w + (uint32_t)(tok * kRows + r) * 4;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int z = 0; z < 8; ++z)
          if (z < p.ks) {
            const float4 b = ld_cluster_f4(at, z);
            a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
          }
        __nv_bfloat16* y = p.Y + (size_t)(m0 + tok) * p.N + n;
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
    cluster_barrier();  // the peers have read this CTA's part
  }
  __syncthreads();
  if (*abort_flag || (RED && poisoned)) {
    if constexpr (RED) {  // peers that have not given up may send parts here until they leave
      cluster_arrive();
      cluster_wait();
    }
    if (tid == 0) atomicCAS(p.status, kStatusOk, kStatusGemmTimeout);
    for (int i = 0; i < 64; ++i) __nanosleep(2000);  // copies in flight land before the shared memory is released
    __syncthreads();
  }
  if (warp == 1 && !freed) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_d, p.tmem_cols);
  }
}

using NarrowKernel = void (*)(const CUtensorMap, const CUtensorMap, const NarrowParams);
struct NarrowForm {
  NarrowKernel kernel;
  int variant, rows, warps, per_sm, smem;
  bool red;
};
// form 0: 128 weight rows, two CTAs per SM; form 1: 256 rows, one CTA.  All of an SM's (or half an SM's) shared memory
// is asked for, needed or not: at most 512 columns' worth of CTAs then fit on an SM, whatever mix of these launches
// overlaps, and no CTA of a cluster waits for tensor memory that a CTA at a cluster barrier holds.
// variant: 0 any group, 1 and 2 groups of 128 by two and by four scales, 3 groups of 64, 4 groups of 32
template <int MB, int DW, int MINB, bool RED>
NarrowKernel narrow_kernel(int variant) {
  static constexpr NarrowKernel kKernels[5] = {w4_gemm_narrow_kernel<MB, DW, MINB, 0, RED>, w4_gemm_narrow_kernel<MB, DW, MINB, 2, RED>,
                                               w4_gemm_narrow_kernel<MB, DW, MINB, 4, RED>, w4_gemm_narrow_kernel<MB, DW, MINB, 64, RED>,
                                               w4_gemm_narrow_kernel<MB, DW, MINB, 32, RED>};
  return kKernels[variant];
}
NarrowForm narrow_form(int form, int variant, bool red) {
  if (form == 0)
    return {red ? narrow_kernel<1, 8, 2, true>(variant) : narrow_kernel<1, 8, 2, false>(variant), variant, 128, 8, 2, kSmemHalf, red};
  return {red ? narrow_kernel<2, 16, 1, true>(variant) : narrow_kernel<2, 16, 1, false>(variant), variant, 256, 16, 1, kSmemFull, red};
}
// Long shares of K in groups of 64 and 32, K a multiple of 256 and not of 512 (variants 5 and 6): there the next scales of some lane
// come from HBM in most steps, later than the one step ahead that they are asked for, and the faster conversion lost by it (31604 x 9984
// at 24 tokens, groups of 64 and of 32: 52.8 and 57 us with the old one, 57 and 63 with the new).  With the sector ahead brought into
// L2 50 and 56 (6400: 30 and 40 for 31 and 44 at 4 tokens).  Not below 48 steps to a CTA (5376 level, 2816 in groups of 32 4 % longer) nor
// for other K, which have no such loss, and kernels of their own, since the code alone costs short launches 1 to 3 %.  Groups of 32 have
// the warp that issues the products ask (5 % shorter), but for parts that are sent (2 % longer).
NarrowForm narrow_form_ahead(int variant, bool red) {
  static constexpr NarrowKernel k64[2] = {w4_gemm_narrow_kernel<2, 16, 1, 64, false, 1>, w4_gemm_narrow_kernel<2, 16, 1, 64, true, 1>};
  static constexpr NarrowKernel k32[2] = {w4_gemm_narrow_kernel<2, 16, 1, 32, false, 2>, w4_gemm_narrow_kernel<2, 16, 1, 32, true, 1>};
  return {variant == 3 ? k64[red] : k32[red], variant + 2, 256, 16, 1, kSmemFull, red};
}
bool narrow_ahead(int form, int variant, int nt, int K, int blocks) {
  return form == 1 && variant >= 3 && nt <= 64 && K % 512 == 256 && blocks >= 48;
}
int narrow_scales_per_load(const void* S, int K, int G) {
  const uintptr_t sa = reinterpret_cast<uintptr_t>(S);
  const int kg = K / G;
  return kg % 4 == 0 && sa % 8 == 0 ? 4 : kg % 2 == 0 && sa % 4 == 0 ? 2 : 1;
}
int narrow_variant(const void* S, int K, int G) {
  const int sv = narrow_scales_per_load(S, K, G);
  if (G == 128 && sv > 1) return sv / 2;
  if (G == 64 && K % kKB == 0 && sv > 1) return 3;
  if (G == 32 && K % kKB == 0 && sv == 4) return 4;
  return 0;
}

int narrow_attributes(const NarrowForm& f, int form, int dev) {
  static std::atomic<bool> done[64][2][7][2];
  if (dev >= 0 && dev < 64 && done[dev][form][f.variant][f.red].load(std::memory_order_acquire)) return 0;
  const cudaError_t e = cudaFuncSetAttribute(f.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, f.smem);
  if (e == cudaSuccess && dev >= 0 && dev < 64) done[dev][form][f.variant][f.red].store(true, std::memory_order_release);
  return (int)e;
}

void narrow_config(const NarrowForm& f, int grid, int ks, bool pdl, cudaLaunchConfig_t* cfg, cudaLaunchAttribute (&attr)[2]) {
  cfg->gridDim = dim3(grid);
  cfg->blockDim = dim3(128 + f.warps * 32);
  cfg->dynamicSmemBytes = f.smem;
  int na = 0;
  if (ks > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = ks;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
  }
  if (pdl) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg->attrs = attr;
  cfg->numAttrs = na;
}

// Clusters of ks one-per-SM CTAs the device runs at a time (a cluster stays inside one GPC, so some SMs of a GPC are left
// out), asked for once per device.
int narrow_clusters(int ks, int sm_count, int dev) {
  if (ks == 1) return sm_count;
  static std::atomic<int> known[64][9];
  const bool cached = dev >= 0 && dev < 64;
  if (cached)
    if (const int v = known[dev][ks].load(std::memory_order_relaxed)) return v;
  const NarrowForm f = narrow_form(1, 2, false);
  int clusters = 0;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[2];
  narrow_config(f, ks, ks, false, &cfg, attr);
  if (narrow_attributes(f, 1, dev) != 0 || cudaOccupancyMaxActiveClusters(&clusters, f.kernel, &cfg) != cudaSuccess ||
      clusters < 1) {
    (void)cudaGetLastError();
    clusters = std::max(1, sm_count / ks * 7 / 8);
  }
  if (cached) known[dev][ks].store(clusters, std::memory_order_relaxed);
  return clusters;
}
// CTAs of a form the device runs at a time.  (Half-SM CTAs: twice the full ones; 288 CTAs in clusters of four were
// measured to take two waves, so the clusters of one do not fill what those of the other leave.)
int narrow_capacity(int form, int ks, int sm_count, int dev) {
  return std::min(sm_count, narrow_clusters(ks, sm_count, dev) * ks) * (form == 0 ? 2 : 1);
}

struct NarrowPlan {
  int form = 0, ks = 1, nt = 16, t_tiles = 1;
  long n_tiles = 0;
  double us = 0;
};

// Estimated time of a form and a cluster size: start-up, the exchange through distributed shared memory when K is cut,
// and waves of CTAs that take their K blocks at a rate that falls with the token columns and with the share of the chip
// at work.  The constants (us) are a least-squares fit to 900 measured launches, 256 to 57344 x 512 to 28672 at 17 to 2300
// tokens, weights from HBM (residual 13 to 15 %); over those shapes the form it picks takes 1.03 times the best one's
// time in the geometric mean.
void narrow_estimate(NarrowPlan* pl, int N, int K, int sm_count, int dev) {
  const int nkb = (K + kKB - 1) / kKB;
  pl->n_tiles = (long)pl->t_tiles * ((N + (pl->form ? 255 : 127)) / (pl->form ? 256 : 128));
  const int cap = narrow_capacity(pl->form, pl->ks, sm_count, dev);
  const long ctas = pl->n_tiles * pl->ks, waves = (ctas + cap - 1) / cap;
  const int blocks = (nkb + pl->ks - 1) / pl->ks;
  const double nt = pl->nt, busy = std::min(1.0, (double)ctas / waves / (sm_count * (pl->form ? 1 : 2)));
  const double cut = pl->ks - 1;
  if (pl->form)
    pl->us = 1.27 + 0.0303 * nt + (cut > 0 ? 0.07 + 0.0071 * nt : 0.0) + cut * (0.130 + 0.0011 * nt) +
             (waves - 1) * (4.42 + 0.0127 * nt) + waves * blocks * (0.449 + 0.0022 * nt + busy * (0.312 - 0.0008 * nt));
  else
    pl->us = 1.24 + 0.0291 * nt + (cut > 0 ? 0.41 + 0.0022 * nt : 0.0) + cut * (0.101 + 0.0010 * nt) +
             (waves - 1) * (1.03 + 0.0163 * nt) + waves * blocks * (0.301 + 0.0017 * nt + busy * (0.509 - 0.0004 * nt));
}

NarrowPlan narrow_plan(int M, int N, int K, int flags, int sm_count, int dev) {
  NarrowPlan best;
  const bool forced = flags & (kFlagGemmNarrow | kFlagDecodeNarrow);
  const int want_form = forced ? (flags >> 24) & 3 : 0, want_ks = forced ? (flags >> 20) & 15 : 0;
  const int nkb = (K + kKB - 1) / kKB;
  bool any = false;
  for (int form = 0; form < 2; ++form) {
    if (want_form && form != want_form - 1) continue;
    for (int ks = 1; ks <= 8 && ks <= nkb; ++ks) {
      if (want_ks && ks != std::min({want_ks, 8, nkb})) continue;
      NarrowPlan pl;
      pl.form = form;
      pl.ks = ks;
      pl.t_tiles = (M + 127) / 128;
      pl.nt = ((M + pl.t_tiles - 1) / pl.t_tiles + 15) / 16 * 16;
      narrow_estimate(&pl, N, K, sm_count, dev);
      if (!any || pl.us < best.us) best = pl;
      any = true;
    }
  }
  return best;
}

int current_device() {
  int dev = -1;
  return cudaGetDevice(&dev) == cudaSuccess ? dev : -1;
}

}  // namespace

// Up to 16 tokens.  Groups that are no multiple of 128 have their weights rounded to bf16 in the GEMV as here, and it
// takes about 4 + 0.195 w + M K / 1e4 us (w = millions of weights, from HBM; 0.1 w more above eight tokens): G = 64,
// 37888 x 3584 M = 4 35.0 against 22.7 here, 3584 x 18944 M = 16 64.4 against 18.4, 3584 x 3584 M = 1 7.3 against 6.9;
// 57344 x 8192 M = 1 stays, 97.6 against 85 and estimated at 100.  Multiples of 128 keep exact weights: the GEMVs' alone.
// Groups whose scales this kernel would read one by one or by two (K / 64 odd, K / 32 not a multiple of four) stay with the
// GEMV: 313 x 28224 in groups of 64, M = 14, 13.7 us against 31.2 here, 8436 x 8032 in groups of 32, M = 6, 24.4 against 39.9;
// over 140 such shapes 1.1 times the GEMV's time, over 100 of the others 0.66 times.
// (Pointers: null = "assume aligned", for the queries that have no operands.)
bool gemm_narrow_takes_decode(const void* X, const void* Wq, const void* S, const void* Y, int M, int N, int K, int G,
                              int flags, int sm_count) {
  if (flags < 0) return true;
  if ((flags & ~kFlagNoPdl) != 0 || M < 1 || N < 1 || K < 32 || G < 32 || K % 32 || G % 32 || K % G || G % 128 == 0) return false;
  if (((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(Wq) | reinterpret_cast<uintptr_t>(Y)) & 15) ||
      (reinterpret_cast<uintptr_t>(S) & 1))
    return false;
  if (narrow_variant(S, K, G) == 0) return false;
  const double w = (double)N * K * 1e-6, gemv = 4.0 + 0.195 * w + 1e-4 * M * K + (M > 8 ? 0.1 * w : 0.0);
  return 1.05 * narrow_plan(M, N, K, 0, sm_count, current_device()).us < gemv;
}

// Whether this kernel takes a GEMM that the general kernel would run in about wide_us microseconds.  The estimate of its
// plan is brought to what it takes where the two are close; the form for any group takes longer by its loads of scales per
// step (groups of 128 one by one, as K = 13696 has them, 1.31; of 64 1.6; of 32 2.4; of 256 by two 1.12).  Over 1900 shapes,
// 17 to 8192 tokens, both kernels timed in turn, the one this picks takes 1.003 times the shorter one's time in the
// geometric mean and is more than 10 % behind in 1 % (before the two fits: 1.51 at 4096 tokens on 4096 x 13696).
bool gemm_narrow_applies(const void* S, int M, int N, int K, int G, int flags, double wide_us, int sm_count) {
  if (M <= 16) return true;  // (decided by gemm_narrow_takes_decode)
  if (flags & (kFlagGemmNoPairs | kFlagGemmWholeTiles | kFlagGemmWide)) return false;  // the other kernel's switches
  if (flags & kFlagGemmNarrow) return true;
  const double slower = narrow_variant(S, K, G) != 0 ? 1.0 : 1.05 + 0.31 * 128.0 / G / narrow_scales_per_load(S, K, G);
  return 1.4 + 0.957 * slower * narrow_plan(M, N, K, flags, sm_count, current_device()).us < wide_us;
}

int gemm_narrow_describe(int M, int N, int K, int G, int flags, int sm_count, char* buf, int buflen) {
  const NarrowPlan pl = narrow_plan(M, N, K, flags, sm_count, current_device());
  static const char* const kScales[5] = {"one by one", "by two", "by four", "by step", "by step"};
  return snprintf(buf, buflen,
                  "few-token GEMM: %ld CTAs (%d per SM), tiles of %d rows x %d tokens, clusters of %d along K, scales %s",
                  pl.n_tiles * pl.ks, pl.form ? 1 : 2, pl.form ? 256 : 128, pl.nt, pl.ks,
                  kScales[narrow_variant(nullptr, K, G)]);
}

// The arguments have been checked by gemm_launch.
int gemm_narrow_launch(const void* X, const void* Wq, const void* S, void* Y, int M, int N, int K, int G,
                       const Workspace& ws, int flags, int sm_count, cudaStream_t stream) {
  const int dev = current_device();
  const NarrowPlan pl = narrow_plan(M, N, K, flags, sm_count, dev);
  if (pl.n_tiles * pl.ks > 0x3fffffff) return kErrBadShape;
  NarrowParams p{};
  p.S = static_cast<const __nv_bfloat16*>(S);
  p.Y = static_cast<__nv_bfloat16*>(Y);
  p.status = ws.status;
  p.M = M; p.N = N; p.K = K; p.G = G;
  p.KG = K / G;
  p.nkb = (K + kKB - 1) / kKB;
  p.t_tiles = pl.t_tiles;
  p.nt = pl.nt;
  p.ks = pl.ks;
  p.sv = narrow_scales_per_load(S, K, G);
  const int variant = narrow_variant(S, K, G);
  NarrowForm f = narrow_form(pl.form, variant, false);
  const int slot_w = f.rows * 128, slot_x = p.nt * 256, room = f.smem - kHeaderBytes - 1024;
  const int x_bytes = pl.form ? 128 << 10 : p.nt > 64 ? 72 << 10 : 48 << 10;  // the rest holds packed words
  const int blocks = (p.nkb + p.ks - 1) / p.ks;
  p.sx = std::max(2, std::min({6, x_bytes / slot_x, blocks}));
  p.sw = std::min(kMaxSlots, (room - p.sx * slot_x) / slot_w);
  // Up to 64 token columns the parts of a cut K have a place of their own where the rings can spare it without a slot that the CTA has
  // work for (39 x 11469 x 9984 with three slots of four 28.7 us, so 25.0): every CTA then sends them as soon as it has them and
  // leaves (3584 x 3584 at 48 tokens 8.1 -> 7.0 us).  More columns are fetched from the rings' place
  // behind a cluster barrier: sixteen bytes at a time, each counted, are slower from there (512 tokens 17.3 against 20.3).
  const int units = p.nt / 16 * (f.rows / 32), parts = (units + p.ks - 1) / p.ks * p.ks * (int)kUnitBytes;
  const int spare = (room - p.sx * slot_x - parts) / slot_w;
  if (p.ks > 1 && p.nt <= 64 && spare >= std::min(p.sw, (blocks + 1) / 2)) {
    p.sw = std::min(kMaxSlots, spare);
    p.red = kHeaderBytes + p.sw * slot_w + p.sx * slot_x;
    f = narrow_form(pl.form, variant, true);
  }
  if (narrow_ahead(pl.form, variant, p.nt, K, blocks)) f = narrow_form_ahead(variant, f.red);
  p.tmem_cols = pl.form ? 512 : 256;
  CUtensorMap tx, tw;
  if (!make_tensor_map_2d(&tx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, X, (uint64_t)M, (uint64_t)K, p.nt, 64,
                          CU_TENSOR_MAP_SWIZZLE_128B) ||
      !make_tensor_map_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, Wq, (uint64_t)N, (uint64_t)K / 8, f.rows, 2 * kKB / 8,
                          CU_TENSOR_MAP_SWIZZLE_128B))
    return kErrDevice;
  if (const int rc = narrow_attributes(f, pl.form, dev)) return rc;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[2];
  narrow_config(f, (int)(pl.n_tiles * pl.ks), pl.ks, (flags & kFlagNoPdl) == 0, &cfg, attr);
  cfg.stream = stream;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, f.kernel, tx, tw, p);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

}  // namespace b2
