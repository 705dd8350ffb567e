// W4A16 decode GEMV on the fifth-generation tensor cores, up to sixteen tokens, groups of 128:
// Y[M,N] (bf16) = X[M,K] (bf16) . dequant(Wq, S)^T with exact weights.
//
// The arithmetic is that of the mma.sync kernels: nibbles as signed bytes 16 (q - 8), X as block fixed point per (token,
// 128-chunk) in byte planes -- 16 bits above four tokens, 32 up to four --, integer products, one conversion to float per joined
// pair of planes and one fused multiply-add per (row, token, chunk).  Here the products run on tcgen05.mma (kind::i8):
//   * 128 weight rows are the M side; the bytes go from registers to tensor memory (three instructions per eight weights; a
//     thread owns a row) and the MMA reads them there.  The byte order the nibble masks give is the order X is stored in: the
//     contraction index is a dummy.  The planes' sixteen rows of bytes (signed, unsigned) are the N side;
//   * X is converted chunk by chunk by warps of its own, ahead of the products, into a ring in shared memory.  (Converted whole
//     before the first product it took 1 to 2 us that did not overlap, and its size forced K into clusters.);
//   * a hand-over is a pair of chunks, K = 256.  Two groups of warps take the pairs in turn: while one group's products run the
//     other converts words, and each reads and scales its sums when it comes back for its buffer;
//   * K is cut over a cluster.  A CTA sends its sums into the shared memory of the CTA that adds them, in the order of ranks and
//     groups (no second launch; st.async counted on a barrier of that CTA).
// What bounds it: HBM's rate once it runs (37888 x 3584 at four tokens: 7.5 TB/s from the seventh pair on, 70 MB in 11 of 15.4
// us; a pair 0.89 us, 5.6 TB/s); above eight tokens no unit alone (a pair at 13 tokens takes 1.09 us by 37888 x 14336 less 37888 x 3584,
// 2150 cycles at 1965 MHz: the issue slots are taken for 1140 of them, the words' bytes 96 instructions per row and pair, the sums 7
// per token, the conversion of X a sixth of all, and HBM runs at 4.6 TB/s; the rest are waits between a group's steps); and around
// that the boundary between launches: the wait for the kernel
// in front returns 0.9 us after its last CTA has left, a CTA starts 0.9 us after the one before it on the SM has (0.3 where
// neither uses tensor memory), first words and X 0.7 later, first products 0.5, the exchange of parts 0.9.
// The chain of a group is what the order in the loop is for: half of a pair's words are converted while the products of the group's last
// pair run, and the sums of that one are added while this pair's do (2530 -> 2300 cycles per pair of a group; 8192 x 28672 at
// eight tokens 30.7 -> 28.6 us).  The parts of a cut K go to the CTA that adds them with a barrier of their own instead of the
// cluster's (4608 x 3584 6.65 -> 5.8 us), tensor memory is freed beside the last sums.  Measured,
// weights from HBM, us at 4 / 8 / 13 tokens, in brackets before that: 37888 x 3584 15.2 / 15.4 / 16.9 (15.4 / 16.1 / 17.8), 3584 x 18944 12.4 / 12.6 / 14.7 (13.2 / 13.5 / 15.2), 4608 x 3584 at 4 and 13 5.8 and
// 6.8 (6.65 and 7.2), 57344 x 8192 at 8 57.9 (61.0).
// Every wait is bounded; a CTA that gives up records a status, still takes part in the cluster barriers and frees its TMEM.
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>

#include "ptx.cuh"
#include "tensor_map.h"
#include "w4_common.cuh"
#include "w4_internal.h"

namespace b2 {
namespace {

constexpr int kStepK = 128, kTokens = 16;
constexpr int kWSlot = 128 * 128;          // packed words: 128 rows, K = 256
constexpr int kXStep = 2 * 16 * 128;       // operand of a step: sixteen rows of unsigned bytes, sixteen of signed ones
constexpr int kXAhead = 2;                 // items of X a warp has in flight
constexpr int kBarOffset = 64;             // barriers of the rings; one per slot of X at kSlotBars
constexpr int kSlotBars = 512;
constexpr int kMaxPairs = 256;             // slots (pairs of steps) of a CTA
constexpr int kSmemHalf = 115712, kSmemFull = 232448;  // (228 KB / 2) - 1 KB, 227 KB

struct TcParams {
  const __nv_bfloat16* S;
  const __nv_bfloat16* X;
  __nv_bfloat16* Y;
  int* status;
  int M, N, K, KG;
  int pairs;    // of steps of 128
  int ks;       // CTAs of a cluster, each with its share of the pairs
  int sw, sx;   // ring slots of a pair: packed words (per block of 128 rows), X
  int ahead;    // slots of packed words that are brought into L2 ahead of the ring
  int x_first;  // the ring's further slots are not asked for before the first X is there
  int off_w, off_x, off_info, off_red;
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
template <int N>
__device__ __forceinline__ void regs_up() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void regs_down() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}
// The sums of a step: unsigned planes' columns from column 0, the signed plane's from column 16.
template <int LO>
__device__ __forceinline__ void tmem_ld_sums(uint32_t taddr, uint32_t (&d)[32]) {
  tmem_ld_32x32(taddr, d);
}
template <int LO>
__device__ __forceinline__ void tmem_ld_sums(uint32_t taddr, uint32_t (&d)[16]) {
  tmem_ld_32x8(taddr, d);
  if constexpr (LO == 8) {
    tmem_ld_32x8(taddr + 16, d + 8);
  } else {
    tmem_ld_32x4(taddr + 8, d + 8);
    tmem_ld_32x4(taddr + 16, d + 12);
  }
}

// MT: token columns (4, 8 or 16).  Four and fewer tokens keep X in 32 bits (three unsigned planes and a signed one), more
// in 16 (one and one).  MB: blocks of 128 weight rows.  SV: scales per load.  TOGETHER: a cluster's CTAs leave as one (gemv_tc_launch).
template <int MB, int MT, int SV, bool TOGETHER = false>
__global__ void __launch_bounds__(MB == 2 ? 896 : 512, MB == 2 ? 1 : 2)
    w4_gemv_tc_kernel(const __grid_constant__ CUtensorMap tmap_w, const TcParams p) {
  constexpr int P = MT == 4 ? 4 : 2;
  constexpr int kLo = MT * (P - 1), kCols = MT * P;  // columns of a row's sums: unsigned planes, then the signed one
  constexpr int kRows = MB * 128, kMain = 8 * MB, kBlocks = kRows / 32, kTmemCols = 256 * MB;
  constexpr int kWarps = MB == 2 ? 28 : 16, kXWarps = 4 * MB;
  constexpr int kWarpW = kMain + kXWarps, kWarpMma = kWarpW + 1;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* gen = smem_raw + (base - smem_u32(smem_raw));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen + 4);
  const uint32_t bar_w_full = base + kBarOffset, bar_w_empty = bar_w_full + 8 * 8;  // [block][slot], at most 4 slots
  const uint32_t bar_a_full = bar_w_empty + 8 * 8, bar_a_empty = bar_a_full + 8 * 4;  // [block][group]
  const uint32_t bar_x_empty = bar_a_empty + 8 * 4;                                   // [slot], at most 16
  const uint32_t bar_x_full = base + kSlotBars;                                       // [pair]
  const uint32_t bar_red = base + 16;                                                 // the parts of a cut K
  const uint32_t bar_done = base + 24;                                                // tensor memory has been read
  const uint32_t ring_w = base + p.off_w, ring_x = base + p.off_x, info = base + p.off_info, red = base + p.off_red;

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int crank = p.ks > 1 ? (int)cluster_rank() : 0;
  const int n0 = (blockIdx.x / p.ks) * kRows;
  const int pr0 = (int)((long)crank * p.pairs / p.ks), np = (int)((long)(crank + 1) * p.pairs / p.ks) - pr0;
  const int groups = (p.M + 3) >> 2;  // of four tokens: one warp's piece of a step's X
  // the blocks of 32 rows that this CTA of a cluster adds up
  const int first_blk = (crank * kBlocks + p.ks - 1) / p.ks, blks = ((crank + 1) * kBlocks + p.ks - 1) / p.ks - first_blk;

  for (int i = tid; i < np; i += kWarps * 32) mbar_init(bar_x_full + 8 * i, 2 * groups);
  // (the barriers of the rings lie one behind the other: 8 + 8 + 4 + 4 + 16)
  if (tid < 40) mbar_init(base + kBarOffset + 8 * tid, tid < 8 ? 1 : tid < 20 ? 4 : tid < 24 ? 1 : MB);
  if (tid == 0) {
    *abort_flag = 0;
    mbar_init(bar_done, kMain);
    if (p.ks > 1) {
      mbar_init(bar_red, 1);
      mbar_arrive_expect_tx(bar_red, (uint32_t)(blks * p.ks * 2 * groups) * 512);
    }
  }
  fence_mbar_init();
  if (warp == kWarpW && lane == 0) tma_prefetch_desc(&tmap_w);
  if (warp == kWarpMma) {
    tmem_alloc(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  pdl_launch_dependents();
  if (p.ks > 1) cluster_arrive();  // (waited for before the first store into a peer: it runs by then, its barrier is set up)
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);  // [block][group]: 64 columns of sums, 64 of bytes
  // (Read by every warp for itself: another CTA may set it in between, so the named barrier below is met either way.  Asked for ahead
  // of the __syncthreads it cost four layers at 4 tokens 155.4 us for 153.6 and at 13 187.3 for 182.4, since all then wait for it.)
  const bool poisoned = __any_sync(0xffffffffu, *reinterpret_cast<volatile int*>(p.status) != 0);
  // The rows' warps need more registers than an even share.  256 rows, 896 threads of 72: 4 x 88 + 2 x 48 + 56 = 7 x 72 by
  // warpgroup; 128 rows, 512 of 64: 2 x 80 + 2 x 48 = 4 x 64.
  if (warp < kMain) regs_up<MB == 2 ? 88 : 80>();
  else if (warp < kWarpW) regs_down<48>();
  else regs_down<MB == 2 ? 56 : 48>();
  // Behind this the rows' warps leave tensor memory alone: the warp that allocated it frees it while they add up and store.
  // (A kernel that frees it last ends 0.14 us later.)
  auto rows_done = [&] { mbar_arrive_if(bar_done, lane == 0); };
  if (!poisoned) {
    if (warp < kMain) {
      // ---- the rows: words -> bytes in TMEM; sums of a step -> registers.  Two groups of warps take the pairs in turn.
      const int quad = warp & 3, mb = (warp >> 2) % MB, grp = warp / (4 * MB);
      const int row = mb * 128 + quad * 32 + lane, n = n0 + row;  // (a warp may touch a quarter of the TMEM lanes)
      const bool live = n < p.N;
      const __nv_bfloat16* s_row = p.S + (size_t)(live ? n : 0) * p.KG;
      auto load_sv = [&](int v) {
        uint2 r = make_uint2(0u, 0u);
        if (live && v * SV < p.KG) {
          if (SV == 4) r = __ldcg(reinterpret_cast<const uint2*>(s_row + v * SV));
          else r.x = __ldcg(reinterpret_cast<const uint32_t*>(s_row + v * SV));
        }
        return r;
      };
      int g = 2 * (pr0 + grp);  // the pair's first step: even
      if (live && g < p.KG) prefetch_l2(s_row + g);  // (the second group has none where the CTA's share is one pair)
      // (with rows of S that start anywhere in a sector the share's next two; 755 x 18688 at three tokens 8.0 -> 7.7 us.  Tiles of 256 rows
      // lost 1 % by it.)
      if (const int next = 2 * pr0 + min(2 * np - 2, 14 + 2 * grp); SV == 2 && MB == 1 && MT < 16 && np > 2 && live && next < p.KG) prefetch_l2(s_row + next);
      pdl_wait_prior_grid();
      // SV == 4: two pairs, this group's one of them; SV == 2: one
      auto pair_scales = [&](int step) {
        const uint2 v = load_sv(step / SV);
        return SV == 4 && (step & 2) ? v.y : v.x;
      };
      uint32_t cur = pair_scales(g), nxt = pair_scales(g + 4);
      const uint32_t slot0 = ring_w + mb * p.sw * kWSlot + (quad * 32 + lane) * 128, swz = (uint32_t)lane & 7u;
      const uint32_t d_src = tmem + ((uint32_t)(quad * 32) << 16) + (mb * 2 + grp) * 128, a_dst = d_src + 64;
      const uint32_t b_wf = bar_w_full + 32 * mb, b_we = bar_w_empty + 32 * mb;
      const uint32_t b_af = bar_a_full + 8 * (mb * 2 + grp), b_ae = bar_a_empty + 8 * (mb * 2 + grp);
      if (p.ks > 1) cluster_wait();
      float acc[MT];
#pragma unroll
      for (int e = 0; e < MT; ++e) acc[e] = 0.f;
      // the sums of a step: planes joined as integers, ...
      auto join = [&](const uint32_t (&d)[kCols], int (&j)[kCols / 2]) {
#pragma unroll
        for (int t = 0; t < MT; ++t) {
          j[t] = (int)d[t] + ((int)d[MT + t] << 8);
          if constexpr (P == 4) j[MT + t] = (int)d[2 * MT + t] + ((int)d[3 * MT + t] << 8);
        }
      };
      // ... one conversion per pair, then scale times the token's factor
      auto add_step = [&](int step, float scale, const int (&j)[kCols / 2]) {
        const float2 scale2 = make_float2(scale, scale);
#pragma unroll
        for (int q = 0; q < MT / 4; ++q) {
          const uint4 f = lds128(info + (step * MT + q * 4) * 4);
          const float2 ff[2] = {make_float2(__uint_as_float(f.x), __uint_as_float(f.y)),
                                make_float2(__uint_as_float(f.z), __uint_as_float(f.w))};
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float v[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int t = q * 4 + h * 2 + e;
              v[e] = (float)j[t];
              if constexpr (P == 4) v[e] = fmaf((float)j[MT + t], 65536.f, v[e]);
            }
            float2 a = make_float2(acc[q * 4 + h * 2], acc[q * 4 + h * 2 + 1]);
            a = fma_f32x2(mul_f32x2(scale2, ff[h]), make_float2(v[0], v[1]), a);
            acc[q * 4 + h * 2] = a.x;
            acc[q * 4 + h * 2 + 1] = a.y;
          }
        }
      };
      // Takes the sums of pair i out of tensor memory; `then` runs as soon as the products may write there again.
      auto add_pair = [&](int i, auto&& then) {
        uint32_t d0[kCols], d1[kCols];
        int j[kCols / 2];
        tmem_ld_sums<kLo>(d_src, d0);
        if constexpr (MT == 16) {  // (no registers for 64 sums)
          tmem_ld_wait();
          join(d0, j);
        }
        tmem_ld_sums<kLo>(d_src + 32, d1);
        tmem_ld_wait();
        then();
        const uint32_t far = pair_scales(g + 8);  // (asked for ahead of the sums: behind them short launches were up to 2 % longer)
        if constexpr (MT != 16) join(d0, j);
        add_step(2 * i, __uint_as_float(cur << 16), j);
        join(d1, j);
        add_step(2 * i + 1, __uint_as_float(cur & 0xFFFF0000u), j);
        cur = nxt;
        g += 4;
        nxt = far;
      };
      uint32_t v[32];  // a step's bytes
      auto convert = [&](uint32_t slot, int half) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 w = lds128(slot + (((uint32_t)(half * 4 + j) ^ swz) << 4));
          const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
          for (int h = 0; h < 2; ++h) {  // two words: their even nibbles, their odd nibbles
            v[8 * j + 4 * h] = ((ww[2 * h] << 4) & 0xF0F0F0F0u) ^ 0x80808080u;
            v[8 * j + 4 * h + 1] = ((ww[2 * h + 1] << 4) & 0xF0F0F0F0u) ^ 0x80808080u;
            v[8 * j + 4 * h + 2] = (ww[2 * h] & 0xF0F0F0F0u) ^ 0x80808080u;
            v[8 * j + 4 * h + 3] = (ww[2 * h + 1] & 0xF0F0F0F0u) ^ 0x80808080u;
          }
        }
      };
      int s = grp;  // (the ring has an even number of slots: a group's slots are its own)
      uint32_t wph = 0, aph = 0;
      for (int i = grp; i < np; i += 2) {
        // Half of the words are converted while the products of the group's last pair may still run; its sums are added while
        // those of this pair do.
        const uint32_t slot = slot0 + s * kWSlot, b_we_this = b_we + 8 * s;
        // (asked for no earlier: with the question behind the last hand-over 4 tokens took 153.3 us for 151.9, 2 x 791 x 19712 9.5 for 9.1)
        mbar_wait(b_wf + 8 * s, wph, abort_flag);
        __syncwarp();
        s += 2;
        if (s >= p.sw) {
          s -= p.sw;
          wph ^= 1;
        }
        convert(slot, 0);
        if (i >= 2) {
          // the bytes of the group's last pair have been read and its sums are complete; so is that pair's X, whose factors
          // were written before it
          if (!__all_sync(0xffffffffu, mbar_try_wait2(b_ae, aph, bar_x_full + 8 * (i - 2), 0))) {
            mbar_wait(b_ae, aph, abort_flag);
            mbar_wait(bar_x_full + 8 * (i - 2), 0, abort_flag);
            __syncwarp();
          }
          aph ^= 1;
          tc_fence_after_sync();
        }
        tmem_st_32x32(a_dst, v);
        convert(slot, 1);
        tmem_st_32x32(a_dst + 32, v);
        auto hand_over = [&] {
          tmem_st_wait();
          tc_fence_before_sync();
          __syncwarp();
          mbar_arrive_if(b_af, lane == 0);
          mbar_arrive_if(b_we_this, lane == 0);
        };
        if (i >= 2)
          add_pair(i - 2, hand_over);
        else
          hand_over();
      }
      if (const int last = np - 1 - ((np - 1 - grp) & 1); last >= 0) {  // the group's last pair
        mbar_wait(b_ae, aph, abort_flag);
        mbar_wait(bar_x_full + 8 * last, 0, abort_flag);
        __syncwarp();
        tc_fence_after_sync();
        add_pair(last, [&] {
          tc_fence_before_sync();
          __syncwarp();
        });
      }
      rows_done();
      if (p.ks == 1) {  // the second group's sums through shared memory
        float* part = reinterpret_cast<float*>(gen + p.off_red) + (row >> 5) * (MT * 32) + lane;
        if (grp == 1) {
#pragma unroll
          for (int e = 0; e < MT; ++e)
            if (e < p.M) part[e * 32] = acc[e];
        }
        asm volatile("bar.sync %0, 256;" ::"r"(1 + mb) : "memory");
        if (grp == 0) {
          __nv_bfloat16* y = p.Y + n;
#pragma unroll
          for (int e = 0; e < MT; ++e)
            if (live && e < p.M) y[(size_t)e * p.N] = __float2bfloat16(acc[e] + part[e * 32]);
        }
      } else {
        // Every part goes to the CTA that sums its block of 32 rows, block * ks / kBlocks of the cluster, which adds the parts
        // in the order of ranks and groups: [block][rank][group][four tokens][32 rows]
        const int blk = row >> 5, owner = blk * p.ks / kBlocks, first = (owner * kBlocks + p.ks - 1) / p.ks;
        const uint32_t at = red + (uint32_t)((((blk - first) * p.ks + crank) * 2 + grp) * (MT / 4) * 32 + lane) * 16;
#pragma unroll
        for (int q = 0; q < MT / 4; ++q)
          if (q < groups) st_async_f4(at + q * 512, bar_red, owner, acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
        if (warp < blks * groups) {
          mbar_wait(bar_red, 0, abort_flag);
          __syncwarp();
        }
        for (int item = warp; item < blks * groups; item += kMain) {
          const int b = item / groups, q = item - b * groups, ny = n0 + (first_blk + b) * 32 + lane;
          const uint32_t part = red + (uint32_t)((b * p.ks * 2 * (MT / 4) + q) * 32 + lane) * 16;
          float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
          for (int z = 0; z < 2 * p.ks; ++z) {
            const uint4 f = lds128(part + z * (MT / 4) * 512);
            sum[0] += __uint_as_float(f.x);
            sum[1] += __uint_as_float(f.y);
            sum[2] += __uint_as_float(f.z);
            sum[3] += __uint_as_float(f.w);
          }
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (ny < p.N && q * 4 + e < p.M) p.Y[(size_t)(q * 4 + e) * p.N + ny] = __float2bfloat16(sum[e]);
        }
      }
    } else if (warp < kWarpW) {
      // ---- X: a warp takes four tokens of a step, a lane 16 consecutive k of a token, the eight lanes of a token side by
      // side.  The largest magnitude of a (token, step) is scaled to below 2^15 (2^31), its values are rounded to integers
      // and split into bytes, in the order the nibble masks produce.
      pdl_wait_prior_grid();
      constexpr int kGroups = MT / 4, kStride = kXWarps / kGroups;  // steps between a warp's items
      const int r = lane & 7, m = ((warp - kMain) % kGroups) * 4 + (lane >> 3), steps = 2 * np;
      const bool mine = ((warp - kMain) % kGroups) < groups, valid = m < p.M;
      const uint4* src = reinterpret_cast<const uint4*>(p.X + (size_t)(valid ? m : 0) * p.K + (size_t)(2 * pr0) * kStepK + r * 16);
      uint4 va[kXAhead], vb[kXAhead];  // items in flight
      auto load = [&](int step, uint4& a, uint4& b) {
        a = b = make_uint4(0u, 0u, 0u, 0u);
        if (step < steps && valid) {
          a = __ldcg(src + step * (kStepK / 8));
          b = __ldcg(src + step * (kStepK / 8) + 1);
        }
      };
      const int step0 = mine ? (warp - kMain) / kGroups : steps;
#pragma unroll
      for (int u = 0; u < kXAhead; ++u) load(step0 + u * kStride, va[u], vb[u]);
      int sl = step0 >> 1;
      uint32_t xph = 1;
      for (int step = step0; step < steps; step += kStride) {
        while (sl >= p.sx) {
          sl -= p.sx;
          xph ^= 1;
        }
        const uint32_t w[8] = {va[0].x, va[0].y, va[0].z, va[0].w, vb[0].x, vb[0].y, vb[0].z, vb[0].w};
#pragma unroll
        for (int u = 0; u + 1 < kXAhead; ++u) {
          va[u] = va[u + 1];
          vb[u] = vb[u + 1];
        }
        load(step + kXAhead * kStride, va[kXAhead - 1], vb[kXAhead - 1]);
        const bool room = mbar_test_wait(bar_x_empty + 8 * sl, xph);
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
        const float down = __uint_as_float((uint32_t)((P == 4 ? 284 : 268) - (int)eb) << 23);
        uint32_t v[16];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float lo = __uint_as_float(w[i] << 16), hi = __uint_as_float(w[i] & 0xFFFF0000u);
          if constexpr (P == 2) {  // the low mantissa bits of x * 2^.. + 1.5 * 2^23
            v[2 * i] = __float_as_uint(fmaf(lo, down, 12582912.f));
            v[2 * i + 1] = __float_as_uint(fmaf(hi, down, 12582912.f));
          } else {
            v[2 * i] = (uint32_t)__float2int_rn(lo * down);
            v[2 * i + 1] = (uint32_t)__float2int_rn(hi * down);
          }
        }
        if (!room) mbar_wait(bar_x_empty + 8 * sl, xph, abort_flag);
        if (valid) {
          const uint32_t at = ring_x + (2 * sl + (step & 1)) * kXStep;
#pragma unroll
          for (int pl = 0; pl < P; ++pl) {
            // plane pl of token m: row pl MT + m of the unsigned operand, row m of the signed one behind its 16 rows
            const int row = pl + 1 < P ? pl * MT + m : 16 + m;
            uint32_t o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int b = (j & 1) * 8 + (j >> 1);  // first k of the word: 0, 8, 1, 9; then every second one
              const uint32_t sel = pl < 2 ? 0x5140 : 0x7362;
              const uint32_t t0 = __byte_perm(v[b], v[b + 2], sel), t1 = __byte_perm(v[b + 4], v[b + 6], sel);
              o[j] = __byte_perm(t0, t1, pl & 1 ? 0x7632 : 0x5410);
            }
            sts128(at + row * 128 + (((uint32_t)r ^ (uint32_t)row) & 7u) * 16, make_uint4(o[0], o[1], o[2], o[3]));
          }
          if (r == 0)
            asm volatile("st.shared.b32 [%0], %1;" ::"r"(info + (step * MT + m) * 4),
                         "r"(bad ? 0x7FC00000u : (uint32_t)((int)eb - (P == 4 ? 34 : 18)) << 23)
                         : "memory");
        }
        fence_proxy_async_smem();
        __syncwarp();
        mbar_arrive_if(bar_x_full + 8 * (step >> 1), lane == 0);
        sl += ((step + kStride) >> 1) - (step >> 1);
      }
    } else if (warp == kWarpW) {
      // ---- packed words.  The kernel in front may be the one that writes them: until it has finished they are only
      // brought into L2, p.ahead slots of them.
      if (lane == 0) {
        for (int i = 0; i < np && i < p.ahead; ++i) {
#pragma unroll
          for (int mb = 0; mb < MB; ++mb) tma_prefetch_2d(&tmap_w, (pr0 + i) * 32, n0 + mb * 128);
        }
        pdl_wait_prior_grid();
        int s = 0;
        uint32_t ph = 1;
        for (int i = 0; i < np; ++i) {
#pragma unroll
          for (int mb = 0; mb < MB; ++mb) {
            if (i >= p.sw) mbar_wait(bar_w_empty + 32 * mb + 8 * s, ph, abort_flag);
            mbar_arrive_expect_tx(bar_w_full + 32 * mb + 8 * s, kWSlot);
            tma_load_2d(ring_w + (mb * p.sw + s) * kWSlot, &tmap_w, (pr0 + i) * 32, n0 + mb * 128,
                        bar_w_full + 32 * mb + 8 * s);
          }
          if (++s == p.sw) { s = 0; ph ^= 1; }
          if (i == 0 && p.x_first) mbar_wait(bar_x_full, 0, abort_flag);
        }
      }
      __syncwarp();
    } else if (warp < kWarpMma + MB) {
      // ---- products, one warp per block of rows: the whole warp runs the loop and one elected lane issues (the
      // descriptors then stay in uniform registers)
      const int mb = warp - kWarpMma;
      constexpr uint32_t id_lo = umma_idesc_s8(0, 128, 16), id_hi = umma_idesc_s8(1, 128, 16);
      const uint64_t desc0 = umma_desc_k128(ring_x);
      pdl_wait_prior_grid();  // the kernel in front may run longer than a bounded wait for X
      int xs = 0;
      for (int i = 0; i < np; ++i) {
        const uint32_t b_af = bar_a_full + 8 * (mb * 2 + (i & 1)), aph = (i >> 1) & 1;
        if (!__all_sync(0xffffffffu, mbar_try_wait2(bar_x_full + 8 * i, 0, b_af, aph))) {
          mbar_wait(bar_x_full + 8 * i, 0, abort_flag);
          mbar_wait(b_af, aph, abort_flag);
          __syncwarp();
        }
        tc_fence_after_sync();
        const uint64_t db = desc0 + xs * (2 * kXStep >> 4);
        const uint32_t d = tmem + (mb * 2 + (i & 1)) * 128, a = d + 64;
        if (elect_one()) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              umma_i8_ts(d + h * 32, a + h * 32 + kk * 8, db + h * (kXStep >> 4) + kk * 2, id_lo, kk > 0 ? 1u : 0u);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              umma_i8_ts(d + h * 32 + 16, a + h * 32 + kk * 8, db + h * (kXStep >> 4) + (16 * 128 >> 4) + kk * 2, id_hi,
                         kk > 0 ? 1u : 0u);
          }
          umma_commit(bar_a_empty + 8 * (mb * 2 + (i & 1)));
          umma_commit(bar_x_empty + 8 * xs);
        }
        __syncwarp();
        // With rows of S that start anywhere in a sector (K / 256 odd) some lane's next scales come from HBM in every pair, which
        // takes longer than a group's turn: the sector of eight pairs ahead is brought into L2.  26965 x 12544 at 5 tokens 43.0 -> 40.4
        // us, 14289 x 25856 at 6 47.1 -> 43.5.  Here, since the same in the rows' warps cost short launches 1 %.
        if constexpr (SV == 2 && (MB == 2 || MT < 16)) {
          if ((i & 7) == 0 && i + 8 < np) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              const int n = n0 + mb * 128 + r * 32 + lane;
              if (n < p.N) prefetch_l2(p.S + (size_t)n * p.KG + 2 * (pr0 + i) + 16);
            }
          }
        }
        if (++xs == p.sx) xs = 0;
      }
    }
  } else if (p.ks == 1 && warp < kMain) {  // the block's other warps may be there, and this barrier has no limit
    asm volatile("bar.sync %0, 256;" ::"r"(1 + (warp >> 2) % MB) : "memory");
  }
  __syncwarp();
  if (poisoned && lane == 0) *abort_flag = 1;  // the CTA's other warps may have read zero: their waits end
  bool freed = false;
  if (warp == kWarpMma && !poisoned) {
    mbar_wait(bar_done, 0, abort_flag);
    if (!__any_sync(0xffffffffu, *abort_flag != 0)) {  // (every product has been waited for)
      tc_fence_after_sync();
      tmem_dealloc(tmem, kTmemCols);
      freed = true;
    }
  }
  if (p.ks > 1 && (warp >= kMain || poisoned)) cluster_wait();
  __syncthreads();
  if constexpr (TOGETHER) {  // (p.ks > 1)
    cluster_arrive();
    cluster_wait();
  }
  if (*abort_flag) {
    if (!TOGETHER && p.ks > 1) {  // peers that have not given up may send parts here until they leave
      cluster_arrive();
      cluster_wait();
    }
    if (tid == 0) atomicCAS(p.status, kStatusOk, kStatusGemvTimeout);
    for (int i = 0; i < 64; ++i) __nanosleep(2000);  // copies in flight land before the shared memory is released
    __syncthreads();
  }
  if (warp == kWarpMma && !freed) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, kTmemCols);
  }
}

using TcKernel = void (*)(const CUtensorMap, const TcParams);

struct TcPlan {
  int form = 0, ks = 1, pairs = 0;  // form 0: 128 rows, two CTAs per SM; 1: 256 rows, one
  double us = 0;                    // (what plans are compared by)
  double busy = 0;                  // the share of the places for CTAs that are taken
  bool several = false;             // waves, with K whole: the line of its own
};

int tc_tokens(int M) { return M <= 4 ? 4 : M <= 8 ? 8 : 16; }

// Shared memory of a plan: offsets from the 1024-aligned base.
void tc_layout(const TcPlan& pl, int M, TcParams* p) {
  const int mt = tc_tokens(M), mb = pl.form + 1, blocks = 4 * mb, room = (mb == 2 ? kSmemFull : kSmemHalf) - 1024;
  const int info = 2 * pl.pairs * mt * 4, red = (blocks + pl.ks - 1) / pl.ks * pl.ks * 2 * mt * 128;
  p->off_w = (kSlotBars + 8 * pl.pairs + 1023) / 1024 * 1024;
  for (p->sw = 4;; p->sw = 2) {  // even: a slot belongs to one group
    p->off_x = p->off_w + mb * p->sw * kWSlot;
    p->sx = std::min(8, (room - 16 - p->off_x - info - red) / (2 * kXStep));
    if (p->sx >= 2 || p->sw == 2) break;
  }
  p->off_info = p->off_x + p->sx * 2 * kXStep;
  p->off_red = (p->off_info + info + 15) / 16 * 16;
}

template <int MB, int SV>
TcKernel tc_kernel_mt(int mt) {
  return mt == 4 ? w4_gemv_tc_kernel<MB, 4, SV> : mt == 8 ? w4_gemv_tc_kernel<MB, 8, SV> : w4_gemv_tc_kernel<MB, 16, SV>;
}
template <int SV>
TcKernel tc_kernel_together(int mt) {
  return mt == 4   ? w4_gemv_tc_kernel<2, 4, SV, true>
         : mt == 8 ? w4_gemv_tc_kernel<2, 8, SV, true>
                   : w4_gemv_tc_kernel<2, 16, SV, true>;
}
// kind: a form, or 2: 256 rows, a cluster's CTAs leave together
TcKernel tc_kernel(int kind, int mt, bool sv4) {
  if (kind == 2) return sv4 ? tc_kernel_together<4>(mt) : tc_kernel_together<2>(mt);
  return kind ? (sv4 ? tc_kernel_mt<2, 4>(mt) : tc_kernel_mt<2, 2>(mt)) : (sv4 ? tc_kernel_mt<1, 4>(mt) : tc_kernel_mt<1, 2>(mt));
}
int tc_attributes(TcKernel kernel, int kind, int mt, bool sv4, int dev) {
  static std::atomic<bool> done[64][3][2][3];
  const bool cached = dev >= 0 && dev < 64;
  if (cached && done[dev][kind][sv4][mt / 8].load(std::memory_order_acquire)) return 0;
  const cudaError_t e =
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kind ? kSmemFull : kSmemHalf);
  if (e == cudaSuccess && cached) done[dev][kind][sv4][mt / 8].store(true, std::memory_order_release);
  return (int)e;
}
void tc_config(int form, int grid, int ks, bool pdl, cudaLaunchConfig_t* cfg, cudaLaunchAttribute (&attr)[2]) {
  cfg->gridDim = dim3(grid);
  cfg->blockDim = dim3(form ? 896 : 512);
  cfg->dynamicSmemBytes = form ? kSmemFull : kSmemHalf;  // all of it: at most 512 TMEM columns' worth of CTAs fit on an SM
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

// CTAs of a form that the device runs at a time in clusters of ks: a cluster stays inside one GPC, so some SMs are left out (256
// rows: 148 of 148 in twos, 135, 132, 130, 132, 105, 120 in threes to eights).  Asked for once per device.
int tc_capacity(int form, int ks, int sm_count, int dev) {
  if (ks == 1) return sm_count * (form ? 1 : 2);
  static std::atomic<int> known[64][2][9];
  const bool cached = dev >= 0 && dev < 64;
  if (cached)
    if (const int v = known[dev][form][ks].load(std::memory_order_relaxed)) return v;
  const TcKernel kernel = tc_kernel(form, 8, true);
  int clusters = 0;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[2];
  tc_config(form, ks, ks, false, &cfg, attr);
  if (tc_attributes(kernel, form, 8, true, dev) != 0 ||
      cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || clusters < 1) {
    (void)cudaGetLastError();
    clusters = std::max(1, sm_count * (form ? 1 : 2) / ks * 7 / 8);
  }
  if (cached) known[dev][form][ks].store(clusters * ks, std::memory_order_relaxed);
  return clusters * ks;
}

// Estimated time (us), a fit to 466 shapes in every form and cluster size (256 to 60000 x 256 to 28672, weights from HBM): start,
// exchange through the cluster, waves of CTAs that take their pairs of steps at the rate of a warp group's chain or of HBM.  The
// 128-row form shares an SM with a second CTA where K is cut or there are more CTAs than SMs.  Several waves with K whole have
// a line of their own (26 shapes of 38000 to 60000 rows): the 256-row form takes whole waves, the 128-row one lets a CTA start
// wherever one ends (53886 x 5632 at three tokens 35 us against 41; 57344 x 8192 60 against 58).  Over 6472 calls on 1627 shapes what
// it picks takes 1.016 times the best plan's time in the geometric mean, 1.11 times in one of twenty; its own time is 6 % short there
// (12 % in the standard deviation), most where the chip is full: gemv_tc_shorter adds that.
bool tc_find_plan(int M, int N, int K, int sm_count, int dev, int wanted_form, int wanted_ks, TcPlan* out) {
  static constexpr double kChain[2][3] = {{0.541, 0.582, 0.879}, {0.734, 0.775, 0.913}}, kShared[3] = {1.042, 1.121, 1.593};
  static constexpr double kToken[3] = {0.0, 0.141, 0.359}, kWave[3] = {0.84, 0.84, 1.04}, kFluid[3] = {0.87, 0.93, 1.35};
  const int total = K / (2 * kStepK), mc = M <= 4 ? 0 : M <= 8 ? 1 : 2;
  bool any = false;
  for (int form = 0; form < 2; ++form) {
    if (wanted_form && form != wanted_form - 1) continue;
    const int rows = form ? 256 : 128;
    const long tiles = (N + rows - 1) / rows;
    for (int ks = 1; ks <= 8 && ks <= total; ++ks) {
      if (wanted_ks && ks != std::min({wanted_ks, 8, total})) continue;
      TcPlan pl;
      pl.form = form;
      pl.ks = ks;
      pl.pairs = (total + ks - 1) / ks;
      if (pl.pairs > kMaxPairs || tiles * ks > 0x3fffffff) continue;
      const long cap = tc_capacity(form, ks, sm_count, dev), ctas = tiles * ks, waves = (ctas + cap - 1) / cap;
      const double act = (double)std::min(ctas, cap);
      pl.busy = act / cap;
      pl.several = waves > 1 && ks == 1;
      const double mix = form ? 0.053 : 0.736;
      const double eff = waves == 1 ? 1.0 : (1.0 - mix) * waves + mix * ctas / cap, in_caps = (double)ctas / cap;
      double chain = kChain[form][mc];
      if (form == 0 && (ks > 1 || ctas > sm_count)) chain = kShared[mc] * std::min(1.0, 0.385 + 0.615 * act / (2.0 * sm_count));
      const double pair = std::max(chain, act * rows * 128 * 1.03 / 7.705e6);
      if (pl.several)
        pl.us = 3.0 + kToken[mc] + pl.pairs * (form ? kWave[mc] * waves : kFluid[mc] * (in_caps + 0.45));
      else
        pl.us = (waves > 1 ? 1.15 : 1.0) * ((form ? 2.0 : 1.76) + (ks > 1 ? 0.85 + 0.043 * ks : 0.0) + kToken[mc] + (eff - 1.0) * 4.23 +
                                            eff * pl.pairs * pair);
      if (!any || pl.us < out->us) *out = pl;
      any = true;
    }
  }
  return any;
}

// A call's rule and its launch ask for the same plan, one behind the other: 0.13 us of an eager call's 3.4 of host time each.
bool tc_plan(int M, int N, int K, int sm_count, int wanted_form, int wanted_ks, TcPlan* out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = -1;
  struct Asked {
    int key[7];
    TcPlan plan;
    bool any;
  };
  static thread_local Asked last{};
  const int key[7] = {M, N, K, sm_count, dev, wanted_form, wanted_ks};
  if (!std::equal(key, key + 7, last.key)) {
    last.any = tc_find_plan(M, N, K, sm_count, dev, wanted_form, wanted_ks, &last.plan);
    std::copy(key, key + 7, last.key);
  }
  *out = last.plan;
  return last.any;
}

bool tc_operands(const void* X, const void* Wq, const void* S, const void* Y, int M, int N, int K, int G) {
  if (G != kStepK || K < 2 * kStepK || K % (2 * kStepK) || N < 1 || M < 1 || M > kTokens) return false;
  return !(((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(Wq)) & 15) || (reinterpret_cast<uintptr_t>(Y) & 1) ||
           (reinterpret_cast<uintptr_t>(S) & 3));
}

}  // namespace

// (Pointers: null = "assume aligned", for the queries that have no operands.)
bool gemv_tc_serves(const void* X, const void* Wq, const void* S, const void* Y, int M, int N, int K, int G, int flags,
                    int sm_count) {
  TcPlan pl;
  return tc_operands(X, Wq, S, Y, M, N, K, G) && tc_plan(M, N, K, sm_count, (flags >> 24) & 3, (flags >> 20) & 15, &pl);
}

// Whether this kernel is shorter than the GEMV that would take a plain call of 1 to 16 tokens, `other` one of kTcOther*.  Lines
// drawn through 2044 calls on random shapes (128 to 60000 rows, K 512 to 28672, weights from HBM, one launch behind the other), every
// kernel and every plan of this one timed, and earlier through 6472 more.
//   * One token (streaming kernel): both hold X in 32 bits.  Only where that kernel has a weakness: up to twelve million weights a
//     launch is its latencies, and it converts the whole of X before its first product (512 x 3584 3.4 us against 4.5); between K of
//     9728 and 16384 it does so several times per thread (4980 x 14080 12.8 against 15.0), above 22000 it cuts K through memory
//     (8192 x 28672 26.6 against 29.2).  Within these lines, which cost a call's host side next to nothing, tiles of 128 rows as they
//     are and tiles of 256 by the estimates of both kernels: by the lines alone these took 3500 x 2048 (5.3 us for 4.4), 2861 x 3584
//     (5.6 for 5.1), 11771 x 28160 (54 for 39, 92 CTAs).  Of 3000 shapes like these 926 come here, 0.843 of their time there in
//     the geometric mean; of all 3000 22 lose 3 % and one 6, with the lines alone 98 and 49 (at most 41).
//   * Two to four tokens (streaming kernel; X has 15 bits there at three and four): shorter here but for many rows of a short K (21667 x
//     1024 at four tokens 4.8 us there, 5.5 here; 18944 x 3584 at two 9.6 and 10.7).  Of 150 calls five lose 3 % (at most 6).
//   * Many-token kernel, five and more tokens: by the estimates of both, this one's with what plans have in common (they come out
//     short where the chip is full): 1.008 and 1.003 times the shortest kernel's time up to eight tokens and above.
//   * Many-token kernel, two to four tokens (K >= 8192): X has 32 bits here and 16 there, so what a line in w (millions of weights),
//     M and K brought here stays.
//   * Ring kernel: never shorter.
bool gemv_tc_shorter(const void* X, const void* Wq, const void* S, const void* Y, int M, int N, int K, int G, int flags,
                     int sm_count, size_t partial_cap, TcOther other) {
  if (M < 1 || (flags & ~kFlagNoPdl) != 0 || !tc_operands(X, Wq, S, Y, M, N, K, G)) return false;
  const double w = 1e-6 * N * K, k3 = 1e-3 * K, mk = 1e-4 * M * K;
  // the lines in N and K first: a call of few tokens is bound by its host side, and most need no plan
  if (M == 1 && !(w <= 12.0 ? K >= 1024 : (K >= 9728 && K <= 16384 && N <= 4992) || (K >= 22016 && N >= 7424))) return false;
  if (M > 1 && other == kTcOtherStream &&
      !(M > 2       ? K >= 2304 || N <= 8000
        : K >= 3840 ? N <= 128 * (sm_count - 1)  // (above, that kernel's CTAs of 128 rows leave no SM over)
                    : N <= (K <= 1536 ? 5800 : 11000)))
    return false;
  TcPlan pl;
  if (!tc_plan(M, N, K, sm_count, 0, 0, &pl)) return false;
  if (M == 1) {
    if (!pl.form) return w > 12.0 || pl.us <= (N <= 4096 ? 8.5 : 3.5);
    if (pl.several) return false;
    return 1.04 * (0.862 * pl.us + 0.009 * w + 3.44 * pl.busy - 0.88) < gemv_stream_us(N, K, sm_count, partial_cap);
  }
  if (other != kTcOtherMany) return true;
  if (M <= 4) return 1.02 * pl.us < 6.65 + 0.11 * w + 0.027 * k3 + 0.074 * mk;
  const double us = pl.us + (pl.form       ? 2.03 * pl.busy * pl.busy
                             : pl.several ? 0.5
                                          : 0.025 * w + 0.7 * pl.busy - (pl.ks > 1 ? 0.34 : 0.0));
  return 1.02 * us < gemv_mid_us(M, N, K, sm_count, partial_cap);
}

int gemv_tc_describe(int M, int N, int K, int flags, int sm_count, char* buf, int buflen) {
  const bool forced = flags < 0;
  TcPlan pl;
  if (!tc_plan(M, N, K, sm_count, forced ? (flags >> 24) & 3 : 0, forced ? (flags >> 20) & 15 : 0, &pl)) return 0;
  const int rows = pl.form ? 256 : 128;
  TcParams p{};
  tc_layout(pl, M, &p);
  return snprintf(buf, buflen,
                  "tcgen05 GEMV: %d CTAs (%d per SM), tiles of %d rows x %d tokens, clusters of %d along K, %d planes (%d-bit "
                  "X), %d ring slots",
                  (N + rows - 1) / rows * pl.ks, pl.form ? 1 : 2, rows,
                  tc_tokens(M), pl.ks, M <= 4 ? 4 : 2, M <= 4 ? 32 : 16, p.sw);
}

// flags: bits 20-23 CTAs per cluster, bits 24-25 tile (1: 128 rows; 2: 256), 0 = the rule.
int gemv_tc_launch(const void* X, const void* Wq, const void* S, void* Y, int M, int N, int K, const Workspace& ws,
                   int flags, int sm_count, cudaStream_t stream) {
  TcParams p{};
  p.S = static_cast<const __nv_bfloat16*>(S);
  p.X = static_cast<const __nv_bfloat16*>(X);
  p.Y = static_cast<__nv_bfloat16*>(Y);
  p.status = ws.status;
  p.M = M; p.N = N; p.K = K;
  p.KG = K / kStepK;
  p.pairs = K / (2 * kStepK);
  const bool forced = flags < 0;
  TcPlan pl;
  if (!tc_plan(M, N, K, sm_count, forced ? (flags >> 24) & 3 : 0, forced ? (flags >> 20) & 15 : 0, &pl)) return kErrTooLarge;
  const int form = pl.form, rows = form ? 256 : 128, mt = tc_tokens(M);
  p.ks = pl.ks;
  tc_layout(pl, M, &p);
  p.ahead = 3;
  // Clusters of three that take every place the device has for them (45 on 148 SMs): where their CTAs leave one by one the next
  // launch's clusters start in other places and some find none, a wave of their own (11300 x 27392 at 4 tokens 32.8 us for 44 then;
  // 11500 x 14336 20.5 for 24.8).  Not below eight pairs to a CTA (11400 x 4096 9.1, together 9.7), nor for other sizes of clusters,
  // full or not: leaving together costs up to 0.7 us there (3800 x 14336 in clusters of eight 10.9 and 11.6).  A kernel of its own: asking
  // at the end cost short launches 2 %.
  const int kind = form && pl.ks == 3 && pl.pairs >= 8 && pl.busy > 0.97 ? 2 : form;
  // Where the rings of nearly all SMs fill at once X waits behind them for two microseconds: then only the first slot goes ahead
  // of it (8192 x 28672 at 8 tokens 30.2 -> 29.3 us, 37888 x 3584 at 13 17.4 -> 16.9).  Elsewhere it is X that is waited for (4608 x
  // 3584 at 4 tokens 5.8 against 6.1), and with a short K and few tokens it is there soon enough between other launches (four
  // 7B-shaped layers at 4 tokens 154.1 against 157.0, at 13 185.9 against 184.5).
  const long ctas = (long)((N + rows - 1) / rows) * p.ks;
  p.x_first = (mt == 16 || p.pairs > 16) && p.pairs / p.ks > 4 && ctas * 10 >= (form ? 8 : 9) * (long)sm_count;
  CUtensorMap tw;
  if (!make_tensor_map_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, Wq, (uint64_t)N, (uint64_t)K / 8, 128, 32,
                          CU_TENSOR_MAP_SWIZZLE_128B))
    return kErrDevice;
  const bool sv4 = p.KG % 4 == 0 && reinterpret_cast<uintptr_t>(S) % 8 == 0;
  const TcKernel kernel = tc_kernel(kind, mt, sv4);
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (const int rc = tc_attributes(kernel, kind, mt, sv4, dev)) return rc;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[2];
  tc_config(form, (N + rows - 1) / rows * p.ks, p.ks, (flags & kFlagNoPdl) == 0, &cfg, attr);
  cfg.stream = stream;
  e = cudaLaunchKernelEx(&cfg, kernel, tw, p);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

}  // namespace b2
