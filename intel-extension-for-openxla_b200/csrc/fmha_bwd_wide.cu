// Attention backward for head sizes above 128 (the reference's fmha_bwd_policy_64x128x256,
// xla/service/gpu/xetla/sdp/fmha_policy.h:107-116, dispatched at fmha_backward.h:931-938).
//
// With 256-wide heads the dK and dV accumulators of a 128-key block alone fill the 512 columns of
// tensor memory, so the single-kernel scheme of fmha_bwd_sm100.cu (S^T, dP^T, dK, dV resident
// together) does not fit.  Here a group of heads is taken in two steps, with P and dS as 16-bit [F, T]
// planes in scratch between them:
//   1. wide_scores_kernel:  S = Q.K^T and dP = dO.V^T into tensor memory side by side, then
//                           P = exp(head_scale*S + bias - lse) and dS = P * (dP - D), both stored once
//                                                                       (fmha_backward.h:489-700)
//   2. wide_grads_kernel:   dV = P^T.dO,   dK = head_scale * dS^T.Q,   dQ = head_scale * dS.K
// Both run on CTA pairs (tcgen05 cta_group::2) and follow the causal mask at tile granularity:
// score tiles above the diagonal are neither computed nor stored, and the K range of every gradient
// tile covers the stored tiles only.  P and dS are rounded to the element type where they become
// matmul operands, all sums are fp32, each gradient is rounded once.  D and -lse*log2(e) come from
// the shared prepare kernel.
//
// Measured at B4 N16 F=T=2048 H256 causal bf16, a call at a time with the L2 flushed: backward 2439 us as a
// chain of five GEMMs and two elementwise passes, 492 as it is: 26 the prepare kernel and four groups of
// 57 + 60 for the two kernels.  Forward and backward back to back, where the clock falls under the power cap:
// 2596 and 713.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "fmha_sm100.h"
#include "ptx.cuh"

namespace ixk {
namespace fmha {

namespace {

constexpr float kLog2e = 1.4426950408889634f;
constexpr int kRowBlock = 256;     // query (or key) rows of a CTA pair's tile: 128 per CTA
constexpr int kKeyTile = 128;      // keys of a score tile
constexpr int kSlabBytes = 128;    // one swizzle span: 64 16-bit elements
constexpr int kMaxSlabs = 4;       // head size <= 256
constexpr int kBoxBytes = 128 * kSlabBytes;   // 128 rows x 128 bytes
constexpr int kHalfBox = 64 * kSlabBytes;     // 64 rows x 128 bytes
constexpr size_t kGroupBudget = static_cast<size_t>(192) << 20;   // scratch per group of heads (see heads_per_group)
constexpr int kHeadChunk = 4;      // heads whose gradient tiles are sorted together

// Where a block of 256 query rows lies in a plane.  Unfolded: at its own rows.  Under a causal mask block
// qb has keys in its first 256 (qb + 1) columns only, so blocks qb and nq - 1 - qb can share one band of
// 256 rows and 256 (nq + 1) columns, which nearly halves the plane.
struct Fold {
  int on, nq;
  __host__ __device__ __forceinline__ bool second(int qb) const { return on != 0 && qb >= (nq + 1) / 2; }
  __host__ __device__ __forceinline__ int band(int qb) const { return second(qb) ? nq - 1 - qb : qb; }
  __host__ __device__ __forceinline__ int column(int qb) const { return second(qb) ? kRowBlock * (nq - qb) : 0; }
};

// wait sites reported in the device status word
enum : int { kSiteScoreQ = 0x51, kSiteScoreKv = 0x52, kSiteScoreAcc = 0x53, kSiteScoreFull = 0x54, kSiteScoreOut = 0x55,
              kSiteGradEmpty = 0x56, kSiteGradFull = 0x57, kSiteGradAcc = 0x58, kSiteGradOut = 0x59 };

__device__ __forceinline__ float bits_to_f32(uint16_t h, bool bf16) {
  return bf16 ? __uint_as_float(static_cast<uint32_t>(h) << 16) : __half2float(__ushort_as_half(h));
}
template <bool kBf16>
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi) {
  if constexpr (kBf16) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  } else {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
}

// 16 words of packed pairs (32 columns) of the calling lane's row into its warp's staging box: 32 rows
// x 128 bytes, swizzled the way a TMA store of 64 16-bit columns reads it (conflict-free).
__device__ __forceinline__ void stage_half_row(uint32_t box, int lane, int half, const uint32_t (&w)[16]) {
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const uint32_t addr = box + static_cast<uint32_t>(lane * 128 + (((half * 4 + g) ^ (lane & 7)) << 4));
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(w[4 * g]), "r"(w[4 * g + 1]), "r"(w[4 * g + 2]),
                 "r"(w[4 * g + 3])
                 : "memory");
  }
}

// ---------------------------------------------------------------------------------------------
// Step 1: P and dS.  A CTA pair works on 256 queries x 128 keys: each CTA keeps its 128 rows of Q and
// dO in shared memory (2 x 64 KB at head size 256) while the keys of a run go by, and loads half of
// every K and V slab (64 keys x 64 head elements) into a ring of 4 slots of two slabs; the even CTA's issuer drives
// both tensor cores.  S and dP are double-buffered in tensor memory (4 x 128 columns), so that the
// 256 compute threads of a CTA (one query row each, two warpgroups of 64 keys) work on one tile while
// the next one is multiplied.  The score tiles of a group are numbered (head, query block, key tile)
// and every pair takes an equal, contiguous share: a run inside one query block re-uses Q and dO, and
// the next run's slabs are requested one by one as the last tile of the current run releases them.
// Bytes through L2 per tile and CTA: 64 KB of K and V, 64 KB of P and dS, and Q and dO once per run,
// about 75 bytes per cycle of the tile's 2048 MMA cycles.
// What bounds it is the issuing warp (clock64 trace, 16 heads of 2048, 16 tiles a pair): of 71k cycles 33k are
// MMAs, 20k waits for loads (half of them at the start of a run) and the rest barrier round trips and
// commits between them; that is why a ring slot holds two slabs.  The stores are 15 % (without them 53 us for
// 62 then).  Twice the compute warps with 32 keys each, and two staging boxes per warp at the price of half the
// ring, were measured and dropped (no change, 5 us a group slower).
struct ScoreCfg {
  static constexpr int kRing = 4;                                   // slots of two K / V slab halves in flight
  static constexpr int kOffQ = 0;
  static constexpr int kOffDo = kMaxSlabs * kBoxBytes;
  static constexpr int kOffRing = 2 * kMaxSlabs * kBoxBytes;
  static constexpr int kOffStage = kOffRing + kRing * 2 * kHalfBox;     // one box per compute warp
  static constexpr int kOffBars = kOffStage + 8 * 32 * 128;
  static constexpr int kSmemBytes = kOffBars + 512 + 1024;          // + alignment slack
  static_assert(kSmemBytes <= 232448, "shared memory budget");
  static constexpr int kThreads = 384;                              // 8 compute warps, producer, issuer, 2 idle
  static constexpr int kProducerWarp = 8;
  static constexpr int kMmaWarp = 9;
};

struct ScoreArgs {
  int N, F, T, bn0, heads;     // heads of this group start at (batch, head) index bn0
  int f_pad;                   // row pitch of neg_lse2 / delta
  int nq, nk, tiles_per_head;
  int total_tiles;
  int slabs;                   // ceil(H / 64)
  int causal;
  Fold fold;
  uint32_t idesc;
  float scale_log2;
  const float* neg_lse2;
  const float* delta;
  const uint16_t* bias;
  int64_t bias_strides[3];
  int bias_vec;
  int* status_word;
};

// Consecutive key tiles of one (head, query block).
struct Run {
  int head, qb, kt0, kt1;
};
__device__ __forceinline__ int key_tiles_of(const ScoreArgs& a, int qb) { return a.causal ? min(a.nk, 2 * qb + 2) : a.nk; }
// The run that starts at flat tile index t and ends at the query block's end or before t_end.
__device__ __forceinline__ Run run_at(const ScoreArgs& a, int t, int t_end) {
  Run r;
  r.head = t / a.tiles_per_head;
  int rem = t - r.head * a.tiles_per_head;
  r.qb = 0;
  int n = key_tiles_of(a, 0);
  while (rem >= n) {
    rem -= n;
    n = key_tiles_of(a, ++r.qb);
  }
  r.kt0 = rem;
  r.kt1 = min(n, rem + (t_end - t));
  return r;
}

template <bool kBf16, bool kBias>
__global__ void __launch_bounds__(ScoreCfg::kThreads, 1)
wide_scores_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_do,
                   const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                   const __grid_constant__ CUtensorMap tmap_p, const __grid_constant__ CUtensorMap tmap_ds,
                   const __grid_constant__ ScoreArgs args) {
  using C = ScoreCfg;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - ptx::smem_u32(smem_raw));
  const uint32_t bars = smem_base + C::kOffBars;
  // Barriers go by two slabs (128 head elements): resident pairs 0, 1 are Q, 2, 3 are dO.
  auto res_full = [&](int s) { return bars + 8u * s; };
  auto res_empty = [&](int s) { return bars + 8u * (8 + s); };
  auto kv_full = [&](int s) { return bars + 8u * (16 + s); };
  auto kv_empty = [&](int s) { return bars + 8u * (24 + s); };
  auto acc_full = [&](int b) { return bars + 8u * (32 + b); };
  auto acc_empty = [&](int b) { return bars + 8u * (34 + b); };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + C::kOffBars + 8 * 36);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + C::kOffBars + 8 * 36 + 4);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();
  ptx::AbortCtl ctl{abort_flag, args.status_word};

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < 8; ++s) {
      ptx::mbar_init(res_full(s), 1);
      ptx::mbar_init(res_empty(s), 1);
      ptx::mbar_init(kv_full(s), 1);
      ptx::mbar_init(kv_empty(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(acc_full(b), 1);
      ptx::mbar_init(acc_empty(b), 2 * 256);   // the compute threads of both CTAs
    }
    ptx::fence_mbar_init();
    ptx::prefetch_tmap(&tmap_q);
    ptx::prefetch_tmap(&tmap_do);
    ptx::prefetch_tmap(&tmap_k);
    ptx::prefetch_tmap(&tmap_v);
    ptx::prefetch_tmap(&tmap_p);
    ptx::prefetch_tmap(&tmap_ds);
  }
  __syncthreads();
  ptx::cluster_sync_all();
  if (warp == C::kMmaWarp) {   // collective over the pair
    ptx::tmem_alloc_pair(ptx::smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::cluster_sync_all();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  // the planes written here may still be read by the previous group's gradient kernels
  ptx::grid_dependency_wait();
  ptx::grid_dependency_trigger();

  const int pair = blockIdx.x >> 1;
  const int64_t pairs = gridDim.x >> 1;
  const int t_begin = static_cast<int>(args.total_tiles * static_cast<int64_t>(pair) / pairs);
  const int t_end = static_cast<int>(args.total_tiles * static_cast<int64_t>(pair + 1) / pairs);

  if (warp == C::kProducerWarp) {
    // ------------------------------------------------------------ TMA producer (each CTA: its rows, its key halves)
    int st = 0;
    uint32_t ph = 0, res_ph = 0;
    bool alive = true;
    for (int t = t_begin; t < t_end && alive; res_ph ^= 1u) {
      const Run run = run_at(args, t, t_end);
      const int bn = args.bn0 + run.head;
      const int n = bn % args.N, b = bn / args.N;
      const int row0 = run.qb * kRowBlock + static_cast<int>(rank) * 128;
      for (int kt = run.kt0; kt < run.kt1 && alive; ++kt) {
        const int key0 = kt * kKeyTile + static_cast<int>(rank) * 64;
        for (int operand = 0; operand < 2 && alive; ++operand) {   // Q.K^T, then dO.V^T
          for (int s = 0; s < args.slabs; s += 2) {
            const int n_slabs = min(2, args.slabs - s);
            if (kt == run.kt0) {
              const int res = operand * 2 + (s >> 1);
              if (!ptx::mbar_wait(res_empty(res), res_ph ^ 1u, ctl, kSiteScoreQ)) {
                alive = false;
                break;
              }
              if (ptx::elect_one()) {
                if (rank == 0) ptx::mbar_expect_tx(res_full(res), n_slabs * 2 * kBoxBytes);
                for (int i = 0; i < n_slabs; ++i)
                  ptx::tma_load_4d_pair(smem_base + (operand * 4 + s + i) * kBoxBytes, operand == 0 ? &tmap_q : &tmap_do,
                                        ptx::map_to_cta(res_full(res), 0), (s + i) * 64, row0, n, b);
              }
              __syncwarp();
            }
            if (!ptx::mbar_wait(kv_empty(st), ph ^ 1u, ctl, kSiteScoreKv)) {
              alive = false;
              break;
            }
            if (ptx::elect_one()) {
              if (rank == 0) ptx::mbar_expect_tx(kv_full(st), n_slabs * 2 * kHalfBox);
              for (int i = 0; i < n_slabs; ++i)
                ptx::tma_load_4d_pair(smem_base + C::kOffRing + (2 * st + i) * kHalfBox, operand == 0 ? &tmap_k : &tmap_v,
                                      ptx::map_to_cta(kv_full(st), 0), (s + i) * 64, key0, n, b);
            }
            __syncwarp();
            if (++st == C::kRing) {
              st = 0;
              ph ^= 1u;
            }
          }
        }
      }
      t += run.kt1 - run.kt0;
    }
  } else if (warp == C::kMmaWarp && rank == 0) {
    // ------------------------------------------------------------ even CTA: MMA issuer for the pair
    int st = 0, buf = 0;
    uint32_t ph = 0, res_ph = 0, acc_ph = 0;
    bool alive = true;
    for (int t = t_begin; t < t_end && alive; res_ph ^= 1u) {
      const Run run = run_at(args, t, t_end);
      for (int kt = run.kt0; kt < run.kt1 && alive; ++kt) {
        if (!ptx::mbar_wait(acc_empty(buf), acc_ph ^ 1u, ctl, kSiteScoreAcc)) {
          alive = false;
          break;
        }
        ptx::tc_fence_after_sync();
        for (int operand = 0; operand < 2 && alive; ++operand) {
          const uint32_t d_tmem = tmem_base + buf * 256 + operand * 128;
          for (int s = 0; s < args.slabs; s += 2) {
            const int n_slabs = min(2, args.slabs - s);
            const int res = operand * 2 + (s >> 1);
            if ((kt == run.kt0 && !ptx::mbar_wait(res_full(res), res_ph, ctl, kSiteScoreFull)) ||
                !ptx::mbar_wait(kv_full(st), ph, ctl, kSiteScoreFull)) {
              alive = false;
              break;
            }
            ptx::tc_fence_after_sync();
            for (int i = 0; i < n_slabs; ++i) {
#pragma unroll
              for (int ks = 0; ks < 4; ++ks) {
                const uint64_t da = ptx::umma_smem_desc(smem_base + (operand * 4 + s + i) * kBoxBytes + ks * 32, 16, 1024);
                const uint64_t db = ptx::umma_smem_desc(smem_base + C::kOffRing + (2 * st + i) * kHalfBox + ks * 32, 16, 1024);
                ptx::umma_ss_pair_elect<ptx::kKindF16>(d_tmem, da, db, args.idesc, (s | i | ks) != 0 ? 1u : 0u);
              }
            }
            ptx::umma_commit_pair_elect(kv_empty(st));
            if (kt == run.kt1 - 1) ptx::umma_commit_pair_elect(res_empty(res));
            if (++st == C::kRing) {
              st = 0;
              ph ^= 1u;
            }
          }
        }
        if (!alive) break;
        ptx::umma_commit_pair_elect(acc_full(buf));
        buf ^= 1;
        if (buf == 0) acc_ph ^= 1u;
      }
      t += run.kt1 - run.kt0;
    }
  } else if (warp < 8) {
    // ------------------------------------------------------------ P and dS: one query row per thread, 64 keys per warpgroup
    const int quarter = warp & 3;
    const int half = warp >> 2;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t box = smem_base + C::kOffStage + warp * 4096;
    int buf = 0;
    uint32_t acc_ph = 0;
    bool alive = true;
    for (int t = t_begin; t < t_end && alive;) {
      const Run run = run_at(args, t, t_end);
      const int bn = args.bn0 + run.head;
      const int2 plane = make_int2(args.fold.column(run.qb),
                                   args.fold.band(run.qb) * kRowBlock + static_cast<int>(rank) * 128 + quarter * 32);
      const int warp_row = run.qb * kRowBlock + static_cast<int>(rank) * 128 + quarter * 32;
      const int f = warp_row + lane;
      const bool row_ok = f < args.F;
      const float neg_lse2 = row_ok ? args.neg_lse2[static_cast<int64_t>(bn) * args.f_pad + f] : -INFINITY;
      const float delta = row_ok ? args.delta[static_cast<int64_t>(bn) * args.f_pad + f] : 0.0f;
      const uint64_t scale2 = ptx::f32x2(args.scale_log2, args.scale_log2);
      const uint64_t nl2 = ptx::f32x2(neg_lse2, neg_lse2);
      const uint64_t delta2 = ptx::f32x2(delta, delta);
      [[maybe_unused]] const uint16_t* bias_row = nullptr;
      if constexpr (kBias) {
        const int n = bn % args.N, b = bn / args.N;
        if (row_ok) bias_row = args.bias + b * args.bias_strides[0] + n * args.bias_strides[1] + f * args.bias_strides[2];
      }
      for (int kt = run.kt0; kt < run.kt1; ++kt) {
        const int key0 = kt * kKeyTile + half * 64;
        if (!ptx::mbar_wait(acc_full(buf), acc_ph, ctl, kSiteScoreOut)) {
          alive = false;
          break;
        }
        ptx::tc_fence_after_sync();
        const uint32_t acc = tmem_base + lane_addr + buf * 256 + half * 64;
        uint32_t s[2][32], dp[2][32];
        ptx::tmem_ld_32x32(acc, s[0]);
        ptx::tmem_ld_32x32(acc + 32, s[1]);
        ptx::tmem_ld_wait();
        ptx::tmem_ld_32x32(acc + 128, dp[0]);        // arrives while the exponentials run
        // P: 0 for keys past the end and for keys the mask hides from this query
        uint64_t p2[2][16];
        auto make_p = [&](auto masked_tag) {
          constexpr bool kMasked = decltype(masked_tag)::value;
          const int limit = min(args.T - key0, args.causal ? f - key0 + 1 : kKeyTile);   // first masked column
#pragma unroll
          for (int c = 0; c < 2; ++c) {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const uint64_t x = ptx::fma2(ptx::f32x2(__uint_as_float(s[c][2 * j]), __uint_as_float(s[c][2 * j + 1])), scale2, nl2);
              float x0, x1;
              ptx::f32x2_split(x, x0, x1);
              const int col = 32 * c + 2 * j;
              if constexpr (kBias) {
                if (bias_row != nullptr) {
                  uint32_t w = 0;
                  if (!kMasked && args.bias_vec) {
                    w = __ldg(reinterpret_cast<const uint32_t*>(bias_row + key0 + col));
                  } else {
                    if (key0 + col < args.T) w = __ldg(bias_row + key0 + col);
                    if (key0 + col + 1 < args.T) w |= static_cast<uint32_t>(__ldg(bias_row + key0 + col + 1)) << 16;
                  }
                  x0 = fmaf(bits_to_f32(static_cast<uint16_t>(w & 0xffffu), kBf16), kLog2e, x0);
                  x1 = fmaf(bits_to_f32(static_cast<uint16_t>(w >> 16), kBf16), kLog2e, x1);
                }
              }
              float e0 = ptx::ex2_approx(x0), e1 = ptx::ex2_approx(x1);
              if constexpr (kMasked) {
                if (col >= limit) e0 = 0.0f;
                if (col + 1 >= limit) e1 = 0.0f;
              }
              p2[c][j] = ptx::f32x2(e0, e1);
            }
          }
        };
        const bool stored = args.fold.on || (warp_row < args.F && key0 < args.T);   // (warp-uniform) the box meets the plane
        const bool masked = key0 + 64 > args.T || (args.causal && key0 + 63 > warp_row);
        if (masked) make_p(std::true_type{}); else make_p(std::false_type{});
        // the box holds the previous tile's dS until its store has read it
        if (lane == 0) ptx::bulk_wait_group_read<0>();
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t w[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            float a0, a1;
            ptx::f32x2_split(p2[c][j], a0, a1);
            w[j] = pack_pair<kBf16>(a0, a1);
          }
          stage_half_row(box, lane, c, w);
        }
        ptx::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          if (stored) ptx::tma_store_3d(&tmap_p, box, key0 + plane.x, plane.y, run.head);
          ptx::bulk_commit_group();
        }
        ptx::tmem_ld_32x32(acc + 128 + 32, dp[1]);
        ptx::tmem_ld_wait();
        // S and dP are in registers: the tile after next may overwrite them
        ptx::tc_fence_before_sync();
        if (rank == 0) ptx::mbar_arrive(acc_empty(buf)); else ptx::mbar_arrive_cluster_tmem(acc_empty(buf), 0);
        buf ^= 1;
        if (buf == 0) acc_ph ^= 1u;
        uint32_t w[2][16];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const uint64_t d = ptx::mul2(p2[c][j], ptx::sub2(ptx::f32x2(__uint_as_float(dp[c][2 * j]), __uint_as_float(dp[c][2 * j + 1])),
                                                             delta2));
            float a0, a1;
            ptx::f32x2_split(d, a0, a1);
            w[c][j] = pack_pair<kBf16>(a0, a1);
          }
        }
        if (lane == 0) ptx::bulk_wait_group_read<0>();   // P has left the box
        __syncwarp();
        stage_half_row(box, lane, 0, w[0]);
        stage_half_row(box, lane, 1, w[1]);
        ptx::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          if (stored) ptx::tma_store_3d(&tmap_ds, box, key0 + plane.x, plane.y, run.head);
          ptx::bulk_commit_group();
        }
      }
      t += run.kt1 - run.kt0;
    }
    if (lane == 0) ptx::bulk_wait_group<0>();   // the boxes outlive their stores; the planes are complete
  }

  if (*abort_flag != 0) __nanosleep(2000000);
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::cluster_sync_all();
  if (warp == C::kMmaWarp) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc_pair(tmem_base, 512);
  }
  ptx::cluster_sync_all();
}

// ---------------------------------------------------------------------------------------------
// Step 2: the three products.  Tile = 256 rows of a gradient x the whole head (256 columns), K = the
// queries (dV, dK) or keys (dQ) that meet those rows; 64-deep slabs of both operands through a 6-slot
// ring, 32 KB per CTA and slab, the accumulator double-buffered.  Tiles are ordered by the length of
// their K range, longest first, over all heads and the three products.
struct GradCfg {
  static constexpr int kStages = 6;
  static constexpr int kStageBytes = 2 * kBoxBytes;                 // A: 128 rows x 64, B: 128 head elements x 64
  static constexpr int kOffStage = kStages * kStageBytes;
  static constexpr int kOffBars = kOffStage + 4 * 2 * 4096;         // two output boxes per epilogue warp
  static constexpr int kSmemBytes = kOffBars + 256 + 1024;
  static_assert(kSmemBytes <= 232448, "shared memory budget");
  static constexpr int kThreads = 192;                              // producer, issuer, 4 epilogue warps
};

enum : int { kProductDv = 0, kProductDk = 1, kProductDq = 2 };

struct GradArgs {
  int N, F, T, H, bn0, heads;
  int nq, nk2, ranks;          // 256-row blocks of queries / keys, and the larger of the two
  int f_lim, t_lim;            // F and T rounded up to a slab
  int causal;
  Fold fold;
  int chunk;                   // heads whose tiles are sorted together
  uint32_t idesc_t, idesc_n;   // A with its rows contiguous (dV, dK) / with K contiguous (dQ)
  float head_scale;
  int* status_word;
};

struct GradMaps {
  CUtensorMap a[3];            // dV: P, dK: dS (boxes of 64 keys x 64 query rows), dQ: dS (64 keys x 128 query rows)
  CUtensorMap b[3];            // dO, Q, K: boxes of 64 head elements x 64 rows
  CUtensorMap d[3];            // dV, dK, dQ: boxes of 64 head elements x 32 rows
};

struct GradTile {
  int product, head, block;
  int k0, slabs;               // first query / key of the K range, 64-deep slabs; slabs < 0: no such tile
};
__device__ __forceinline__ GradTile grad_tile(const GradArgs& a, int u) {
  GradTile g;
  const int chunk = u / (3 * a.chunk * a.ranks);
  const int chunk_heads = min(a.chunk, a.heads - chunk * a.chunk);
  const int per_rank = 3 * chunk_heads;
  const int in_chunk = u - chunk * (3 * a.chunk * a.ranks);
  const int rank = in_chunk / per_rank;
  const int rest = in_chunk - rank * per_rank;
  g.product = rest / chunk_heads;
  g.head = a.heads - 1 - chunk * a.chunk - (rest - g.product * chunk_heads);   // the scores written last are read first
  if (g.product == kProductDq) {
    g.block = a.nq - 1 - rank;            // the last query block meets the most keys
    g.k0 = 0;
    g.slabs = g.block < 0 ? -1 : (a.causal ? min(a.t_lim, (g.block + 1) * kRowBlock) : a.t_lim) / 64;
  } else {
    g.block = rank;                       // the first key block meets the most queries
    g.k0 = a.causal ? g.block * kRowBlock : 0;
    g.slabs = g.block >= a.nk2 ? -1 : max(0, a.f_lim - g.k0) / 64;
  }
  return g;
}

template <bool kBf16>
__global__ void __launch_bounds__(GradCfg::kThreads, 1)
wide_grads_kernel(const __grid_constant__ GradMaps maps, const __grid_constant__ GradArgs args) {
  using C = GradCfg;
  constexpr int kStages = C::kStages;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - ptx::smem_u32(smem_raw));
  const uint32_t bars = smem_base + C::kOffBars;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (kStages + s); };
  auto acc_full = [&](int b) { return bars + 8u * (2 * kStages + b); };
  auto acc_empty = [&](int b) { return bars + 8u * (2 * kStages + 2 + b); };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + C::kOffBars + 8 * (2 * kStages + 4));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + C::kOffBars + 8 * (2 * kStages + 4) + 4);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = ptx::cluster_ctarank();
  ptx::AbortCtl ctl{abort_flag, args.status_word};

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(full_bar(s), 1);
      ptx::mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(acc_full(b), 1);
      ptx::mbar_init(acc_empty(b), 2 * 128);
    }
    ptx::fence_mbar_init();
    for (int i = 0; i < 3; ++i) {
      ptx::prefetch_tmap(&maps.a[i]);
      ptx::prefetch_tmap(&maps.b[i]);
      ptx::prefetch_tmap(&maps.d[i]);
    }
  }
  __syncthreads();
  ptx::cluster_sync_all();
  if (warp == 1) {
    ptx::tmem_alloc_pair(ptx::smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
    ptx::tmem_relinquish_pair();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::cluster_sync_all();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  ptx::grid_dependency_wait();      // for the score kernel's planes
  ptx::grid_dependency_trigger();

  const int pair = blockIdx.x >> 1;
  const int pairs = gridDim.x >> 1;
  const int num_tiles = 3 * args.heads * args.ranks;
  // tiles are dealt to the pairs in rounds of alternating direction
  auto tile_index = [&](int round) { return round * pairs + ((round & 1) ? pairs - 1 - pair : pair); };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    int st = 0;
    uint32_t ph = 0;
    bool alive = true;
    for (int r = 0; alive; ++r) {
      const int u = tile_index(r);
      if (u >= num_tiles) break;
      const GradTile g = grad_tile(args, u);
      const int bn = args.bn0 + g.head;
      const int n = bn % args.N, b = bn / args.N;
      const int m0 = g.block * kRowBlock + static_cast<int>(rank) * 128;
      const CUtensorMap* ma = &maps.a[g.product];
      const CUtensorMap* mb = &maps.b[g.product];
      for (int s = 0; s < g.slabs; ++s) {
        if (!ptx::mbar_wait(empty_bar(st), ph ^ 1u, ctl, kSiteGradEmpty)) {
          alive = false;
          break;
        }
        const uint32_t a_dst = smem_base + st * C::kStageBytes;
        const uint32_t b_dst = a_dst + kBoxBytes;
        const uint32_t bar = ptx::map_to_cta(full_bar(st), 0);
        const int k = g.k0 + s * 64;
        if (ptx::elect_one()) {
          if (rank == 0) ptx::mbar_expect_tx(full_bar(st), 2 * C::kStageBytes);
          const int qb = g.product == kProductDq ? g.block : k / kRowBlock;
          const int x0 = args.fold.column(qb);
          const int y0 = args.fold.band(qb) * kRowBlock;
          if (g.product == kProductDq) {
            ptx::tma_load_3d_pair(a_dst, ma, bar, x0 + k, y0 + static_cast<int>(rank) * 128, g.head);
          } else {
            const int y = y0 + k % kRowBlock;
            ptx::tma_load_3d_pair(a_dst, ma, bar, x0 + m0, y, g.head);
            ptx::tma_load_3d_pair(a_dst + kHalfBox, ma, bar, x0 + m0 + 64, y, g.head);
          }
          ptx::tma_load_4d_pair(b_dst, mb, bar, static_cast<int>(rank) * 128, k, n, b);
          ptx::tma_load_4d_pair(b_dst + kHalfBox, mb, bar, static_cast<int>(rank) * 128 + 64, k, n, b);
        }
        __syncwarp();
        if (++st == kStages) {
          st = 0;
          ph ^= 1u;
        }
      }
    }
  } else if (warp == 1 && rank == 0) {
    // ------------------------------------------------------------ even CTA: MMA issuer for the pair
    int st = 0, buf = 0;
    uint32_t ph = 0, acc_ph = 0;
    bool alive = true;
    for (int r = 0; alive; ++r) {
      const int u = tile_index(r);
      if (u >= num_tiles) break;
      const GradTile g = grad_tile(args, u);
      if (g.slabs <= 0) continue;
      if (!ptx::mbar_wait(acc_empty(buf), acc_ph ^ 1u, ctl, kSiteGradAcc)) break;
      ptx::tc_fence_after_sync();
      const uint32_t d_tmem = tmem_base + buf * 256;
      const bool k_major = g.product == kProductDq;
      const uint32_t idesc = k_major ? args.idesc_n : args.idesc_t;
      const uint32_t a_lbo = k_major ? 16 : kHalfBox;
      const uint32_t a_step = k_major ? 32 : 16 * kSlabBytes;
      for (int s = 0; s < g.slabs; ++s) {
        if (!ptx::mbar_wait(full_bar(st), ph, ctl, kSiteGradFull)) {
          alive = false;
          break;
        }
        ptx::tc_fence_after_sync();
        const uint32_t a_src = smem_base + st * C::kStageBytes;
        const uint32_t b_src = a_src + kBoxBytes;
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          const uint64_t da = ptx::umma_smem_desc(a_src + ks * a_step, a_lbo, 1024);
          const uint64_t db = ptx::umma_smem_desc(b_src + ks * (16 * kSlabBytes), kHalfBox, 1024);
          ptx::umma_ss_pair_elect<ptx::kKindF16>(d_tmem, da, db, idesc, (s | ks) != 0 ? 1u : 0u);
        }
        ptx::umma_commit_pair_elect(empty_bar(st));
        if (++st == kStages) {
          st = 0;
          ph ^= 1u;
        }
      }
      if (!alive) break;
      ptx::umma_commit_pair_elect(acc_full(buf));
      buf ^= 1;
      if (buf == 0) acc_ph ^= 1u;
    }
  } else if (warp >= 2) {
    // ------------------------------------------------------------ epilogue: one rounding, TMA stores
    const int quarter = warp & 3;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t boxes = smem_base + C::kOffStage + quarter * 8192;
    int buf = 0;
    uint32_t acc_ph = 0, n_store = 0;
    for (int r = 0;; ++r) {
      const int u = tile_index(r);
      if (u >= num_tiles) break;
      const GradTile g = grad_tile(args, u);
      if (g.slabs < 0) continue;
      const int bn = args.bn0 + g.head;
      const int n = bn % args.N, b = bn / args.N;
      const int row = g.block * kRowBlock + static_cast<int>(rank) * 128 + quarter * 32;
      const int rows = g.product == kProductDq ? args.F : args.T;
      const float mul = g.product == kProductDv ? 1.0f : args.head_scale;
      if (g.slabs > 0) {
        if (!ptx::mbar_wait(acc_full(buf), acc_ph, ctl, kSiteGradOut)) break;
        ptx::tc_fence_after_sync();
      }
      const uint32_t acc = tmem_base + lane_addr + buf * 256;
      if (row < rows) {      // (warp-uniform)
#pragma unroll 1
        for (int c0 = 0; c0 < args.H; c0 += 64) {
          const uint32_t box = boxes + (n_store & 1) * 4096;
          if (lane == 0) ptx::bulk_wait_group_read<1>();
          __syncwarp();
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t v[32], w[16];
            if (g.slabs > 0) {
              ptx::tmem_ld_32x32(acc + c0 + 32 * c, v);
              ptx::tmem_ld_wait();
            } else {         // keys that no query sees
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = 0u;
            }
#pragma unroll
            for (int i = 0; i < 16; ++i)
              w[i] = pack_pair<kBf16>(__uint_as_float(v[2 * i]) * mul, __uint_as_float(v[2 * i + 1]) * mul);
            stage_half_row(box, lane, c, w);
          }
          ptx::fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            ptx::tma_store_4d(&maps.d[g.product], box, c0, row, n, b);
            ptx::bulk_commit_group();
          }
          ++n_store;
        }
      }
      if (g.slabs > 0) {
        ptx::tc_fence_before_sync();
        if (rank == 0) ptx::mbar_arrive(acc_empty(buf)); else ptx::mbar_arrive_cluster_tmem(acc_empty(buf), 0);
        buf ^= 1;
        if (buf == 0) acc_ph ^= 1u;
      }
    }
    if (lane == 0) ptx::bulk_wait_group<0>();
  }

  if (*abort_flag != 0) __nanosleep(2000000);
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::cluster_sync_all();
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc_pair(tmem_base, 512);
  }
  ptx::cluster_sync_all();
}

// ------------------------------------------------------------------------------------- host side

int64_t plane_pitch(int T) { return (static_cast<int64_t>(T) + 7) / 8 * 8; }   // keys of a plane's row: 16-byte rows

// Heads of one batch that are taken together, and the scratch that the entry point asks for: 6 bytes per
// query-key pair of a group, of which the planes of P and dS use 4.
int heads_per_group(const Problem& p) {
  const size_t per_head = static_cast<size_t>(p.F) * plane_pitch(p.T) * 6;
  if (per_head == 0) return 1;
  return static_cast<int>(std::min<size_t>(std::max<size_t>(kGroupBudget / per_head, 1), static_cast<size_t>(std::max(p.N, 1))));
}

size_t scratch_bytes(const Problem& p) {
  const size_t scores = static_cast<size_t>(heads_per_group(p)) * p.F * plane_pitch(p.T);
  return (scores * 4 + 255) / 256 * 256 + (scores * 2 + 255) / 256 * 256;
}

struct Plan {
  int group;          // heads of a group
  int chunk;          // heads whose gradient tiles are sorted together
  Fold fold;
  int64_t rows, keys; // extents of a plane: stores are clipped there, loads read zeros beyond
};
// Groups are as large as the scratch holds, over batches as well as heads, and their planes are folded where
// that makes them smaller: every group costs about 18 us beside its work (ramp-up and the last round of both
// kernels), more than planes that fit L2 would save (B4 N16 S2048 H256 causal, unfolded planes of 128 MB a
// group: 691 us forward + backward, of 64 MB: 780, of 32 MB: 1116 and more).
Plan make_plan(const Problem& p) {
  Plan plan{};
  const int nq = (p.F + kRowBlock - 1) / kRowBlock;
  plan.fold = Fold{0, nq};
  plan.rows = p.F;
  plan.keys = plane_pitch(p.T);
  const int64_t folded_rows = static_cast<int64_t>(kRowBlock) * ((nq + 1) / 2), folded_keys = static_cast<int64_t>(kRowBlock) * (nq + 1);
  if (p.causal && folded_rows * folded_keys < plan.rows * plan.keys) {
    plan.fold.on = 1;
    plan.rows = folded_rows;
    plan.keys = folded_keys;
  }
  const int64_t heads = static_cast<int64_t>(p.B) * p.N;
  const int64_t fit = std::min<int64_t>(static_cast<int64_t>(scratch_bytes(p)) / (plan.rows * plan.keys * 4), heads);
  const int64_t groups = (heads + fit - 1) / fit;
  plan.group = static_cast<int>((heads + groups - 1) / groups);       // groups of (almost) one size
  plan.chunk = std::min(plan.group, kHeadChunk);
  return plan;
}

template <typename Kernel, typename... Args>
int launch_pairs(Kernel* fn, int pairs, int threads, int smem, bool overlap, cudaStream_t stream, const Args&... kargs) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * pairs, 1, 1);
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = overlap ? 2 : 1;
  IXK_CUDA_OK(cudaLaunchKernelEx(&cfg, fn, kargs...));
  count_launch();
  return IXK_OK;
}

template <bool kBf16>
int launch_typed(const BwdProblem& bp, const DeviceInfo& dev, const float* neg_lse2, const float* delta, int f_pad,
                 void* scratch, cudaStream_t stream) {
  const Problem& p = bp.fwd;
  const CUtensorMapDataType dt = kBf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  const int all_pairs = std::max(dev.sm_count / 2, 1);
  const Plan plan = make_plan(p);
  const int group = plan.group;
  const int64_t rows = plan.rows, keys = plan.keys;
  uint16_t* plane_p = static_cast<uint16_t*>(scratch);
  uint16_t* plane_ds = plane_p + static_cast<int64_t>(group) * rows * keys;

  // [B, N, S, H] operands and results as rank-4 maps (head element, row, head, batch)
  auto tensor_map = [&](CUtensorMap* out, const void* base, const int64_t* strides, int s_rows, int box_rows) -> int {
    TmapSpec s{};
    s.dtype = dt;
    s.rank = 4;
    s.swizzle128 = true;
    s.dims[0] = p.H;
    s.dims[1] = s_rows;
    s.dims[2] = p.N;
    s.dims[3] = p.B;
    auto stride_bytes = [](int64_t st, uint64_t fallback) -> uint64_t {
      return st > 0 ? static_cast<uint64_t>(st) * 2 : fallback;   // size-1 dimensions still need a legal stride
    };
    const uint64_t pitch = stride_bytes(strides[2], static_cast<uint64_t>(p.H) * 2);
    s.strides_bytes[0] = pitch;
    s.strides_bytes[1] = stride_bytes(strides[1], pitch * s_rows);
    s.strides_bytes[2] = stride_bytes(strides[0], pitch * s_rows * p.N);
    s.box[0] = 64;
    s.box[1] = box_rows;
    s.box[2] = s.box[3] = 1;
    return encode_tmap(out, base, s);
  };
  // a score plane [heads of the group, rows, keys]
  auto plane_map = [&](CUtensorMap* out, const void* base, int box_rows) -> int {
    TmapSpec s{};
    s.dtype = dt;
    s.rank = 3;
    s.swizzle128 = true;
    s.dims[0] = keys;
    s.dims[1] = rows;
    s.dims[2] = group;
    s.strides_bytes[0] = static_cast<uint64_t>(keys) * 2;
    s.strides_bytes[1] = static_cast<uint64_t>(keys) * rows * 2;
    s.box[0] = 64;
    s.box[1] = box_rows;
    s.box[2] = 1;
    return encode_tmap(out, base, s);
  };
  CUtensorMap tq, tdo, tk, tv, tp, tds;
  GradMaps gm;
  int rc;
  if ((rc = tensor_map(&tq, p.q, p.q_strides, p.F, 128)) != IXK_OK) return rc;
  if ((rc = tensor_map(&tdo, bp.grad_out, bp.do_strides, p.F, 128)) != IXK_OK) return rc;
  if ((rc = tensor_map(&tk, p.k, p.k_strides, p.T, 64)) != IXK_OK) return rc;
  if ((rc = tensor_map(&tv, p.v, p.v_strides, p.T, 64)) != IXK_OK) return rc;
  if ((rc = plane_map(&tp, plane_p, 32)) != IXK_OK) return rc;
  if ((rc = plane_map(&tds, plane_ds, 32)) != IXK_OK) return rc;
  if ((rc = plane_map(&gm.a[kProductDv], plane_p, 64)) != IXK_OK) return rc;
  if ((rc = plane_map(&gm.a[kProductDk], plane_ds, 64)) != IXK_OK) return rc;
  if ((rc = plane_map(&gm.a[kProductDq], plane_ds, 128)) != IXK_OK) return rc;
  if ((rc = tensor_map(&gm.b[kProductDv], bp.grad_out, bp.do_strides, p.F, 64)) != IXK_OK) return rc;
  if ((rc = tensor_map(&gm.b[kProductDk], p.q, p.q_strides, p.F, 64)) != IXK_OK) return rc;
  gm.b[kProductDq] = tk;
  if ((rc = tensor_map(&gm.d[kProductDv], bp.dv, bp.dv_strides, p.T, 32)) != IXK_OK) return rc;
  if ((rc = tensor_map(&gm.d[kProductDk], bp.dk, bp.dk_strides, p.T, 32)) != IXK_OK) return rc;
  if ((rc = tensor_map(&gm.d[kProductDq], bp.dq, bp.dq_strides, p.F, 32)) != IXK_OK) return rc;

  const uint32_t fmt = kBf16 ? 1u : 0u;
  ScoreArgs sa{};
  sa.N = p.N; sa.F = p.F; sa.T = p.T;
  sa.f_pad = f_pad;
  sa.nq = (p.F + kRowBlock - 1) / kRowBlock;
  sa.nk = (p.T + kKeyTile - 1) / kKeyTile;
  sa.slabs = (p.H + 63) / 64;
  sa.causal = p.causal ? 1 : 0;
  sa.fold = plan.fold;
  sa.tiles_per_head = 0;
  for (int qb = 0; qb < sa.nq; ++qb) sa.tiles_per_head += p.causal ? std::min(sa.nk, 2 * qb + 2) : sa.nk;
  sa.idesc = ptx::umma_idesc(fmt, fmt, 0, 0, 2 * 128, kKeyTile);
  sa.scale_log2 = p.head_scale * kLog2e;
  sa.neg_lse2 = neg_lse2;
  sa.delta = delta;
  sa.bias = static_cast<const uint16_t*>(p.bias);
  sa.bias_vec = p.bias != nullptr && (reinterpret_cast<uintptr_t>(p.bias) & 3u) == 0;
  for (int i = 0; i < 3; ++i) {
    sa.bias_strides[i] = p.bias_strides[i];
    sa.bias_vec = sa.bias_vec && p.bias_strides[i] % 2 == 0;
  }
  sa.status_word = dev.status_word;

  GradArgs ga{};
  ga.N = p.N; ga.F = p.F; ga.T = p.T; ga.H = p.H;
  ga.nq = sa.nq;
  ga.nk2 = (p.T + kRowBlock - 1) / kRowBlock;
  ga.ranks = std::max(ga.nq, ga.nk2);
  ga.f_lim = (p.F + 63) / 64 * 64;
  ga.t_lim = (p.T + 63) / 64 * 64;
  ga.causal = sa.causal;
  ga.fold = plan.fold;
  ga.chunk = plan.chunk;
  ga.idesc_t = ptx::umma_idesc(fmt, fmt, 1, 1, 2 * 128, 256);
  ga.idesc_n = ptx::umma_idesc(fmt, fmt, 0, 1, 2 * 128, 256);
  ga.head_scale = p.head_scale;
  ga.status_word = dev.status_word;

  auto* scores = p.bias != nullptr ? &wide_scores_kernel<kBf16, true> : &wide_scores_kernel<kBf16, false>;
  auto* grads = &wide_grads_kernel<kBf16>;
  static thread_local int configured_device = -1;
  if (configured_device != dev.device) {
    for (auto* fn : {&wide_scores_kernel<kBf16, true>, &wide_scores_kernel<kBf16, false>})
      IXK_CUDA_OK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, ScoreCfg::kSmemBytes));
    IXK_CUDA_OK(cudaFuncSetAttribute(grads, cudaFuncAttributeMaxDynamicSharedMemorySize, GradCfg::kSmemBytes));
    configured_device = dev.device;
  }
  bool first = true;
  const int heads_all = p.B * p.N;
  for (int bn0 = 0; bn0 < heads_all;) {
    const int g = std::min(group, heads_all - bn0);
    sa.bn0 = ga.bn0 = bn0;
    sa.heads = ga.heads = g;
    bn0 += g;
    const int64_t total = static_cast<int64_t>(sa.tiles_per_head) * g;
    const int64_t grad_tiles = static_cast<int64_t>(3) * g * ga.ranks;
    if (total > 0x7fffffff || grad_tiles > 0x7fffffff) return fail(IXK_UNIMPLEMENTED, "too many score tiles");
    sa.total_tiles = static_cast<int>(total);
    if ((rc = launch_pairs(scores, static_cast<int>(std::min<int64_t>(total, all_pairs)), ScoreCfg::kThreads, ScoreCfg::kSmemBytes, !first,
                           stream, tq, tdo, tk, tv, tp, tds, sa)) != IXK_OK)
      return rc;
    first = false;
    if ((rc = launch_pairs(grads, static_cast<int>(std::min<int64_t>(grad_tiles, all_pairs)), GradCfg::kThreads, GradCfg::kSmemBytes, true,
                           stream, gm, ga)) != IXK_OK)
      return rc;
  }
  return IXK_OK;
}

}  // namespace

size_t bwd_wide_scratch_bytes(const Problem& p) {
  return scratch_bytes(p);
}

// Per group of heads: one launch of the score kernel over all SM pairs, then one of the gradient kernel
// (programmatic dependent launches: each sets itself up while its predecessor runs and waits for its end
// before it touches the planes).
int launch_bwd_wide(const BwdProblem& bp, const DeviceInfo& dev, const float* neg_lse2, const float* delta, int f_pad,
                    void* scratch, cudaStream_t stream) {
  return bp.fwd.dtype == IXK_BF16 ? launch_typed<true>(bp, dev, neg_lse2, delta, f_pad, scratch, stream)
                                  : launch_typed<false>(bp, dev, neg_lse2, delta, f_pad, scratch, stream);
}

}  // namespace fmha
}  // namespace ixk
