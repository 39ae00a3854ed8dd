// Attention for 2..16 query rows against a long key/value cache, all rows in one pass over the cache.
//
// The step is a stream of K and V from HBM; what the split-key kernel of fmha_decode_sm100.cu does per
// row on the FMA pipe (a dot product, its shuffles, an accumulator) bounds it by instruction issue from
// two rows on, so there the cache is streamed ceil(F / 2) times.  Here the rows are the N side of small
// tensor-core products whose M side is the cache:
//   S^T [keys, rows] = K . Q^T         A = K as it lies in memory, B = Q (registers)
//   O^T [head, rows] += V^T . P^T      A = V^T (transposing fragment loads), B = P
// (mma.sync and not tcgen05: with 8 rows the product is 3 % of what the tensor core could do in the time;
// what counts is that nothing has to travel through tensor memory between the two products.)
//
//   CTAs      persistent, at most one per SM; the (batch, head) units are cut into tiles of keys, the tiles
//             numbered through, and every CTA takes whole units, a range of one unit, or an equal share of
//             all tiles (make_plan)
//   warp 8    TMA producer: K and V of a tile into one slot of a ring of up to 192 KB
//   warps 0-7 16 keys of a tile each (so that a tile goes to 2 or 4 warps and the ring's slots are
//             worked on side by side), every warp with its own running maximum, sum and O^T; merged
//             through shared memory where a unit ends
// A unit that a range boundary cuts leaves unnormalised partials (O, maximum, sum) in scratch, which
// fmha_decode_mma_combine_kernel merges.
//
// Precision is that of the fp32 arithmetic it replaces.  P goes into the second product as the sum of two
// tf32 numbers (hi + lo, 22 bits of P at fp32's range of exponents; a pair of fp16 numbers would lose P
// below 2^-25 of the row's largest), V as tf32, which holds both 16-bit types exactly.  The tensor core
// truncates what it accumulates, so every product starts at zero and is added to S and O in fp32.
// Measured against 64 bits, B2 N16 T2000, heads of 64 to 256, 4 and 16 rows: relative error of O equal to the
// split-key kernel's to six digits (1.6617e-3 bf16, 2.0851e-4 fp16 at head size 256), of one key far above
// 2000 others up to 2^36 times smaller 1.9e-4 (fp16); lse 3.6e-7 to 4.2e-7 there, 3.3e-7 to 3.7e-7 here.
// B32 N16 T3001 H256 bf16: F = 2 411 -> 265 us, 4 765 -> 267 (5.9 TB/s), 8 1410 -> 269, 12 2106 -> 345, 16 2771 -> 377.
// Short caches are bound by what surrounds the stream.  Started under the kernel before it, barriers set by a thread each,
// the warps' O merged without bank conflicts (read row by row they met 8 or 16 to a bank) and by all threads, the merge
// kernel a CTA per cut unit with its loads together, in place of one per range that read part after part (calls back to
// back, bf16, us): B1 N16 F16 T2127 H64 21.0 -> 10.6, B2 N16 F8 T1126 H128 14.7 -> 9.4, B1 N8 F2 T4000 H128 14.4 -> 9.6,
// B11 N16 F8 T64 H256 14.4 -> 11.3, B20 N16 F16 T130 H256 47 -> 39, B64 N8 F2 T700 H128 39 -> 35, and F = 4 above 251 -> 246.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "fmha_sm100.h"
#include "ptx.cuh"

namespace ixk {
namespace fmha {

namespace {

constexpr int kWarps = 8;                         // compute warps: two warpgroups
constexpr int kThreads = (kWarps + 4) * 32;       // and one of which a single warp works, on the loads
// Registers per thread.  At launch 168 (65536 / 384, a multiple of 8); the third warpgroup gives its share up:
// 256 x 240 + 128 x 24 = 384 x 168.  (With 168 for all, the kernels for two blocks of rows spill up to 250 bytes.)
constexpr int kComputeRegs = 240;
constexpr int kLoadRegs = 24;
constexpr size_t kMaxPartialBytes = IXK_STATIC_SCRATCH_BYTES;  // also the scratch of ixk_fmha_fwd_static_scratch
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

// wait sites reported in the device status word
enum : int { kSiteEmpty = 0x61, kSiteFull = 0x62 };

constexpr int gcd(int a, int b) { return b == 0 ? a : gcd(b, a % b); }
constexpr int lcm(int a, int b) { return a / gcd(a, b) * b; }

template <int kSlabs, int kNT>
struct Cfg {
  static constexpr int kKeys = kSlabs > 2 ? 32 : 64;             // keys of a tile
  static constexpr int kBoxBytes = kKeys * 128;                  // 64 head elements of them
  static constexpr int kTileBytes = kSlabs * kBoxBytes;          // K or V
  static constexpr int kStageBytes = 2 * kTileBytes;
  static constexpr int kRows = kNT * 8;
  static constexpr int kHPad = kSlabs * 64;
  static constexpr int kMergeBytes = kWarps / 2 * kRows * kHPad * 4;
  static constexpr int kTailBytes = 2048;                        // barriers, maxima and sums
  // Q as B fragments takes kSlabs * kNT * 8 registers; beside the O^T of two blocks of rows and three or
  // four slabs it would spill, and is read from shared memory for every 16 keys instead
  static constexpr bool kQShared = kNT == 2 && kSlabs >= 3;
  static constexpr int kQBytes = kQShared ? kRows * kHPad * 2 : 0;
  static constexpr int kFit = (232448 - 1024 - kMergeBytes - kTailBytes - kQBytes) / kStageBytes;
  static constexpr int kStages = kFit < 16 ? kFit : 16;
  static constexpr int kWarpsPerTile = kKeys / 16;
  static constexpr int kGroups = kWarps / kWarpsPerTile;         // tiles worked on side by side
  // A tile's barriers: the tile's number modulo this, so that each is used by one slot and one group of
  // warps only.  (Barriers per slot would not do: a group comes back to a slot after other groups' turns,
  // and a wait by parity cannot tell their phases from its own.)
  static constexpr int kBars = lcm(kStages, kGroups);
  static constexpr int kSmemBytes = kStages * kStageBytes + kMergeBytes + kQBytes + kTailBytes + 1024;
  static_assert(kSmemBytes <= 232448, "shared memory budget");
  static_assert(kStages >= kGroups, "every group of warps needs a slot of its own");
  static_assert(2 * kWarps * kRows * 4 + 16 * kBars + 8 <= kTailBytes, "tail");
};

struct Args {
  int B, N, H, F, T;
  float scale_log2;
  int tiles_per_unit, pieces, piece, slots;
  const uint16_t* q;
  const uint16_t* bias;
  uint16_t* out;
  float* lse;
  float* partial;   // [grid][slots][F][H + 2]: with two, the unit a CTA's range starts inside of and the one it starts
  int k_head_mul, k_batch_mul, v_head_mul, v_batch_mul;   // 0: one K / V for all heads / batches
  int64_t q_strides[3], o_strides[3], bias_strides[3];
  int* status_word;
};

// First tile of a CTA's range: equal shares of `pieces` pieces of `piece` tiles (one tile, or a whole unit).
__host__ __device__ __forceinline__ int range_begin(int pieces, int piece, int cta, int ctas) {
  return static_cast<int>(static_cast<int64_t>(pieces) * cta / ctas) * piece;
}

template <bool kBf16>
__device__ __forceinline__ float to_f32(uint16_t h) {
  return kBf16 ? __uint_as_float(static_cast<uint32_t>(h) << 16) : __half2float(__ushort_as_half(h));
}
template <bool kBf16>
__device__ __forceinline__ uint16_t from_f32(float x) {
  return kBf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(x)) : __half_as_ushort(__float2half_rn(x));
}

// p >= 0 as the sum of two tf32 numbers.  hi is the largest of 11 bits strictly below p (0 for p = 0), so that
// lo > 0 wherever p > 0: with lo = 0 an infinite V would turn p * inf into inf + 0 * inf = NaN.
__device__ __forceinline__ void split_tf32(float p, uint32_t& hi, uint32_t& lo) {
  const uint32_t bits = __float_as_uint(p);
  hi = (p > 0.0f ? bits - 1u : bits) & 0xffffe000u;   // (NaN stays NaN)
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(p - __uint_as_float(hi)));
}
// The two 16-bit numbers of a register as tf32 (exact: tf32 has fp16's mantissa and bf16's exponents).
template <bool kBf16>
__device__ __forceinline__ void widen(uint32_t w, uint32_t& first, uint32_t& second) {
  if constexpr (kBf16) {
    first = w << 16;
    second = w & 0xffff0000u;
  } else {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
    first = __float_as_uint(f.x);
    second = __float_as_uint(f.y);
  }
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ uint32_t transpose_8x8(uint32_t x) {
  uint32_t y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}
// d = a . b
template <bool kBf16>
__device__ __forceinline__ void mma_16x8x16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (kBf16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}
// d += a . b
__device__ __forceinline__ void mma_16x8x8_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int kSlabs, int kNT, bool kBf16>
__global__ void __launch_bounds__(kThreads, 1)
fmha_decode_mma_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                       const __grid_constant__ Args a) {
  using C = Cfg<kSlabs, kNT>;
  constexpr int kSteps = kSlabs * 4;              // 16 head elements each
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - ptx::smem_u32(smem_raw));
  float* merge = reinterpret_cast<float*>(smem_gen + C::kStages * C::kStageBytes);   // [4][head][rows]
  uint8_t* q_rows = smem_gen + C::kStages * C::kStageBytes + C::kMergeBytes;            // [rows][head], 16-byte pieces swizzled
  uint8_t* tail = q_rows + C::kQBytes;
  float* sm_m = reinterpret_cast<float*>(tail);                  // [8 warps][rows]
  float* sm_l = sm_m + kWarps * C::kRows;
  // barriers (8 bytes each)
  const uint32_t bars = smem_base + C::kStages * C::kStageBytes + C::kMergeBytes + C::kQBytes + 2 * kWarps * C::kRows * 4;
  auto full = [&](int i) { return bars + 8u * i; };
  auto empty = [&](int i) { return bars + 8u * (C::kBars + i); };
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 2 * kWarps * C::kRows * 4 + 16 * C::kBars);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  ptx::AbortCtl ctl{abort_flag, a.status_word};
  static_assert(C::kBars < kThreads, "a thread per pair of barriers");
  if (threadIdx.x < C::kBars) {
    ptx::mbar_init(full(threadIdx.x), 1);
    ptx::mbar_init(empty(threadIdx.x), C::kWarpsPerTile);
    ptx::fence_mbar_init();
  }
  if (threadIdx.x == kThreads - 1) {
    *abort_flag = 0;
    ptx::prefetch_tmap(&tmap_k);
    ptx::prefetch_tmap(&tmap_v);
  }
  __syncthreads();
  ptx::grid_dependency_sync();   // (the combine kernel is set up meanwhile; it waits for this grid's end)

  const int t_begin = range_begin(a.pieces, a.piece, blockIdx.x, gridDim.x);
  const int t_end = range_begin(a.pieces, a.piece, blockIdx.x + 1, gridDim.x);

  if (warp >= kWarps) {
    // ------------------------------------------------------------ TMA producer
    ptx::setmaxnreg_dec<kLoadRegs>();
    if (warp == kWarps && lane == 0) {
      int unit = t_begin / a.tiles_per_unit;
      int in_unit = t_begin - unit * a.tiles_per_unit;
      for (int seq = 0; seq < t_end - t_begin; ++seq) {
        const int head = unit % a.N, batch = unit / a.N;
        const int before = seq - C::kStages;      // the tile that had the slot
        if (before >= 0 &&
            !ptx::mbar_wait(empty(before % C::kBars), static_cast<uint32_t>(before / C::kBars) & 1u, ctl, kSiteEmpty))
          break;
        const uint32_t bar = full(seq % C::kBars);
        ptx::mbar_expect_tx(bar, C::kStageBytes);
        const uint32_t dst = smem_base + seq % C::kStages * C::kStageBytes;
#pragma unroll
        for (int s = 0; s < kSlabs; ++s)
          ptx::tma_load_4d(dst + s * C::kBoxBytes, &tmap_k, bar, s * 64, in_unit * C::kKeys, head * a.k_head_mul,
                           batch * a.k_batch_mul);
#pragma unroll
        for (int s = 0; s < kSlabs; ++s)
          ptx::tma_load_4d(dst + C::kTileBytes + s * C::kBoxBytes, &tmap_v, bar, s * 64, in_unit * C::kKeys,
                           head * a.v_head_mul, batch * a.v_batch_mul);
        if (++in_unit == a.tiles_per_unit) {
          in_unit = 0;
          ++unit;
        }
      }
    }
  } else {
    ptx::setmaxnreg_inc<kComputeRegs>();
    const int g = lane >> 2, c = lane & 3;        // fragment row / column-pair index
    const int group = warp / C::kWarpsPerTile;
    const int key_row = (warp % C::kWarpsPerTile) * 16;
    // ldmatrix row addresses of this lane (row of the box, 16-byte column before the swizzle)
    const int k_row = key_row + (lane & 7) + ((lane >> 3) & 1) * 8;
    const int k_col = lane >> 4;
    const int v_row = key_row + (lane & 7) + (lane >> 4) * 8;
    const int v_col = (lane >> 3) & 1;
    bool alive = true;

    for (int t = t_begin; t < t_end;) {
      // ---- one unit's part of the range (the loop is the same for all eight warps, barriers included)
      const int unit = t / a.tiles_per_unit;
      const int head = unit % a.N, batch = unit / a.N;
      const int unit_t0 = unit * a.tiles_per_unit;
      const int seg_end = min(t_end, unit_t0 + a.tiles_per_unit);

      const uint16_t* q_base = a.q + batch * a.q_strides[0] + head * a.q_strides[1];
      [[maybe_unused]] uint32_t qf[C::kQShared ? 1 : kSteps][kNT][2];
      if constexpr (C::kQShared) {
        // (every warp is past the previous unit's last tile: it has gone through that unit's merge)
        for (int i = threadIdx.x; i < C::kRows * kSlabs * 8; i += kWarps * 32) {
          const int f = i / (kSlabs * 8), piece = i % (kSlabs * 8);
          uint4 w = make_uint4(0u, 0u, 0u, 0u);
          if (f < a.F && piece * 8 < a.H) w = *reinterpret_cast<const uint4*>(q_base + f * a.q_strides[2] + piece * 8);
          *reinterpret_cast<uint4*>(q_rows + f * C::kHPad * 2 + ((piece ^ (f & 7)) << 4)) = w;
        }
        ptx::named_barrier_sync(1, kWarps * 32);
      } else {
#pragma unroll
        for (int nt = 0; nt < kNT; ++nt) {
          const int f = nt * 8 + g;
          const uint16_t* qrow = q_base + f * a.q_strides[2];
#pragma unroll
          for (int ks = 0; ks < kSteps; ++ks) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int d = ks * 16 + i * 8 + 2 * c;
              qf[ks][nt][i] = (f < a.F && d < a.H) ? *reinterpret_cast<const uint32_t*>(qrow + d) : 0u;   // H is a multiple of 8
            }
          }
        }
      }
      const uint16_t* bias_row[kNT][2];
#pragma unroll
      for (int nt = 0; nt < kNT; ++nt) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int fr = nt * 8 + 2 * c + i;
          bias_row[nt][i] = (a.bias != nullptr && fr < a.F)
                                ? a.bias + batch * a.bias_strides[0] + head * a.bias_strides[1] + fr * a.bias_strides[2]
                                : nullptr;
        }
      }
      float o[kSteps][kNT][4];
      float m_run[kNT][2], l_run[kNT][2];
#pragma unroll
      for (int nt = 0; nt < kNT; ++nt) {
        m_run[nt][0] = m_run[nt][1] = -INFINITY;
        l_run[nt][0] = l_run[nt][1] = 0.0f;
#pragma unroll
        for (int mt = 0; mt < kSteps; ++mt)
#pragma unroll
          for (int i = 0; i < 4; ++i) o[mt][nt][i] = 0.0f;
      }

      // ---- this warp's tiles: every kGroups-th of the CTA's sequence
      int seq = t - t_begin;
      seq += (group - seq % C::kGroups + C::kGroups) % C::kGroups;
      for (; alive && t_begin + seq < seg_end; seq += C::kGroups) {
        const int slot = seq % C::kStages;
        const int key0 = (t_begin + seq - unit_t0) * C::kKeys + key_row;   // first of this warp's 16 keys
        float bias_v[kNT][4];
#pragma unroll
        for (int nt = 0; nt < kNT; ++nt)
#pragma unroll
          for (int i = 0; i < 4; ++i) bias_v[nt][i] = 0.0f;
        if (a.bias != nullptr) {
#pragma unroll
          for (int nt = 0; nt < kNT; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int key = key0 + g + (i >> 1) * 8;
              if (bias_row[nt][i & 1] != nullptr && key < a.T) bias_v[nt][i] = to_f32<kBf16>(bias_row[nt][i & 1][key]);
            }
        }
        const int bar = seq % C::kBars;
        if (!ptx::mbar_wait(full(bar), static_cast<uint32_t>(seq / C::kBars) & 1u, ctl, kSiteFull)) {
          alive = false;
          break;
        }
        const uint32_t k_tile = smem_base + slot * C::kStageBytes;
        const uint32_t v_tile = k_tile + C::kTileBytes;
        // S^T: the products of 16 head elements each, summed in fp32 in two chains
        float acc[2][kNT][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int nt = 0; nt < kNT; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][nt][e] = 0.0f;
#pragma unroll
        for (int ks = 0; ks < kSteps; ++ks) {
          uint32_t af[4];
          ldmatrix_x4(k_tile + (ks >> 2) * C::kBoxBytes + k_row * 128 + (((2 * (ks & 3) + k_col) ^ (k_row & 7)) << 4), af);
          float part[kNT][4];
          if constexpr (C::kQShared) {
            uint32_t qb[4];     // b0, b1 of rows 0-7, b0, b1 of rows 8-15
            const int row = (lane & 7) + (lane >> 4) * 8;
            ldmatrix_x4(ptx::smem_u32(q_rows) + row * C::kHPad * 2 + (((2 * ks + ((lane >> 3) & 1)) ^ (row & 7)) << 4), qb);
            mma_16x8x16<kBf16>(part[0], af, qb[0], qb[1]);
            mma_16x8x16<kBf16>(part[kNT - 1], af, qb[2], qb[3]);
          } else {
#pragma unroll
            for (int nt = 0; nt < kNT; ++nt) mma_16x8x16<kBf16>(part[nt], af, qf[ks][nt][0], qf[ks][nt][1]);
          }
#pragma unroll
          for (int nt = 0; nt < kNT; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[ks & 1][nt][e] += part[nt][e];
        }
        const bool edge = key0 + 16 > a.T;   // (warp-uniform)
        uint32_t p_hi[kNT][4], p_lo[kNT][4];   // row g (of a block): keys 2c, 2c + 1, 2c + 8, 2c + 9
#pragma unroll
        for (int nt = 0; nt < kNT; ++nt) {
          float x[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            x[i] = (acc[0][nt][i] + acc[1][nt][i]) * a.scale_log2;
            if (a.bias != nullptr) x[i] = fmaf(bias_v[nt][i], kLog2e, x[i]);
            if (edge && key0 + g + (i >> 1) * 8 >= a.T) x[i] = -INFINITY;
          }
          float mx[2] = {fmaxf(x[0], x[2]), fmaxf(x[1], x[3])};
#pragma unroll
          for (int off = 4; off < 32; off <<= 1) {
            mx[0] = fmaxf(mx[0], __shfl_xor_sync(0xffffffffu, mx[0], off));
            mx[1] = fmaxf(mx[1], __shfl_xor_sync(0xffffffffu, mx[1], off));
          }
          const bool raised = mx[0] > m_run[nt][0] || mx[1] > m_run[nt][1];
          if (__any_sync(0xffffffffu, raised)) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const float m_new = fmaxf(m_run[nt][i], mx[i]);
              const float corr = m_new == -INFINITY ? 1.0f : ptx::ex2_approx(m_run[nt][i] - m_new);   // 0 from -inf
              m_run[nt][i] = m_new;
              l_run[nt][i] *= corr;
#pragma unroll
              for (int mt = 0; mt < kSteps; ++mt) {
                o[mt][nt][i] *= corr;
                o[mt][nt][i + 2] *= corr;
              }
            }
          }
          float p[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float m = m_run[nt][i & 1];
            p[i] = ptx::ex2_approx(x[i] - (m == -INFINITY ? 0.0f : m));   // 0 for masked / absent keys
            l_run[nt][i & 1] += p[i];
          }
#pragma unroll
          for (int i = 0; i < 2; ++i) {   // keys g (+ 8): [key][row] blocks turned over, the halves of P each
            const uint32_t p0 = __float_as_uint(p[2 * i]), p1 = __float_as_uint(p[2 * i + 1]);
            const uint32_t upper = transpose_8x8(__byte_perm(p0, p1, 0x7632));
            const uint32_t lower = transpose_8x8(__byte_perm(p0, p1, 0x5410));
            split_tf32(__uint_as_float(__byte_perm(lower, upper, 0x5410)), p_hi[nt][2 * i], p_lo[nt][2 * i]);
            split_tf32(__uint_as_float(__byte_perm(lower, upper, 0x7632)), p_hi[nt][2 * i + 1], p_lo[nt][2 * i + 1]);
          }
        }
#pragma unroll
        for (int mt = 0; mt < kSteps; ++mt) {
          uint32_t af[4];
          ldmatrix_x4_trans(v_tile + (mt >> 2) * C::kBoxBytes + v_row * 128 + (((2 * (mt & 3) + v_col) ^ (v_row & 7)) << 4), af);
          // two products of 8 keys: 2c takes the place of key c, 2c + 1 that of c + 4, on both sides
          uint32_t a8[2][4];
          float part[kNT][4];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            widen<kBf16>(af[2 * i], a8[i][0], a8[i][2]);
            widen<kBf16>(af[2 * i + 1], a8[i][1], a8[i][3]);
          }
#pragma unroll
          for (int nt = 0; nt < kNT; ++nt) {
#pragma unroll
            for (int e = 0; e < 4; ++e) part[nt][e] = 0.0f;
#pragma unroll
            for (int i = 0; i < 2; ++i) mma_16x8x8_tf32(part[nt], a8[i], p_lo[nt][2 * i], p_lo[nt][2 * i + 1]);
#pragma unroll
            for (int i = 0; i < 2; ++i) mma_16x8x8_tf32(part[nt], a8[i], p_hi[nt][2 * i], p_hi[nt][2 * i + 1]);
#pragma unroll
            for (int e = 0; e < 4; ++e) o[mt][nt][e] += part[nt][e];
          }
        }
        ptx::fence_proxy_async_smem();   // these reads come before the slot's next TMA write
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(empty(bar));
      }

      // ---- merge the eight warps: the upper four into the lower four, then all threads over the rest
      // Element (d, row) of a warp's O in the merge buffer: rows in pairs, the pairs of a d exchanged by d, so that a warp
      // that reads one pair of 32 consecutive d meets no bank twice in 128 bytes.
      auto merge_at = [&](int w4, int d, int pair) {
        return merge + (w4 * C::kHPad + d) * C::kRows + 2 * (pair ^ (kNT == 1 ? (d >> 2) & 3 : (d >> 1) & 7));
      };
      auto put = [&](int w4) {
#pragma unroll
        for (int nt = 0; nt < kNT; ++nt) {
#pragma unroll
          for (int mt = 0; mt < kSteps; ++mt) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              *reinterpret_cast<float2*>(merge_at(w4, mt * 16 + g + i * 8, nt * 4 + c)) = make_float2(o[mt][nt][2 * i], o[mt][nt][2 * i + 1]);
            }
          }
        }
      };
#pragma unroll
      for (int nt = 0; nt < kNT; ++nt)
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int off = 4; off < 32; off <<= 1) l_run[nt][i] += __shfl_xor_sync(0xffffffffu, l_run[nt][i], off);
      auto put_stats = [&]() {
        if (g == 0) {
#pragma unroll
          for (int nt = 0; nt < kNT; ++nt)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              sm_m[warp * C::kRows + nt * 8 + 2 * c + i] = m_run[nt][i];
              sm_l[warp * C::kRows + nt * 8 + 2 * c + i] = l_run[nt][i];
            }
        }
      };
      ptx::named_barrier_sync(1, kWarps * 32);    // the previous unit's merge has been read
      if (warp >= 4) {
        put(warp - 4);
        put_stats();
      }
      ptx::named_barrier_sync(1, kWarps * 32);
      if (warp < 4) {
#pragma unroll
        for (int nt = 0; nt < kNT; ++nt) {
          float cs[2], co[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int r = nt * 8 + 2 * c + i;
            const float m_o = sm_m[(warp + 4) * C::kRows + r], l_o = sm_l[(warp + 4) * C::kRows + r];
            const float m_new = fmaxf(m_run[nt][i], m_o);
            cs[i] = m_run[nt][i] == -INFINITY ? 0.0f : ptx::ex2_approx(m_run[nt][i] - m_new);
            co[i] = m_o == -INFINITY ? 0.0f : ptx::ex2_approx(m_o - m_new);
            l_run[nt][i] = l_run[nt][i] * cs[i] + l_o * co[i];
            m_run[nt][i] = m_new;
          }
#pragma unroll
          for (int mt = 0; mt < kSteps; ++mt) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const float2 v = *reinterpret_cast<const float2*>(merge_at(warp, mt * 16 + g + i * 8, nt * 4 + c));
              o[mt][nt][2 * i] = o[mt][nt][2 * i] * cs[0] + v.x * co[0];
              o[mt][nt][2 * i + 1] = o[mt][nt][2 * i + 1] * cs[1] + v.y * co[1];
            }
          }
        }
        put(warp);       // (each warp overwrites what it alone has read)
        put_stats();
      }
      ptx::named_barrier_sync(1, kWarps * 32);
      const bool whole = t == unit_t0 && seg_end == unit_t0 + a.tiles_per_unit;
      float* part = a.partial + (static_cast<int64_t>(blockIdx.x) * a.slots + (a.slots == 2 && t == unit_t0 ? 1 : 0)) * a.F * (a.H + 2);
      // A thread takes one d of two rows at a time, neighbours the next d.
      for (int item = threadIdx.x; item < (a.F + 1) / 2 * C::kHPad; item += kWarps * 32) {
        const int pair = item / C::kHPad, d = item % C::kHPad;
        float2 v[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) v[w] = *reinterpret_cast<const float2*>(merge_at(w, d, pair));
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int f = 2 * pair + i;
          if (f >= a.F) break;
          float m_all = -INFINITY;
#pragma unroll
          for (int w = 0; w < 4; ++w) m_all = fmaxf(m_all, sm_m[w * C::kRows + f]);
          float l_all = 0.0f, o_all = 0.0f;
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            const float m_w = sm_m[w * C::kRows + f];
            const float cw = m_w == -INFINITY ? 0.0f : ptx::ex2_approx(m_w - m_all);
            l_all += sm_l[w * C::kRows + f] * cw;
            o_all += (i == 0 ? v[w].x : v[w].y) * cw;
          }
          if (d < a.H) {
            if (whole)
              a.out[batch * a.o_strides[0] + head * a.o_strides[1] + f * a.o_strides[2] + d] = from_f32<kBf16>(o_all / l_all);
            else
              part[f * (a.H + 2) + d] = o_all;
          }
          if (d == 0) {
            if (whole) {
              if (a.lse != nullptr) a.lse[static_cast<int64_t>(unit) * a.F + f] = fmaf(m_all, kLn2, logf(l_all));
            } else {
              part[f * (a.H + 2) + a.H] = m_all;
              part[f * (a.H + 2) + a.H + 1] = l_all;
            }
          }
        }
      }
      t = seg_end;
    }
  }
  if (*abort_flag != 0) __nanosleep(2000000);
}

// One CTA per (cut unit, row), thread = head element.  Units cut into `ranges` equal ranges: a CTA for each.  Ranges that
// end anywhere (ranges 0): a CTA for each boundary, of which the first one inside a unit merges it.
template <bool kBf16>
__global__ void __launch_bounds__(256)
fmha_decode_mma_combine_kernel(const __grid_constant__ Args a, int ctas, int ranges) {
  ptx::grid_dependency_wait();
  const int f = blockIdx.y;
  int unit, cta, last;   // CTA cta - 1 starts the unit or has its first tiles, CTA last finishes it
  if (ranges > 0) {
    unit = blockIdx.x;
    cta = unit * ranges + 1;
    last = cta + ranges - 2;
  } else {
    cta = blockIdx.x + 1;
    const int cut = range_begin(a.pieces, a.piece, cta, ctas);
    unit = cut / a.tiles_per_unit;
    const int unit_t0 = unit * a.tiles_per_unit;
    if (cut == unit_t0 || range_begin(a.pieces, a.piece, cta - 1, ctas) > unit_t0) return;
    last = cta;
    while (last + 1 < ctas && range_begin(a.pieces, a.piece, last + 1, ctas) < unit_t0 + a.tiles_per_unit) ++last;
  }
  const int64_t pitch = static_cast<int64_t>(a.F) * (a.H + 2);
  const float* row = a.partial + f * (a.H + 2);
  auto part = [&](int c) { return row + (a.slots * c + (a.slots == 2 && c == cta - 1 ? 1 : 0)) * pitch; };
  // Maxima, sums and values of many parts are asked for together: one trip to memory in place of one for each.
  constexpr int kHeld = 16;
  const int d = threadIdx.x;
  float m_all = -INFINITY, l_all = 0.0f, o = 0.0f;
  for (int c0 = cta - 1; c0 <= last; c0 += kHeld) {
    float m[kHeld], l[kHeld], v[kHeld];
#pragma unroll
    for (int i = 0; i < kHeld; ++i) {
      m[i] = -INFINITY;
      l[i] = v[i] = 0.0f;
      if (c0 + i <= last) {
        const float* pc = part(c0 + i);
        m[i] = pc[a.H];
        l[i] = pc[a.H + 1];
        if (d < a.H) v[i] = pc[d];
      }
    }
    float m_new = m_all;
#pragma unroll
    for (int i = 0; i < kHeld; ++i) m_new = fmaxf(m_new, m[i]);
    const float old = m_all == -INFINITY ? 0.0f : ptx::ex2_approx(m_all - m_new);
    l_all *= old;
    o *= old;
#pragma unroll
    for (int i = 0; i < kHeld; ++i) {
      const float coef = m[i] == -INFINITY ? 0.0f : ptx::ex2_approx(m[i] - m_new);
      l_all += l[i] * coef;
      o += v[i] * coef;
    }
    m_all = m_new;
  }
  const int head = unit % a.N, batch = unit / a.N;
  if (d < a.H) a.out[batch * a.o_strides[0] + head * a.o_strides[1] + f * a.o_strides[2] + d] = from_f32<kBf16>(o / l_all);
  if (d == 0 && a.lse != nullptr) a.lse[static_cast<int64_t>(unit) * a.F + f] = fmaf(m_all, kLn2, logf(l_all));
}

int slabs_of(int H) { return (H + 63) / 64; }

struct Plan {
  int tiles_per_unit = 0, pieces = 0, piece = 1, ctas = 0;
  int slots = 0;      // partials that a CTA may leave: 0 whole units, 1 a range inside a unit, 2 a range over several
};

// What the two kernels take, in ns (L2-warm launches in a CUDA graph, bf16, heads of 64, 128 and 256, 4 to 512 units, 40 to
// 4000 keys, 2 to 16 rows; fitted with 4 to 7 % mean error, heads of up to 192 in between).  The split-key kernel runs two
// rows a CTA and two CTAs an SM in waves; here a unit costs its merge, which grows with the rows and the head, beside its
// keys, and a cut unit the merge kernel.
struct Cost {
  int split_per_key, split_merge, split_percent;   // [slabs - 1]
  int unit[2], row[2], per_key_tenths[2], cut_per_range[2];   // up to 8 rows, more
};
constexpr Cost kCosts[4] = {{14, 2800, 100, {760, 1110}, {29, 70}, {56, 86}, {30, 20}},
                            {30, 3200, 93, {850, 1970}, {129, 170}, {70, 126}, {30, 36}},
                            {59, 3900, 90, {960, 3000}, {172, 190}, {137, 180}, {50, 70}},
                            {59, 4300, 88, {1350, 3660}, {255, 224}, {169, 240}, {80, 100}}};
constexpr int kCutCost[2] = {2300, 2600}, kShareCost[2] = {4200, 4900};   // (400 above the fit of a cut: near it whole units win)
// With no SM left free, the merge and the kernel behind it start only as these CTAs, which fill an SM's registers, end
// (8 units of 4000 keys H64, 16 and 18 ranges: F4 6.6 and 8.4 us, F16 9.3 and 12.5; 16 of 2000 keys, 8 and 9: F4 6.4 and 8.3).
constexpr int64_t kFullCost = 2000;

bool make_plan(const Problem& p, int sm_count, Plan* plan) {
  const int keys = slabs_of(p.H) > 2 ? 32 : 64;
  const int64_t per_unit = (static_cast<int64_t>(p.T) + keys - 1) / keys;
  const int64_t units = static_cast<int64_t>(p.B) * p.N, total = per_unit * units;
  if (p.F < 2 || p.F > kDecodeMaxQueries || total <= 0 || total > 0x7fffffff) return false;
  // Under the mask row f sees keys 0..f: at most F keys of the cache count, and those behind them may not
  // have been written yet (a product with P = 0 would turn their NaN into the result's).  The split-key
  // kernel ends at the last row's key: B32 N16 H256, 3001 keys, F = 4: 38 us there, 271 as a pass over the
  // whole cache; F = 16: 57 and 377.
  if (p.causal) return false;
  const Cost& cost = kCosts[slabs_of(p.H) - 1];
  const int wide = p.F > 8 ? 1 : 0;
  const int64_t fit = static_cast<int64_t>(kMaxPartialBytes / (static_cast<size_t>(p.F) * (p.H + 2) * sizeof(float)));
  const int64_t unit_ns = cost.unit[wide] + static_cast<int64_t>(cost.row[wide]) * p.F;
  const int64_t keys_ns = static_cast<int64_t>(cost.per_key_tenths[wide]) * p.T / 10;
  // Whole units; or, with no more units than SMs, each cut into equal ranges (equal shares of the tiles, which end
  // anywhere, were slower there: 16 units of 480 keys H256 F4 17 us, 11 whole); or, with more, equal shares (B20 N16
  // H256 F16, 130 keys: 59 us, 43 whole; 160 to 512 units H256, where the CTAs that go without in the last round could
  // take 64 to 128 keys each, 1 : 0.73, at 1000 to 1400 keys 1 : 1.13).
  int64_t ns = (units + sm_count - 1) / sm_count * (unit_ns + keys_ns), ranges = 1;
  plan->slots = 0;
  for (int64_t r = 2; r <= std::min({sm_count / units, static_cast<int64_t>(p.T / 128), fit / units}); ++r) {
    const int64_t t = unit_ns + keys_ns / r + kCutCost[wide] + cost.cut_per_range[wide] * r + (units * r * 8 > sm_count * 7 ? kFullCost : 0);
    if (t < ns) {
      ns = t;
      ranges = r;
      plan->slots = 1;
    }
  }
  const int64_t shares = std::min<int64_t>(sm_count, fit / 2);
  if (units > sm_count && shares > 1) {
    const int64_t t = unit_ns + units * (unit_ns + keys_ns) / shares + kShareCost[wide];
    if (t < ns) {
      ns = t;
      plan->slots = 2;
    }
  }
  // The split-key kernel stays where the estimates do not put this one 5 % ahead: short caches with many units and few
  // rows, and few units of 256-wide heads with many rows (one-pass against split-key, us: 4 units of 300 keys H256 F16 14
  // and 12; 16 units of 40 keys H128 F8 4.0 and 3.5; the other way 4 units of 4000 keys H64 F16 9.1 and 19, H128 F4 7.4 and
  // 15, 16 of 1000 keys H64 F16 7.8 and 15, 64 of 40 keys H64 F16 4.4 and 7.8).
  const int splits = decode_splits(p, sm_count);
  const int64_t split_ctas = units * ((p.F + 1) / 2) * splits, waves = (split_ctas + 2 * sm_count - 1) / (2 * sm_count);
  const int64_t split_ns = 550 + waves * (2750 + static_cast<int64_t>(cost.split_per_key) * ((p.T + splits - 1) / splits)) +
                           (splits > 1 ? cost.split_merge : 0);
  if ((2000 + ns) * 105 > split_ns * cost.split_percent) return false;
  plan->tiles_per_unit = static_cast<int>(per_unit);
  plan->piece = plan->slots == 0 ? static_cast<int>(per_unit) : 1;
  plan->pieces = static_cast<int>(plan->slots == 0 ? units : total);
  plan->ctas = static_cast<int>(plan->slots == 0 ? std::min<int64_t>(units, sm_count) : plan->slots == 1 ? units * ranges : shares);
  return true;
}
size_t partial_bytes(const Problem& p, const Plan& plan) {
  return static_cast<size_t>(plan.ctas) * plan.slots * p.F * (p.H + 2) * sizeof(float);
}

template <int kSlabs, int kNT, bool kBf16>
int launch_typed(const CUtensorMap& tk, const CUtensorMap& tv, const Args& a, const Plan& plan, const DeviceInfo& dev,
                 cudaStream_t stream) {
  using C = Cfg<kSlabs, kNT>;
  auto* fn = &fmha_decode_mma_kernel<kSlabs, kNT, kBf16>;
  static thread_local int configured_device = -1;
  if (configured_device != dev.device) {
    IXK_CUDA_OK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes));
    configured_device = dev.device;
  }
  const int rc = launch_overlapped(fn, dim3(plan.ctas), dim3(kThreads), C::kSmemBytes, stream, tk, tv, a);
  if (rc != IXK_OK || plan.slots == 0) return rc;
  // (slots 1: equal ranges inside units, ctas = units * ranges)
  const int units = plan.pieces / plan.tiles_per_unit, ranges = plan.slots == 1 ? plan.ctas / units : 0;
  return launch_overlapped(&fmha_decode_mma_combine_kernel<kBf16>, dim3(ranges > 0 ? units : plan.ctas - 1, a.F), dim3(kSlabs * 64), 0, stream, a,
                           plan.ctas, ranges);
}

}  // namespace

size_t decode_mma_workspace_bytes(const Problem& p, int sm_count) {
  Plan plan;
  return make_plan(p, sm_count, &plan) ? partial_bytes(p, plan) : 0;
}

bool decode_mma_applies(const Problem& p, const DeviceInfo& dev, const void* workspace, size_t workspace_bytes) {
  Plan plan;
  if (!make_plan(p, dev.sm_count, &plan)) return false;
  const size_t need = partial_bytes(p, plan);
  return need == 0 || (workspace != nullptr && workspace_bytes >= need && (reinterpret_cast<uintptr_t>(workspace) & 15u) == 0);
}

int launch_decode_mma(const Problem& p, const DeviceInfo& dev, void* workspace, cudaStream_t stream) {
  Plan plan;
  if (!make_plan(p, dev.sm_count, &plan)) return fail(IXK_UNIMPLEMENTED, "decode problem outside the tensor-core kernel's range");
  const int slabs = slabs_of(p.H);
  auto make_map = [&](CUtensorMap* out, const void* base, const int64_t* strides) -> int {
    TmapSpec s{};
    s.dtype = p.dtype == IXK_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    s.rank = 4;
    s.swizzle128 = true;
    s.dims[0] = p.H;
    s.dims[1] = p.T;
    s.dims[2] = strides[1] == 0 ? 1 : p.N;
    s.dims[3] = strides[0] == 0 ? 1 : p.B;
    // extent-1 dimensions still need a legal stride; any 16-byte multiple will do
    auto stride_bytes = [&](int64_t st, uint64_t fallback) -> uint64_t { return st > 0 ? static_cast<uint64_t>(st) * 2 : fallback; };
    const uint64_t pitch = stride_bytes(strides[2], static_cast<uint64_t>(p.H) * 2);
    s.strides_bytes[0] = pitch;
    s.strides_bytes[1] = stride_bytes(strides[1], pitch * p.T);
    s.strides_bytes[2] = stride_bytes(strides[0], pitch * p.T * p.N);
    s.box[0] = 64;
    s.box[1] = slabs > 2 ? 32 : 64;
    s.box[2] = s.box[3] = 1;
    return encode_tmap(out, base, s);
  };
  CUtensorMap tk, tv;
  if (make_map(&tk, p.k, p.k_strides) != IXK_OK || make_map(&tv, p.v, p.v_strides) != IXK_OK) return IXK_UNIMPLEMENTED;
  Args a{};
  a.B = p.B; a.N = p.N; a.H = p.H; a.F = p.F; a.T = p.T;
  a.scale_log2 = p.head_scale * kLog2e;
  a.tiles_per_unit = plan.tiles_per_unit;
  a.pieces = plan.pieces;
  a.piece = plan.piece;
  a.slots = plan.slots;
  a.q = static_cast<const uint16_t*>(p.q);
  a.bias = static_cast<const uint16_t*>(p.bias);
  a.out = static_cast<uint16_t*>(p.out);
  a.lse = p.lse;
  a.partial = static_cast<float*>(workspace);
  a.k_head_mul = p.k_strides[1] == 0 ? 0 : 1;
  a.k_batch_mul = p.k_strides[0] == 0 ? 0 : 1;
  a.v_head_mul = p.v_strides[1] == 0 ? 0 : 1;
  a.v_batch_mul = p.v_strides[0] == 0 ? 0 : 1;
  for (int i = 0; i < 3; ++i) {
    a.q_strides[i] = p.q_strides[i];
    a.o_strides[i] = p.o_strides[i];
    a.bias_strides[i] = p.bias_strides[i];
  }
  a.status_word = dev.status_word;
  auto go = [&](auto slabs_tag) {
    constexpr int kSlabs = decltype(slabs_tag)::value;
    if (p.dtype == IXK_BF16)
      return p.F <= 8 ? launch_typed<kSlabs, 1, true>(tk, tv, a, plan, dev, stream)
                      : launch_typed<kSlabs, 2, true>(tk, tv, a, plan, dev, stream);
    return p.F <= 8 ? launch_typed<kSlabs, 1, false>(tk, tv, a, plan, dev, stream)
                    : launch_typed<kSlabs, 2, false>(tk, tv, a, plan, dev, stream);
  };
  switch (slabs) {
    case 1: return go(std::integral_constant<int, 1>{});
    case 2: return go(std::integral_constant<int, 2>{});
    case 3: return go(std::integral_constant<int, 3>{});
    default: return go(std::integral_constant<int, 4>{});
  }
}

}  // namespace fmha
}  // namespace ixk
