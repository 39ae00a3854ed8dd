// Attention forward over at most 128 keys (the cross-attention of an image model to its prompt, short
// sequences) for head sizes up to 128.
//
// One block of keys is the whole row: no running maximum, no rescale, no ring.  What a call costs is latency
// (set-up, Q and K arriving, two products, a row's softmax, the store), so the work is cut into tiles of 128
// query rows that are each a CTA of their own, small enough for two to four on an SM: one tile's loads and
// stores run under the others' arithmetic, and a launch is one wave where fmha_prefill_kernel's 256-row items,
// one per SM at a time, make two rounds of the longest chain.  B2 N20 F1024 T77 H64 fp16: 12.5 -> 8.1 us.
//
//   warps 0-3  softmax and epilogue: thread = one query row = one lane of tensor memory
//   warp 4     TMA loads, both products
//
// Tensor memory: S in columns [0, 128), P over it as 16-bit pairs in [0, 64); O behind S, or for heads of up
// to 64 in [64, 128), which P.V may overwrite because every score has been read by then.  The scores are read
// twice (maximum, then exponentials) instead of held in 128 registers.  O leaves through Q's shared memory.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "fmha_sm100.h"
#include "ptx.cuh"

namespace ixk {
namespace fmha {

namespace {

constexpr int kTileQ = 128;
constexpr int kMaxKeys = 128;
constexpr int kAssumedSms = 148;
constexpr int kThreads = 160;
constexpr int kBoxElems = 64;                 // 16-bit elements per 128-byte swizzle row
constexpr int kQBoxBytes = kTileQ * 128;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

enum : int { kSiteShortQK = 221, kSiteShortP = 222, kSiteShortV = 223, kSiteShortS = 224, kSiteShortO = 225 };

struct ShortArgs {
  int N, H, F, T;
  int qtiles, keys;          // keys: T rounded up to 16
  int causal, is_bf16, out_tma;
  int k_head_mul, k_batch_mul, v_head_mul, v_batch_mul;   // 0: one K / V for all heads or batches
  float scale_log2;
  uint16_t* out;
  int64_t o_strides[3];
  float* lse;
  int* status_word;
};

__device__ __forceinline__ uint32_t pack2(float lo, float hi, bool bf16) {
  if (bf16) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

template <int kBoxes>   // 64-element boxes of a row: 1 (H <= 64) or 2
__global__ void __launch_bounds__(kThreads, kBoxes == 1 ? 4 : 2)
fmha_short_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                  const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_o, const ShortArgs args) {
  constexpr int kHeadDim = kBoxes * kBoxElems;
  constexpr int kTmemCols = kBoxes == 1 ? 128 : 256;
  constexpr int kTmemO = kBoxes == 1 ? 64 : 128;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t q_smem = smem_base;
  const int kv_box = args.keys * 128;
  const uint32_t k_smem = q_smem + kBoxes * kQBoxBytes;
  const uint32_t v_smem = k_smem + kBoxes * kv_box;
  __shared__ __align__(8) uint64_t bars[5];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  const uint32_t qk_full = ptx::smem_u32(&bars[0]), v_full = ptx::smem_u32(&bars[1]), s_full = ptx::smem_u32(&bars[2]),
                 p_full = ptx::smem_u32(&bars[3]), o_full = ptx::smem_u32(&bars[4]);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  ptx::AbortCtl ctl{&abort_word, args.status_word};

  const int pair = blockIdx.x / args.qtiles;
  const int q0 = (blockIdx.x - pair * args.qtiles) * kTileQ;
  const int head = pair % args.N, batch = pair / args.N;

  if (warp == 4) {
    if (lane == 0) {
      abort_word = 0;
      ptx::mbar_init(qk_full, 1);
      ptx::mbar_init(v_full, 1);
      ptx::mbar_init(s_full, 1);
      ptx::mbar_init(p_full, 128);
      ptx::mbar_init(o_full, 1);
      ptx::fence_mbar_init();
      ptx::prefetch_tmap(&tmap_q);
      ptx::prefetch_tmap(&tmap_k);
      ptx::prefetch_tmap(&tmap_v);
      if (args.out_tma) ptx::prefetch_tmap(&tmap_o);
    }
    __syncwarp();
    ptx::tmem_alloc(ptx::smem_u32(&tmem_slot), kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem = *const_cast<volatile uint32_t*>(&tmem_slot);
  ptx::grid_dependency_sync();

  if (warp == 4) {
    if (ptx::elect_one()) {
      ptx::mbar_expect_tx(qk_full, kBoxes * (kQBoxBytes + kv_box));
      ptx::mbar_expect_tx(v_full, kBoxes * kv_box);
#pragma unroll
      for (int c = 0; c < kBoxes; ++c) {
        ptx::tma_load_4d(k_smem + c * kv_box, &tmap_k, qk_full, c * kBoxElems, 0, head * args.k_head_mul, batch * args.k_batch_mul);
        ptx::tma_load_4d(q_smem + c * kQBoxBytes, &tmap_q, qk_full, c * kBoxElems, q0, head, batch);
      }
#pragma unroll
      for (int c = 0; c < kBoxes; ++c)
        ptx::tma_load_4d(v_smem + c * kv_box, &tmap_v, v_full, c * kBoxElems, 0, head * args.v_head_mul, batch * args.v_batch_mul);
    }
    __syncwarp();
    const uint32_t fmt = args.is_bf16 ? 1u : 0u;
    if (ptx::mbar_wait(qk_full, 0, ctl, kSiteShortQK)) {
      ptx::tc_fence_after_sync();
      const uint32_t idesc_s = ptx::umma_idesc(fmt, fmt, 0, 0, kTileQ, args.keys);
#pragma unroll
      for (int ks = 0; ks < kHeadDim / 16; ++ks)
        ptx::umma_ss_elect<ptx::kKindF16>(tmem, ptx::umma_smem_desc(q_smem + (ks >> 2) * kQBoxBytes + (ks & 3) * 32, 16, 1024),
                                          ptx::umma_smem_desc(k_smem + (ks >> 2) * kv_box + (ks & 3) * 32, 16, 1024), idesc_s, ks != 0);
      ptx::umma_commit_elect(s_full);
      if (ptx::mbar_wait(v_full, 0, ctl, kSiteShortV) && ptx::mbar_wait(p_full, 0, ctl, kSiteShortP)) {
        ptx::tc_fence_after_sync();
        const uint32_t idesc_o = ptx::umma_idesc(fmt, fmt, 0, 1, kTileQ, kHeadDim);
        for (int ks = 0; ks < args.keys / 16; ++ks)
          if (ptx::elect_one())
            ptx::umma_ts_f16(tmem + kTmemO, tmem + ks * 8, ptx::umma_smem_desc(v_smem + ks * 2048, kv_box, 1024), idesc_o, ks != 0);
        __syncwarp();
        ptx::umma_commit_elect(o_full);
      }
    }
  } else {
    const bool bf16 = args.is_bf16 != 0;
    const int row = warp * 32 + lane;
    const int f = q0 + row;
    const uint32_t t_addr = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    const int limit = args.causal ? min(args.T, f + 1) : args.T;   // keys that this row sees
    if (ptx::mbar_wait(s_full, 0, ctl, kSiteShortS)) {
      ptx::tc_fence_after_sync();
      // scores in the log2 domain; the columns behind `limit` are left out of both passes
      float mx = -INFINITY;
#pragma unroll 1
      for (int c0 = 0; c0 < args.keys; c0 += 32) {
        uint32_t r[32];
        ptx::tmem_ld_32x32(t_addr + c0, r);
        ptx::tmem_ld_wait();
        float m[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float x = __uint_as_float(r[i]) * args.scale_log2;
          m[i & 3] = fmaxf(m[i & 3], c0 + i < limit ? x : -INFINITY);
        }
        mx = fmaxf(mx, fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3])));
      }
      const float m_use = mx == -INFINITY ? 0.0f : mx;
      float sums[2] = {0.0f, 0.0f};
#pragma unroll 1
      for (int c0 = 0; c0 < args.keys; c0 += 32) {
        uint32_t r[32], pk[16];
        ptx::tmem_ld_32x32(t_addr + c0, r);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float p[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float x = __uint_as_float(r[i + e]) * args.scale_log2;
            p[e] = c0 + i + e < limit ? ptx::ex2_approx(x - m_use) : 0.0f;
            sums[e] += p[e];
          }
          pk[i >> 1] = pack2(p[0], p[1], bf16);
        }
        ptx::tmem_st_32x16(t_addr + c0 / 2, pk);   // (over scores of columns already read twice)
      }
      ptx::tmem_st_wait();
      ptx::tc_fence_before_sync();
      ptx::mbar_arrive(p_full);
      const float l = sums[0] + sums[1];
      const float inv_l = 1.0f / l;
      const bool row_ok = f < args.F;
      if (args.lse != nullptr && row_ok)
        args.lse[(static_cast<int64_t>(batch) * args.N + head) * args.F + f] = (mx + log2f(l)) * kLn2;
      if (ptx::mbar_wait(o_full, 0, ctl, kSiteShortO)) {
        ptx::tc_fence_after_sync();
#pragma unroll
        for (int c = 0; c < kHeadDim / 32; ++c) {
          if (c * 32 >= args.H) break;
          uint32_t o[32], wv[16];
          ptx::tmem_ld_32x32(t_addr + kTmemO + c * 32, o);
          ptx::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i)
            wv[i] = pack2(__uint_as_float(o[2 * i]) * inv_l, __uint_as_float(o[2 * i + 1]) * inv_l, bf16);
          if (args.out_tma) {
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              const int piece = (c & 1) * 4 + g;
              const uint32_t addr = q_smem + (c >> 1) * kQBoxBytes + row * 128 + ((piece ^ (row & 7)) << 4);
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(wv[4 * g]), "r"(wv[4 * g + 1]),
                           "r"(wv[4 * g + 2]), "r"(wv[4 * g + 3])
                           : "memory");
            }
          } else if (row_ok) {
            uint16_t* orow = args.out + batch * args.o_strides[0] + head * args.o_strides[1] + static_cast<int64_t>(f) * args.o_strides[2] + c * 32;
            const int count = min(32, args.H - c * 32);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              if (2 * i < count) orow[2 * i] = static_cast<uint16_t>(wv[i] & 0xffffu);
              if (2 * i + 1 < count) orow[2 * i + 1] = static_cast<uint16_t>(wv[i] >> 16);
            }
          }
          __syncwarp();
        }
      }
    }
    if (args.out_tma) {
      ptx::fence_proxy_async_smem();
      ptx::named_barrier_sync(1, 128);
      if (threadIdx.x == 0 && *const_cast<volatile int*>(&abort_word) == 0) {
#pragma unroll
        for (int c = 0; c < kBoxes; ++c)
          if (c * kBoxElems < args.H) ptx::tma_store_4d(&tmap_o, q_smem + c * kQBoxBytes, c * kBoxElems, q0, head, batch);
        ptx::bulk_commit_group();
        ptx::bulk_wait_group<0>();
      }
    }
  }

  if (*const_cast<volatile int*>(&abort_word) != 0) __nanosleep(2000000);
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 4) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem, kTmemCols);
  }
}

}  // namespace

// Heads of up to 64 always (four CTAs per SM: 0.41 to 0.96 of the general kernel's time over 186 sizes).  Wider ones, two
// CTAs per SM, up to four tiles an SM, or sixteen with up to 64 keys, beyond which the general kernel's ring hides more
// than this one's neighbours (H 96 to 128, us, general and this: 4 tiles an SM 0.7 to 1.0 of its time; T 71, 5 tiles an SM,
// 21.1 and 23.0; T 95, 21 tiles 54 and 73; T 125, 80 tiles 176 and 290; T 28, 20 tiles 50.7 and 53.1).
bool short_applies(const Problem& p) {
  const int64_t ctas = static_cast<int64_t>(p.B) * p.N * ((p.F + kTileQ - 1) / kTileQ);
  if (p.T > kMaxKeys || p.H > 128 || p.bias != nullptr || ctas > 0x7fffffff) return false;
  return p.H <= kBoxElems || ctas <= (p.T <= 64 ? 16 : 4) * kAssumedSms;
}

int launch_short(const Problem& p, const DeviceInfo& dev, cudaStream_t stream) {
  const CUtensorMapDataType dt = p.dtype == IXK_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  const int keys = (p.T + 15) / 16 * 16;
  // (strides as in the general kernel: 0 over heads or batches of K and V is one tensor for all of them)
  auto make_map = [&](CUtensorMap* out, const void* base, const int64_t* strides, int rows, int box_rows) -> int {
    TmapSpec s{};
    s.dtype = dt;
    s.rank = 4;
    s.swizzle128 = true;
    s.dims[0] = p.H;
    s.dims[1] = rows;
    s.dims[2] = strides[1] == 0 ? 1 : p.N;
    s.dims[3] = strides[0] == 0 ? 1 : p.B;
    auto stride_bytes = [&](int64_t st, uint64_t fallback) -> uint64_t { return st > 0 ? static_cast<uint64_t>(st) * 2 : fallback; };
    const uint64_t row_pitch = stride_bytes(strides[2], static_cast<uint64_t>(p.H) * 2);
    s.strides_bytes[0] = row_pitch;
    s.strides_bytes[1] = stride_bytes(strides[1], row_pitch * rows);
    s.strides_bytes[2] = stride_bytes(strides[0], row_pitch * rows * p.N);
    s.box[0] = kBoxElems;
    s.box[1] = box_rows;
    s.box[2] = s.box[3] = 1;
    return encode_tmap(out, base, s);
  };
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = make_map(&tq, p.q, p.q_strides, p.F, kTileQ)) != IXK_OK) return rc;
  if ((rc = make_map(&tk, p.k, p.k_strides, p.T, keys)) != IXK_OK) return rc;
  if ((rc = make_map(&tv, p.v, p.v_strides, p.T, keys)) != IXK_OK) return rc;
  CUtensorMap to = tq;
  bool out_tma = (reinterpret_cast<uintptr_t>(p.out) & 15u) == 0 && p.o_strides[2] >= p.H;
  for (int i = 0; i < 3; ++i) out_tma = out_tma && p.o_strides[i] % 8 == 0;
  if (out_tma && (rc = make_map(&to, p.out, p.o_strides, p.F, kTileQ)) != IXK_OK) return rc;

  ShortArgs a{};
  a.N = p.N;
  a.H = p.H;
  a.F = p.F;
  a.T = p.T;
  a.qtiles = (p.F + kTileQ - 1) / kTileQ;
  a.keys = keys;
  a.causal = p.causal ? 1 : 0;
  a.is_bf16 = p.dtype == IXK_BF16 ? 1 : 0;
  a.out_tma = out_tma ? 1 : 0;
  a.k_head_mul = p.k_strides[1] == 0 ? 0 : 1;
  a.k_batch_mul = p.k_strides[0] == 0 ? 0 : 1;
  a.v_head_mul = p.v_strides[1] == 0 ? 0 : 1;
  a.v_batch_mul = p.v_strides[0] == 0 ? 0 : 1;
  a.scale_log2 = p.head_scale * kLog2e;
  a.out = static_cast<uint16_t*>(p.out);
  for (int i = 0; i < 3; ++i) a.o_strides[i] = p.o_strides[i];
  a.lse = p.lse;
  a.status_word = dev.status_word;
  const unsigned ctas = static_cast<unsigned>(static_cast<int64_t>(p.B) * p.N * a.qtiles);
  auto go = [&](auto boxes_tag) -> int {
    constexpr int kBoxes = decltype(boxes_tag)::value;
    auto* fn = &fmha_short_kernel<kBoxes>;
    static thread_local int configured_device = -1;
    if (configured_device != dev.device) {
      IXK_CUDA_OK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 1024 + kBoxes * (kQBoxBytes + 2 * kMaxKeys * 128)));
      configured_device = dev.device;
    }
    return launch_overlapped(fn, dim3(ctas), dim3(kThreads), 1024 + kBoxes * (kQBoxBytes + 2 * keys * 128), stream, tq, tk, tv, to, a);
  };
  return p.H <= kBoxElems ? go(std::integral_constant<int, 1>{}) : go(std::integral_constant<int, 2>{});
}

}  // namespace fmha
}  // namespace ixk
