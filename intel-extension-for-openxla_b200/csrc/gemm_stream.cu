// GEMM for few rows (M <= 128: decode-time projections): the time is one stream of the weight matrix through the
// chip, so everything here serves the stream.
//
//   D^T[n, m] = sum_k B[k, n] A[m, k]
//
// The weights are the M side of the MMA (128 columns of B = 128 lanes of tensor memory) and the rows of A
// its N side (16 to 128 wide, M rounded up to 16), so a pipeline stage is 16 KB of weights and 2 KB of A at
// M <= 16 where gemm_kernel moves and zero-fills 16 KB of A whatever M is.  One CTA works on 128 columns and
// one chunk of K; chunk count and shared memory are chosen so that all CTAs are on the chip at once, up to
// three per SM, and HBM sees one even wave instead of rounds of whole tiles (up to 56832 columns on 148 SMs;
// wider products run in rounds: see stream_alone).  While the kernel before it in
// the stream still runs, a CTA asks for its first stages of weights to be brought into L2 (a hint that reads
// nothing, so it needs no ordering with that kernel), which uses the HBM time that a decode step's small
// kernels leave idle.  With several chunks each CTA leaves an fp32 partial [M, 128] in scratch for
// splitk_reduce_kernel, otherwise it finishes the tile itself.
//
// Bound by HBM.  Calls back to back in a graph, gemm_kernel -> this (M x N x K, us; at 6.46 TB/s): 1 x 12288 x 3072
// 21.2 -> 15.1 (11.7), 1 x 3072 x 4096 10.6 -> 9.0 (3.9), 1 x 49152 x 3072 with GeGLU 75.4 -> 48.6 (46.7),
// 1 x 3072 x 24576 32.6 -> 26.4 (23.4); the same with 64 rows 20.5 -> 18.7, 11.4 -> 10.7, 59.5 -> 56.8, 31.4 -> 30.9;
// 16 x 1000 x 5000, whose K gemm_kernel did not cut, 21.2 -> 7.8.  Without the L2 hint 0.2 to 1 us more; chunks for one
// CTA per SM with the whole ring, or for three, up to 1 us more.  Every 32 rows cost the epilogue 1 us, which a CTA that
// finishes D itself has nothing to hide behind: see stream_alone.
//
// 192 threads: warp 0 TMA producer, warp 1 tensor memory + MMA issue, warps 2-5 epilogue (thread = one
// column of D, so a warp's accesses to a row of D are 32 consecutive elements).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "gemm_sm100.h"
#include "ptx.cuh"

namespace ixk {
namespace gemm {

namespace {

constexpr int kThreads = 192;
constexpr int kTileN = 128;          // columns of D per CTA
constexpr int kSlabBytes = 128;      // bytes of K per stage and row (one swizzle span)
constexpr int kWeightBytes = kTileN * kSlabBytes;
constexpr int kMaxStages = 12;
constexpr int kTailBytes = 256;      // barriers, tensor-memory address, abort flag
constexpr int kAssumedSms = 148;
constexpr int kCtasPerSm = 2;        // CTAs of an SM that a problem is cut for
constexpr int kMaxCtasPerSm = 3;     // ... and that there are at once where the columns alone are more
constexpr int kAloneTiles = 96;      // tiles of columns that one chunk of K is enough for
constexpr int kShortK = 2048;        // bytes of K
constexpr int kMinChunk = 8;         // slabs of K worth a CTA
constexpr int kMaxChunks = 32;

enum : int { kSiteProducer = 121, kSiteMma = 122, kSiteEpilogue = 123 };

struct StreamArgs {
  int M, N, tiles, slabs, chunk;     // chunk: slabs of K per CTA
  int stages, x_bytes, tmem_cols;
  int w_mn_major;
  uint32_t idesc;
  float acc_scale, beta;
  float* partial;                    // [chunks][M][N], or nullptr: the CTA writes D itself
  const void* bias;
  const void* c;
  void* d;
  int64_t ldc, ldd;
  int out_dtype, bias_dtype, act;
  int d_pairs;                       // 16-bit D whose columns come in 4-byte pairs
  int* status_word;
};

__device__ __forceinline__ float gelu_tanh(float x) {
  const float u = 0.7978845608028654f * x * fmaf(0.044715f * x, x, 1.0f);
  const float e = ptx::ex2_approx(-2.885390081777927f * u);
  return __fdividef(x, 1.0f + e);
}
__device__ __forceinline__ float load_f32(const void* p, int64_t i, int dtype) {
  if (dtype == IXK_F32) return static_cast<const float*>(p)[i];
  const uint16_t h = static_cast<const uint16_t*>(p)[i];
  return dtype == IXK_BF16 ? __uint_as_float(static_cast<uint32_t>(h) << 16) : __half2float(__ushort_as_half(h));
}
// 32 rows of one column, a pitch apart (the lanes of a warp are 32 consecutive columns).  All loads go out together, the
// type decided once for them: with a decision for each element each load waited for the one before (100 x 16208 x 80 with C
// in fp32: 34 us, 6.7 like this; 100 x 182192 x 320, bf16: 222, 62).
__device__ __forceinline__ void load_rows_f32(const void* src, int64_t at, int64_t pitch, int dtype, int rows, bool ok, float (&v)[32]) {
  if (dtype == IXK_F32) {
    const float* p = static_cast<const float*>(src) + at;
#pragma unroll
    for (int i = 0; i < 32; ++i, p += pitch) v[i] = ok && i < rows ? *p : 0.0f;
  } else {
    const uint16_t* p = static_cast<const uint16_t*>(src) + at;
    uint16_t h[32];
#pragma unroll
    for (int i = 0; i < 32; ++i, p += pitch) h[i] = ok && i < rows ? *p : static_cast<uint16_t>(0);
    const bool bf16 = dtype == IXK_BF16;
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = bf16 ? __uint_as_float(static_cast<uint32_t>(h[i]) << 16) : __half2float(__ushort_as_half(h[i]));
  }
}
__device__ __forceinline__ void store_rows_f32(float* dst, int64_t pitch, const float (&v)[32], int rows, bool ok) {
  if (!ok) return;
  if (rows == 32) {
#pragma unroll
    for (int i = 0; i < 32; ++i, dst += pitch) *dst = v[i];
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i, dst += pitch)
      if (i < rows) *dst = v[i];
  }
}

template <int kKind>
__global__ void __launch_bounds__(kThreads, 3)
gemm_stream_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const StreamArgs args) {
  constexpr int kElemBytes = kKind == ptx::kKindF16 ? 2 : 1;
  constexpr int kSlabElems = kSlabBytes / kElemBytes;
  constexpr int kUmmaK = 32 / kElemBytes;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  const int stage_bytes = kWeightBytes + args.x_bytes;
  const uint32_t bar_base = smem_base + args.stages * stage_bytes;
  uint8_t* tail = smem_raw + (bar_base - ptx::smem_u32(smem_raw)) + 8 * (2 * kMaxStages + 1);
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kMaxStages + s); };
  const uint32_t acc_bar = bar_base + 8u * (2 * kMaxStages);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(tail);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 4);
  static_assert(8 * (2 * kMaxStages + 1) + 8 <= kTailBytes, "barrier area");

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  ptx::AbortCtl ctl{abort_flag, args.status_word};

  const int tile = blockIdx.x % args.tiles;      // neighbouring CTAs read neighbouring columns of the same k rows
  const int split = blockIdx.x / args.tiles;
  const int n0 = tile * kTileN;
  const int slab0 = split * args.chunk;
  const int slabs = min(args.chunk, args.slabs - slab0);   // >= 1 by the launch

  if (threadIdx.x == 0) {
    ptx::prefetch_tmap(&tmap_w);
    ptx::prefetch_tmap(&tmap_x);
    const int ahead = min(slabs, args.stages);
    for (int s = 0; s < ahead; ++s) {
      const int k0 = (slab0 + s) * kSlabElems;
      if (args.w_mn_major) {
#pragma unroll
        for (int i = 0; i < kTileN / kSlabElems; ++i)
          if (n0 + i * kSlabElems < args.N) ptx::tma_prefetch_l2_2d(&tmap_w, n0 + i * kSlabElems, k0);
      } else {
        ptx::tma_prefetch_l2_2d(&tmap_w, k0, n0);
      }
    }
  }
  if (threadIdx.x == 32) {
    *abort_flag = 0;
    for (int s = 0; s < args.stages; ++s) {
      ptx::mbar_init(full_bar(s), 1);
      ptx::mbar_init(empty_bar(s), 1);
    }
    ptx::mbar_init(acc_bar, 1);
    ptx::fence_mbar_init();
  }
  if (warp == 1) {
    __syncwarp();
    ptx::tmem_alloc(ptx::smem_u32(const_cast<uint32_t*>(tmem_slot)), args.tmem_cols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  ptx::grid_dependency_sync();

  if (warp == 0) {
    int stage = 0;
    uint32_t phase = 0;
    for (int s = 0; s < slabs; ++s) {
      if (!ptx::mbar_wait(empty_bar(stage), phase ^ 1u, ctl, kSiteProducer)) break;
      const uint32_t w_dst = smem_base + stage * stage_bytes;
      const uint32_t bar = full_bar(stage);
      const int k0 = (slab0 + s) * kSlabElems;
      if (ptx::elect_one()) {
        ptx::mbar_expect_tx(bar, stage_bytes);
        if (args.w_mn_major) {
#pragma unroll
          for (int i = 0; i < kTileN / kSlabElems; ++i)
            ptx::tma_load_2d(w_dst + i * (kSlabElems * kSlabBytes), &tmap_w, bar, n0 + i * kSlabElems, k0);
        } else {
          ptx::tma_load_2d(w_dst, &tmap_w, bar, k0, n0);
        }
        ptx::tma_load_2d(w_dst + kWeightBytes, &tmap_x, bar, k0, 0);
      }
      __syncwarp();
      if (++stage == args.stages) {
        stage = 0;
        phase ^= 1u;
      }
    }
  } else if (warp == 1) {
    int stage = 0;
    uint32_t phase = 0;
    bool alive = true;
    const uint32_t w_lbo = args.w_mn_major ? kSlabElems * kSlabBytes : 16;
    const uint32_t w_kstep = args.w_mn_major ? kUmmaK * kSlabBytes : 32;
    for (int s = 0; s < slabs; ++s) {
      if (!ptx::mbar_wait(full_bar(stage), phase, ctl, kSiteMma)) {
        alive = false;
        break;
      }
      ptx::tc_fence_after_sync();
      const uint32_t w_src = smem_base + stage * stage_bytes;
      const uint32_t x_src = w_src + kWeightBytes;
#pragma unroll
      for (int ks = 0; ks < kSlabElems / kUmmaK; ++ks) {
        const uint64_t da = ptx::umma_smem_desc(w_src + ks * w_kstep, w_lbo, 1024);
        const uint64_t db = ptx::umma_smem_desc(x_src + ks * 32, 16, 1024);
        ptx::umma_ss_elect<kKind>(tmem_base, da, db, args.idesc, (s | ks) != 0 ? 1u : 0u);
      }
      ptx::umma_commit_elect(empty_bar(stage));
      if (++stage == args.stages) {
        stage = 0;
        phase ^= 1u;
      }
    }
    if (alive) ptx::umma_commit_elect(acc_bar);
  } else {
    const int quarter = warp & 3;
    const int n = n0 + quarter * 32 + lane;
    const bool n_ok = n < args.N;
    if (ptx::mbar_wait(acc_bar, 0, ctl, kSiteEpilogue)) {
      ptx::tc_fence_after_sync();
      const uint32_t acc = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
      const float bias = args.partial == nullptr && args.bias != nullptr && n_ok ? load_f32(args.bias, n, args.bias_dtype) : 0.0f;
#pragma unroll 1
      for (int m0 = 0; m0 < args.M; m0 += 32) {
        const int rows = min(32, args.M - m0);
        float c[32];
        if (args.c != nullptr) load_rows_f32(args.c, m0 * args.ldc + n, args.ldc, args.out_dtype, rows, n_ok, c);
        __syncwarp();
        uint32_t r[32];
        ptx::tmem_ld_32x32(acc + m0, r);
        ptx::tmem_ld_wait();
        float v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]) * args.acc_scale;
        if (args.partial != nullptr) {
          store_rows_f32(args.partial + (static_cast<int64_t>(split) * args.M + m0) * args.N + n, args.N, v, rows, n_ok);
          continue;
        }
        if (args.bias != nullptr) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] += bias;
        }
        if (args.c != nullptr) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = fmaf(args.beta, c[i], v[i]);
        }
        if (args.act == kActRelu) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = fmaxf(v[i], 0.0f);
        } else if (args.act == kActGelu) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = gelu_tanh(v[i]);
        }
        if (args.out_dtype == IXK_F32) {
          store_rows_f32(static_cast<float*>(args.d) + m0 * args.ldd + n, args.ldd, v, rows, n_ok);
        } else {
          // Rows 2k and 2k + 1 as 16-bit pairs; neighbouring lanes swap halves, so that even lanes hold two columns of
          // the first row, odd lanes two of the second: 4-byte stores, 64 bytes of two rows per instruction.
          __syncwarp();
          uint16_t* d = static_cast<uint16_t*>(args.d) + m0 * args.ldd + n;
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            uint32_t w;
            if (args.out_dtype == IXK_BF16) {
              const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
              w = *reinterpret_cast<const uint32_t*>(&h);
            } else {
              const __half2 h = __floats2half2_rn(v[2 * k], v[2 * k + 1]);
              w = *reinterpret_cast<const uint32_t*>(&h);
            }
            if (args.d_pairs != 0) {
              const uint32_t other = __shfl_xor_sync(0xffffffffu, w, 1);
              const uint32_t both = (lane & 1) == 0 ? __byte_perm(w, other, 0x5410) : __byte_perm(other, w, 0x7632);
              if (n_ok && 2 * k + (lane & 1) < rows) *reinterpret_cast<uint32_t*>(d + (2 * k + (lane & 1)) * args.ldd - (lane & 1)) = both;
            } else if (n_ok) {
              if (2 * k < rows) d[2 * k * args.ldd] = static_cast<uint16_t>(w & 0xffffu);
              if (2 * k + 1 < rows) d[(2 * k + 1) * args.ldd] = static_cast<uint16_t>(w >> 16);
            }
          }
        }
      }
    }
  }

  if (*abort_flag != 0) __nanosleep(2000000);
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem_base, args.tmem_cols);
  }
}

}  // namespace

bool stream_takes(int64_t M) { return M <= 128; }

bool stream_applies(const Problem& p) {
  return stream_takes(p.M) && p.batch == 1 && (p.kind == kKindF16 || p.kind == kKindF8) && !p.a_mn_major && p.aux == nullptr &&
         p.scatter_world == 0 && p.force_block_n == 0;
}

// One chunk of K, D finished by the CTAs: up to 32 rows, or where the columns alone make a CTA for two SMs of three; else
// gemm_kernel's narrower tiles are level or ahead (us, gemm_kernel and this, bf16: 16 x 512 x 1024 6.3 and 6.1, 64 rows
// 6.4 and 7.2; 16 x 4096 x 4096 17.8 and 16.7, 128 rows 18.2 and 20.3; 16 x 16384 x 4096 32.4 and 22.6, 128 rows 32.8
// and 26.6; 64 x 8192 x 8192 32.5 and 32.3).  fp8 with more rows only on K-major weights (128 x 16384 x 4096: 18.5 and
// 16.8, N-major 13.7 and 16.3).  More tiles than three CTAs per SM are rounds, each with a set-up and an epilogue that
// nothing hides, which more than 64 rows do not bear (128 x 59824 x 224 13.1 and 19.7, 80 x 58128 x 6576 128 and 168; 64
// rows 0.83 of gemm_kernel's time on average and 1.09 at most, 32 rows 0.67), nor more than 16 where a long K is streamed
// once more for a second round of a third of the CTAs or fewer (64 x 60000 x 6600 132 and 153, 32 x 60000 x 3088 62 and
// 69); and nor does the epilogue of more than 96 rows behind a short K pay (128 x 35984 x 464 11.4 and 13.9).
bool stream_alone(const Problem& p) {
  const int64_t tiles = (p.N + kTileN - 1) / kTileN, k_bytes = p.K * (p.kind == kKindF16 ? 2 : 1);
  const bool rounds = tiles > kMaxCtasPerSm * kAssumedSms;
  if (rounds && tiles <= (kMaxCtasPerSm + 1) * kAssumedSms && k_bytes >= 2 * kShortK) return p.M <= 16;
  if (p.M <= 32) return true;
  if (tiles < kAloneTiles || (p.kind == kKindF8 && p.b_mn_major)) return false;
  if (rounds) return p.M <= 64;
  return p.M <= 96 || tiles > kCtasPerSm * kAssumedSms || k_bytes >= kShortK;
}

// Chunks of K: as many as give every SM its two CTAs in one wave, each of kMinChunk slabs at least, no more than
// the scratch holds partials of, and none that would make writing and reading the partials (8 bytes an element) more
// than half of the weights' bytes.  Where the columns alone make a CTA for two SMs of three, a second chunk gains less than
// the pass over the partials costs (one chunk and two, us: 16 x 12832 x 1312 9.8 and 10.9, 64 x 15888 x 2944 19.0 and 23.8,
// 80 x 13248 x 22368 92.7 and 94.0), unless there is a pass over them anyway (`summed`: GeGLU).
int stream_splits(int64_t M, int64_t N, int64_t K, int elem_bytes, size_t workspace_bytes, bool summed) {
  const int64_t tiles = (N + kTileN - 1) / kTileN, slabs = (K * elem_bytes + kSlabBytes - 1) / kSlabBytes;
  if (tiles > kAloneTiles && !summed) return 1;
  const int64_t fit = static_cast<int64_t>(workspace_bytes / (static_cast<size_t>(M) * N * sizeof(float)));
  int64_t chunks = std::min<int64_t>({kCtasPerSm * kAssumedSms / tiles, slabs / kMinChunk, kMaxChunks, fit, K * elem_bytes / (16 * M)});
  chunks = std::max<int64_t>(chunks, 1);
  const int64_t chunk = (slabs + chunks - 1) / chunks;
  return static_cast<int>((slabs + chunk - 1) / chunk);
}

// `partial`: nullptr (one chunk, D finished here) or scratch for splits x M x N floats.
int launch_stream(const Problem& p, int splits, float* partial, const DeviceInfo& dev, cudaStream_t stream) {
  const int es = p.kind == kKindF16 ? 2 : 1;
  const int slab_elems = kSlabBytes / es;
  const int rows = static_cast<int>((p.M + 15) / 16) * 16;

  const CUtensorMapDataType dt = es == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                         : (p.ab_dtype == IXK_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16);
  CUtensorMap tw, tx;
  TmapSpec s{};
  s.dtype = dt;
  s.rank = 2;
  s.swizzle128 = true;
  s.dims[0] = p.b_mn_major ? p.N : p.K;
  s.dims[1] = p.b_mn_major ? p.K : p.N;
  s.strides_bytes[0] = static_cast<uint64_t>(p.ldb) * es;
  s.box[0] = slab_elems;
  s.box[1] = p.b_mn_major ? slab_elems : kTileN;
  int rc = encode_tmap(&tw, p.b, s);
  if (rc != IXK_OK) return rc;
  s.dims[0] = p.K;
  s.dims[1] = p.M;
  s.strides_bytes[0] = static_cast<uint64_t>(p.lda) * es;
  s.box[0] = slab_elems;
  s.box[1] = rows;
  if ((rc = encode_tmap(&tx, p.a, s)) != IXK_OK) return rc;

  StreamArgs a{};
  a.M = static_cast<int>(p.M);
  a.N = static_cast<int>(p.N);
  a.tiles = static_cast<int>((p.N + kTileN - 1) / kTileN);
  a.slabs = static_cast<int>((p.K + slab_elems - 1) / slab_elems);
  a.chunk = (a.slabs + splits - 1) / splits;
  a.x_bytes = rows * kSlabBytes;
  a.tmem_cols = 32;
  while (a.tmem_cols < rows) a.tmem_cols *= 2;
  a.w_mn_major = p.b_mn_major ? 1 : 0;
  a.idesc = ptx::umma_idesc(p.b_fmt, p.a_fmt, a.w_mn_major, 0, kTileN, rows);
  a.acc_scale = p.acc_scale;
  a.beta = p.beta;
  a.partial = partial;
  a.bias = p.bias;
  a.c = partial == nullptr && p.beta != 0.0f ? p.c : nullptr;   // (with chunks their sum adds it)
  a.d = p.d;
  a.ldc = p.ldc;
  a.ldd = p.ldd;
  a.out_dtype = p.out_dtype;
  a.bias_dtype = p.bias_dtype;
  a.act = p.act;
  a.d_pairs = p.N % 2 == 0 && p.ldd % 2 == 0 && (reinterpret_cast<uintptr_t>(p.d) & 3u) == 0 ? 1 : 0;
  a.status_word = dev.status_word;
  const int64_t ctas = static_cast<int64_t>(a.tiles) * splits;
  if (ctas > 0x7fffffff) return fail(IXK_UNIMPLEMENTED, "too many tiles");
  // Shared memory for as many CTAs per SM as one wave takes (the ring of a lone CTA is as deep as there is room), three
  // at most, and no more than tensor memory has columns for.
  const int per_sm = ctas <= dev.sm_count ? 1 : ctas > kCtasPerSm * dev.sm_count && a.tmem_cols <= 128 ? kMaxCtasPerSm : kCtasPerSm;
  const int stage_bytes = kWeightBytes + a.x_bytes;
  a.stages = std::min<int>(kMaxStages, ((228 * 1024) / per_sm - 2 * 1024 - kTailBytes) / stage_bytes);
  const size_t smem = static_cast<size_t>(a.stages) * stage_bytes + kTailBytes + 1024;
  auto go = [&](auto kind_tag) -> int {
    auto* fn = &gemm_stream_kernel<decltype(kind_tag)::value>;
    static thread_local int configured_device = -1;
    if (configured_device != dev.device) {
      IXK_CUDA_OK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024));
      configured_device = dev.device;
    }
    return launch_overlapped(fn, dim3(static_cast<unsigned>(ctas)), dim3(kThreads), smem, stream, tw, tx, a);
  };
  return p.kind == kKindF16 ? go(std::integral_constant<int, kKindF16>{}) : go(std::integral_constant<int, kKindF8>{});
}

}  // namespace gemm
}  // namespace ixk
