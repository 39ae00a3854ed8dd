// Split-K for skinny GEMMs (decode-time projections, where the whole problem is one
// stream of the weight matrix through the chip).  With a single row of output tiles there are too
// few tiles to occupy 148 SMs, so the K range is cut into `splits` chunks, each of which leaves an fp32
// partial [M, N] in the caller's workspace (gemm_stream_kernel; for an A with its rows contiguous, which that kernel
// does not take, and for more rows in few tiles, the batch dimension of gemm_kernel), and this file's kernel sums the
// partials and applies the epilogue once.
// The reference reaches the same end with shared-local-memory k-slicing inside a work-group
// (SLM_KS in xla/service/gpu/xetla/gemm/gemm_dispatch.h:183-214); here the slices are CTAs.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "gemm_sm100.h"
#include "ptx.cuh"

namespace ixk {
namespace gemm {

namespace {

constexpr int kAssumedSms = 148;
constexpr int kSlabBytes = 128;    // bytes of K per pipeline stage
constexpr int kSlabElems16 = kSlabBytes / 2;
constexpr int kMinChunk = 512;     // smallest K chunk worth a CTA
constexpr int64_t kSlabNarrowNs = 160, kSlabWideNs = 210, kReduceNs = 3500, kReduceBytesPerNs = 2500;   // see tiled_splits
// CTAs of a reduce launch at most, per SM.  It is set up while the GEMM still runs, whose CTA leaves an SM room for seven
// of the eight CTAs of 256 threads it otherwise holds: a grid of just eight would end with a round of stragglers (128 x
// 12288 x 3072 in a graph: 24.3 us with 8, 24.1 with 6, 22.8 with 16; 23.3 launched in order with 8).
constexpr int kReduceCtasPerSm = 16;

__device__ __forceinline__ float gelu_tanh_f(float x) {
  const float u = 0.7978845608028654f * x * fmaf(0.044715f * x, x, 1.0f);
  const float e = ptx::ex2_approx(-2.885390081777927f * u);
  return __fdividef(x, 1.0f + e);
}
__device__ __forceinline__ float load_as_f32(const void* p, int64_t i, int dtype) {
  if (dtype == IXK_F32) return static_cast<const float*>(p)[i];
  const uint16_t h = static_cast<const uint16_t*>(p)[i];
  return dtype == IXK_BF16 ? __uint_as_float(static_cast<uint32_t>(h) << 16) : __half2float(__ushort_as_half(h));
}
__device__ __forceinline__ void store_from_f32(void* p, int64_t i, int dtype, float v) {
  if (dtype == IXK_F32) {
    static_cast<float*>(p)[i] = v;
  } else if (dtype == IXK_BF16) {
    static_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v);
  } else {
    static_cast<__half*>(p)[i] = __float2half_rn(v);
  }
}

struct ReduceArgs {
  const float* partial;  // [splits][M][N]
  int splits, M, N;
  const void* bias;
  const void* c;
  void* d;
  int64_t ldc, ldd;
  int out_dtype, bias_dtype, act;
  float beta;
  int geglu;   // the N columns are [gate | up] halves: out[m, n] = round(gelu(gate)) * round(up), N / 2 columns
};

__device__ __forceinline__ void reduce_epilogue_store(const ReduceArgs& a, int m, int n, float v) {
  if (a.bias != nullptr) v += load_as_f32(a.bias, n, a.bias_dtype);
  if (a.c != nullptr) v = fmaf(a.beta, load_as_f32(a.c, static_cast<int64_t>(m) * a.ldc + n, a.out_dtype), v);
  if (a.act == kActRelu) v = fmaxf(v, 0.0f);
  if (a.act == kActGelu) v = gelu_tanh_f(v);
  store_from_f32(a.d, static_cast<int64_t>(m) * a.ldd + n, a.out_dtype, v);
}

// Four consecutive columns of one row summed over the chunks, in chunk order, with the loads of up to eight chunks in
// flight together: a decode step's reduce is a few dozen threads whose time is the number of trips to L2.  kHeld is no more
// than there are chunks, up to a power of two: room for eight in every thread left a pass over one or two large planes with
// too few threads (GeGLU, us, four one by one, eight, and as many as there are: 128 x 42992 x 768 28.9, 29.8, 24.8; 112 x
// 54512 x 640 27.2, 31.0, 25.6).
template <int kHeld>
__device__ __forceinline__ float4 sum_chunks(const float4* src, int64_t plane4, int splits) {
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int s0 = 0; s0 < splits; s0 += kHeld) {
    float4 v[kHeld];
#pragma unroll
    for (int i = 0; i < kHeld; ++i) v[i] = s0 + i < splits ? src[(s0 + i) * plane4] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < kHeld; ++i) {
      acc.x += v[i].x;
      acc.y += v[i].y;
      acc.z += v[i].z;
      acc.w += v[i].w;
    }
  }
  return acc;
}
// (N is a multiple of 4, so the partial planes can be read 16 bytes at a time; otherwise one element per thread.)
__device__ __forceinline__ float round_to(float v, int dtype) {
  if (dtype == IXK_BF16) return __bfloat162float(__float2bfloat16_rn(v));
  if (dtype == IXK_F16) return __half2float(__float2half_rn(v));
  return v;
}

// GeGLU over the two halves of a [M, 2 N'] product: thread = four consecutive output columns; the
// gate is activated and rounded, the up half rounded, then multiplied (the values a gate GEMM with
// a GELU epilogue, an up GEMM and an elementwise product would have produced one after the other).
template <int kHeld>
__global__ void splitk_reduce_geglu_kernel(const ReduceArgs a) {
  ptx::grid_dependency_sync();
  const int half = a.N / 2, h4 = half / 4;
  const int64_t plane4 = static_cast<int64_t>(a.M) * a.N / 4;
  const int64_t total = static_cast<int64_t>(a.M) * h4;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int m = static_cast<int>(i / h4);
    const int n = static_cast<int>(i - static_cast<int64_t>(m) * h4) * 4;
    const float4* gsrc = reinterpret_cast<const float4*>(a.partial) + (static_cast<int64_t>(m) * a.N + n) / 4;
    const float4* usrc = gsrc + h4;
    const float4 g = sum_chunks<kHeld>(gsrc, plane4, a.splits), u = sum_chunks<kHeld>(usrc, plane4, a.splits);
    const float gs[4] = {g.x, g.y, g.z, g.w}, us[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int e = 0; e < 4; ++e)
      store_from_f32(a.d, static_cast<int64_t>(m) * a.ldd + n + e, a.out_dtype,
                     round_to(gelu_tanh_f(gs[e]), a.out_dtype) * round_to(us[e], a.out_dtype));
  }
}

template <int kHeld>   // 0: N is not a multiple of 4
__global__ void splitk_reduce_kernel(const ReduceArgs a) {
  ptx::grid_dependency_sync();
  const int64_t plane = static_cast<int64_t>(a.M) * a.N;
  if constexpr (kHeld > 0) {
    const int64_t total = plane / 4;
    const int n4 = a.N / 4;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
      const int m = static_cast<int>(i / n4);
      const int n = static_cast<int>(i - static_cast<int64_t>(m) * n4) * 4;
      const float4 acc = sum_chunks<kHeld>(reinterpret_cast<const float4*>(a.partial) + i, plane / 4, a.splits);
      reduce_epilogue_store(a, m, n, acc.x);
      reduce_epilogue_store(a, m, n + 1, acc.y);
      reduce_epilogue_store(a, m, n + 2, acc.z);
      reduce_epilogue_store(a, m, n + 3, acc.w);
    }
  } else {
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < plane;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
      const int m = static_cast<int>(i / a.N);
      const int n = static_cast<int>(i - static_cast<int64_t>(m) * a.N);
      float v = 0.0f;
      for (int s = 0; s < a.splits; ++s) v += a.partial[s * plane + i];
      reduce_epilogue_store(a, m, n, v);
    }
  }
}

}  // namespace

// Threads and CTAs for `total` items: small CTAs where that spreads few items over more SMs.
struct ReduceGrid {
  unsigned blocks, threads;
};
static ReduceGrid reduce_grid(int64_t total, int sm_count) {
  const unsigned threads = total <= 256 * static_cast<int64_t>(sm_count) ? 64 : 256;
  const int64_t blocks = std::min<int64_t>((total + threads - 1) / threads, static_cast<int64_t>(kReduceCtasPerSm) * sm_count);
  return ReduceGrid{static_cast<unsigned>(blocks), threads};
}

int split_k_factor(int64_t M, int64_t N, int64_t K, int64_t batch, bool fp8) {
  if (batch != 1 || M > 128 || fp8) return 1;
  const int64_t tiles = (N + 127) / 128;  // one row of 128 x 128 tiles
  if (K % kSlabElems16 != 0) return 1;
  // One CTA per SM at this kernel's shared-memory size, so tiles x chunks run in waves of the SM
  // count: pick the chunk count whose last wave is fullest, charging every further wave for the
  // CTAs' fixed part (set-up, pipeline fill, epilogue).  Every chunk is a whole number of pipeline
  // slabs (no chunk reads into the next) of at least kMinChunk elements; at most four waves.
  auto score = [&](int64_t ctas) {
    const int64_t waves = (ctas + kAssumedSms - 1) / kAssumedSms;
    return static_cast<double>(ctas) / static_cast<double>(waves * kAssumedSms) - 0.04 * static_cast<double>(waves - 1);
  };
  int best = 1;
  double best_score = score(tiles);
  for (int s = 2; s <= 16; ++s) {
    if (K % (static_cast<int64_t>(s) * kSlabElems16) != 0 || K / s < kMinChunk) continue;
    const int64_t ctas = tiles * s;
    if ((ctas + kAssumedSms - 1) / kAssumedSms > 4) continue;
    if (score(ctas) >= best_score - 1e-9) {
      best = s;
      best_score = score(ctas);
    }
  }
  return best;
}

// Problems whose tiles leave half of the SMs or more without work.  An estimate of both ways; cut where that is a tenth
// shorter.  Whole -> cut, us: bf16 300 x 512 x 8192 31.7 -> 13.6, 500 x 512 x 16384 60 -> 19, 2000 x 256 x 8192 32 -> 18,
// 900 x 304 x 16000 59 -> 21; fp8 250 x 512 x 16384 72 -> 18.
int tiled_splits(int64_t M, int64_t N, int64_t K, int64_t batch, int elem_bytes, size_t workspace_bytes) {
  const int64_t tiles = (M + 127) / 128 * ((N + 127) / 128), slabs = (K * elem_bytes + kSlabBytes - 1) / kSlabBytes;
  const int64_t plane = M * N * static_cast<int64_t>(sizeof(float));
  const int64_t splits = std::min<int64_t>({kAssumedSms / tiles, slabs / 8, 16, static_cast<int64_t>(workspace_bytes) / plane});
  if (batch != 1 || elem_bytes > 2 || splits < 2) return 1;
  // ns: a slab of a 128 x 64 tile (what the problem runs on unsplit) and of a 128 x 128 tile, the pass over the
  // partials and its launch
  const int64_t whole = slabs * kSlabNarrowNs, cut = (slabs + splits - 1) / splits * kSlabWideNs + kReduceNs + splits * plane / kReduceBytesPerNs;
  if (cut * 10 > whole * 9) return 1;
  const int64_t chunk = (slabs + splits - 1) / splits;
  return static_cast<int>((slabs + chunk - 1) / chunk);
}

size_t split_k_workspace_bytes(int64_t M, int64_t N, int splits) {
  return splits <= 1 ? 0 : static_cast<size_t>(splits) * M * N * sizeof(float);
}

int launch_split_k(const Problem& p, int splits, void* workspace, const DeviceInfo& dev, cudaStream_t stream, bool geglu) {
  const int slab = kSlabBytes / (p.kind == kKindF16 ? 2 : 1);
  const int slabs = static_cast<int>((p.K + slab - 1) / slab);
  Problem part = p;
  part.batch = splits;
  part.k_chunk = (slabs + splits - 1) / splits;
  part.c = nullptr;
  part.bias = nullptr;
  part.beta = 0.0f;
  part.act = kActNone;
  part.d = workspace;
  part.out_dtype = IXK_F32;
  part.ldd = p.N;
  part.d_batch_stride = p.M * p.N;
  part.force_block_n = 128;
  int rc = stream_applies(p) ? launch_stream(p, splits, static_cast<float*>(workspace), dev, stream) : launch(part, dev, stream);
  if (rc != IXK_OK) return rc;

  ReduceArgs r{};
  r.partial = static_cast<const float*>(workspace);
  r.splits = splits;
  r.M = static_cast<int>(p.M);
  r.N = static_cast<int>(p.N);
  r.bias = p.bias;
  r.c = p.beta != 0.0f ? p.c : nullptr;
  r.d = p.d;
  r.ldc = p.ldc;
  r.ldd = p.ldd;
  r.out_dtype = p.out_dtype;
  r.bias_dtype = p.bias_dtype;
  r.act = p.act;
  r.beta = p.beta;
  r.geglu = geglu ? 1 : 0;
  if (geglu) {
    const int64_t total = p.M * (p.N / 8);
    const ReduceGrid g = reduce_grid(total, dev.sm_count);
    auto* fn = splits == 1 ? splitk_reduce_geglu_kernel<1> : splits == 2 ? splitk_reduce_geglu_kernel<2>
             : splits <= 4 ? splitk_reduce_geglu_kernel<4> : splitk_reduce_geglu_kernel<8>;
    return launch_overlapped(fn, dim3(g.blocks), dim3(g.threads), 0, stream, r);
  }
  const bool vec = p.N % 4 == 0 && (reinterpret_cast<uintptr_t>(workspace) & 15u) == 0;
  const int64_t total = vec ? p.M * p.N / 4 : p.M * p.N;
  const ReduceGrid g = reduce_grid(total, dev.sm_count);
  auto* fn = !vec ? splitk_reduce_kernel<0> : splits == 2 ? splitk_reduce_kernel<2> : splits <= 4 ? splitk_reduce_kernel<4> : splitk_reduce_kernel<8>;
  return launch_overlapped(fn, dim3(g.blocks), dim3(g.threads), 0, stream, r);
}

}  // namespace gemm
}  // namespace ixk
