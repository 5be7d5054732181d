// Matrix product on the CUDA cores: out[t, o] (+)= sum_k x[t, k] * w[o, k].
//
// This is the true 32-bit path (float32 storage, float32 fused multiply-adds, no
// reduced-precision matrix mode; few tokens take hx_gemm_few.cu and many hx_gemm_split.cu, whose sums are
// closer still) and also the bfloat16 path for shapes the tensor
// core kernel refuses.  Each output element is one sequential sum over k in
// ascending order, so in this kernel its value never depends on how many rows the call has or
// on which tile it falls into (a product that one of those two takes for its number of rows is
// another order of the same sums).  The reference's counterpart is its 16x16 tiled kernel
// (src/kernels/cuda/matmul.cu:36-71).
//
// Prompt portions are bound by the multiply-adds and by the 16-byte loads from shared memory
// that feed them, a few tokens by the stream of the weights.  Both operands keep their rows in
// shared memory, filled by cp.async several stages ahead (bfloat16 rows are converted on the
// way through registers); a thread owns RM x RN outputs whose rows lie (TM / RM) and (TN / RN)
// apart, so the lanes of a quarter warp read rows side by side, which a row stride of BK + 4
// floats puts on different banks, four k at a time.
//
// Measured (one B200, float32, alone): 512 tokens by [17,280 x 3,200] 2,243 -> 1,573 us (36
// TFLOP/s), by [3,200 x 8,640] 2,287 -> 1,071 us, by [4,096 x 4,096] 1,262 -> 512 us; one token
// by the same 667 -> 68 us (3.2 TB/s of weights), 770 -> 100 us, 296 -> 52 us (a few float32 tokens of
// a depth from 256 on whose rows begin on 16 bytes are hx_gemm_few.cu's: 51, 29 and 21 us).
#include "hx_mma.cuh"

#include <mutex>

namespace {

enum Epilogue : int { EPI_STORE = 0, EPI_STORE_F32 = 1, EPI_ADD_F32 = 2 };

struct SimtArgs {
  const void* x;
  int ldx;
  const void* w;
  int ldw;
  void* out;
  int ldo, tokens, features, depth;
  float softcap;
};

// TM tokens x TN features a CTA, RM x RN of them a thread, BK of the depth a stage; CTAS of an
// SM bound the registers.
template <int TM_, int TN_, int RM_, int RN_, int BK_, int STAGES_, int CTAS_>
struct SimtTile {
  static constexpr int TM = TM_, TN = TN_, RM = RM_, RN = RN_, BK = BK_, STAGES = STAGES_;
  static constexpr int kCtas = CTAS_;
  static constexpr int kThreads = (TM / RM) * (TN / RN);
  static constexpr int kStride = BK + 4;
  static constexpr int kStageFloats = (TM + TN) * kStride;
  static constexpr int kBytes = STAGES * kStageFloats * 4;
};

__device__ __forceinline__ void simt_copy_4(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes)
               : "memory");
}

// ROWS rows of BK values from column k0 on into a stage, zeros where there is no row or no k.
template <typename T, typename Tile, int ROWS>
__device__ __forceinline__ void stage_rows(float* dst, const T* src, int ld, int row0, int rows,
                                           int k0, int depth, bool wide) {
  constexpr int kPieces = Tile::BK / 4;
#pragma unroll
  for (int e = threadIdx.x; e < ROWS * kPieces; e += Tile::kThreads) {
    const int row = e / kPieces, k = k0 + (e - row * kPieces) * 4;
    float* to = dst + row * Tile::kStride + (e - row * kPieces) * 4;
    const bool there = row0 + row < rows;
    const T* from = src + static_cast<size_t>(there ? row0 + row : 0) * ld;
    const int live = there ? max(0, min(4, depth - k)) : 0;
    if constexpr (sizeof(T) == 4) {
      if (wide) {      // rows begin on 16 bytes; the last piece may end inside its own
        hx_cp_async_16(hx_shared_address(to), live > 0 ? from + k : from, live * 4);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          simt_copy_4(hx_shared_address(to + i), i < live ? from + k + i : from, i < live ? 4 : 0);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) to[i] = i < live ? hx_to_float<T>(from[k + i]) : 0.0f;
    }
  }
}

template <typename T, typename Tile, int EPI>
__global__ __launch_bounds__(Tile::kThreads, Tile::kCtas) void gemm_simt_kernel(const SimtArgs a) {
  constexpr int TM = Tile::TM, TN = Tile::TN, RM = Tile::RM, RN = Tile::RN, BK = Tile::BK;
  constexpr int kTokenStep = TM / RM, kFeatureStep = TN / RN;
  extern __shared__ float4 simt_stages[];
  float* stages = reinterpret_cast<float*>(simt_stages);
  hx_pdl_prologue();
  const T* x = static_cast<const T*>(a.x);
  const T* w = static_cast<const T*>(a.w);
  const int token0 = blockIdx.y * TM, feature0 = blockIdx.x * TN;
  const int tx = threadIdx.x % kFeatureStep, ty = threadIdx.x / kFeatureStep;
  const bool wide_x = a.ldx % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  const bool wide_w = a.ldw % 4 == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0;
  const int steps = (a.depth + BK - 1) / BK;

  auto fill = [&](int step) {
    if (step < steps) {
      float* stage = stages + (step % Tile::STAGES) * Tile::kStageFloats;
      stage_rows<T, Tile, TM>(stage, x, a.ldx, token0, a.tokens, step * BK, a.depth, wide_x);
      stage_rows<T, Tile, TN>(stage + TM * Tile::kStride, w, a.ldw, feature0, a.features, step * BK,
                              a.depth, wide_w);
    }
    hx_cp_async_commit();      // an empty group keeps the count
  };

  float acc[RM][RN];
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < RN; ++j) acc[i][j] = 0.0f;
#pragma unroll
  for (int s = 0; s < Tile::STAGES - 1; ++s) fill(s);
  for (int step = 0; step < steps; ++step) {
    hx_cp_async_wait<Tile::STAGES - 2>();
    __syncthreads();      // this step's rows are there, and the last step's stage is free
    fill(step + Tile::STAGES - 1);
    const float* stage = stages + (step % Tile::STAGES) * Tile::kStageFloats;
    const float* xs = stage + ty * Tile::kStride;
    const float* ws = stage + (TM + tx) * Tile::kStride;
#pragma unroll 2
    for (int k = 0; k < BK; k += 4) {
      float4 b[RN];
#pragma unroll
      for (int j = 0; j < RN; ++j)
        b[j] = *reinterpret_cast<const float4*>(ws + j * kFeatureStep * Tile::kStride + k);
#pragma unroll
      for (int i = 0; i < RM; ++i) {
        const float4 v = *reinterpret_cast<const float4*>(xs + i * kTokenStep * Tile::kStride + k);
#pragma unroll
        for (int j = 0; j < RN; ++j) acc[i][j] = fmaf(v.x, b[j].x, acc[i][j]);
#pragma unroll
        for (int j = 0; j < RN; ++j) acc[i][j] = fmaf(v.y, b[j].y, acc[i][j]);
#pragma unroll
        for (int j = 0; j < RN; ++j) acc[i][j] = fmaf(v.z, b[j].z, acc[i][j]);
#pragma unroll
        for (int j = 0; j < RN; ++j) acc[i][j] = fmaf(v.w, b[j].w, acc[i][j]);
      }
    }
  }

#pragma unroll
  for (int i = 0; i < RM; ++i) {
    const int token = token0 + ty + i * kTokenStep;
    if (token >= a.tokens) continue;
#pragma unroll
    for (int j = 0; j < RN; ++j) {
      const int feature = feature0 + tx + j * kFeatureStep;
      if (feature >= a.features) continue;
      const size_t index = static_cast<size_t>(token) * a.ldo + feature;
      if (EPI == EPI_STORE) {
        static_cast<T*>(a.out)[index] = hx_from_float<T>(acc[i][j]);
      } else if (EPI == EPI_STORE_F32) {
        static_cast<float*>(a.out)[index] =
            a.softcap > 0.0f ? a.softcap * tanhf(acc[i][j] / a.softcap) : acc[i][j];
      } else {
        static_cast<float*>(a.out)[index] += acc[i][j];
      }
    }
  }
}

template <typename T, typename Tile, int EPI>
int launch_tile(const SimtArgs& a, cudaStream_t stream) {
  static std::once_flag once;
  static cudaError_t configured = cudaSuccess;
  std::call_once(once, [] {
    configured = cudaFuncSetAttribute(gemm_simt_kernel<T, Tile, EPI>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, Tile::kBytes);
    if (configured != cudaSuccess) cudaGetLastError();
  });
  if (configured != cudaSuccess) {
    hx_set_error("hx_gemm_simt: cannot reserve %d bytes of shared memory", Tile::kBytes);
    return HX_ERR_LAUNCH;
  }
  const dim3 grid((a.features + Tile::TN - 1) / Tile::TN, (a.tokens + Tile::TM - 1) / Tile::TM);
  hx_launch(gemm_simt_kernel<T, Tile, EPI>, grid, Tile::kThreads, Tile::kBytes, stream, a);
  return HX_OK;
}

using WideTile = SimtTile<128, 128, 8, 8, 16, 4, 2>;
using MiddleTile = SimtTile<64, 64, 4, 8, 16, 4, 4>;
using SmallTile = SimtTile<32, 32, 4, 4, 32, 4, 6>;
using FewTile = SimtTile<16, 16, 2, 2, 32, 6, 7>;        // up to 16 tokens: a stream of the weights
using SingleTile = SimtTile<4, 16, 1, 1, 32, 8, 8>;      // up to 4 tokens

// The widest tile that the tokens fill and that still gives every SM a CTA: smaller tiles read
// their operands more often but leave fewer SMs without work.  512 tokens by [3,200 x 8,640], 100
// tiles of 128 or 400 of 64: 1,766 against 1,071 us; by [17,280 x 3,200], 540 tiles of 128: 36
// TFLOP/s, where tiles of 64 reach 26 to 33.
template <typename T, int EPI>
int launch_epilogue(const SimtArgs& a, int sms, cudaStream_t stream) {
  auto ctas = [&](int tm, int tn) {
    return static_cast<long long>((a.tokens + tm - 1) / tm) * ((a.features + tn - 1) / tn);
  };
  if (a.tokens <= 4) return launch_tile<T, SingleTile, EPI>(a, stream);
  if (a.tokens <= 16) return launch_tile<T, FewTile, EPI>(a, stream);
  if constexpr (sizeof(T) == 4) {
    if (a.tokens > 64 && ctas(128, 128) >= sms) return launch_tile<T, WideTile, EPI>(a, stream);
  }
  if (a.tokens > 32 && ctas(64, 64) >= sms) return launch_tile<T, MiddleTile, EPI>(a, stream);
  return launch_tile<T, SmallTile, EPI>(a, stream);
}

template <typename T>
int launch(const SimtArgs& a, int epilogue, cudaStream_t stream) {
  const int sms = hx_device_sm_count();
  if (sms <= 0) return HX_ERR_LAUNCH;
  switch (epilogue) {
    case EPI_STORE: return launch_epilogue<T, EPI_STORE>(a, sms, stream);
    case EPI_STORE_F32: return launch_epilogue<T, EPI_STORE_F32>(a, sms, stream);
    case EPI_ADD_F32: return launch_epilogue<T, EPI_ADD_F32>(a, sms, stream);
    default:
      hx_set_error("hx_gemm_simt: unknown epilogue %d", epilogue);
      return HX_ERR_ARGUMENT;
  }
}

}  // namespace

// epilogue 0: out (compute dtype) = x w^T; 1: out (float32) = x w^T; 2: out (float32) += x w^T
// softcap > 0 (epilogue 1 only): the sums run into a level, softcap * tanh(x w^T / softcap)
HX_API int hx_gemm_simt_softcapped(const void* x, int ldx, const void* w, int ldw, void* out,
                                   int ldo, int dtype, int tokens, int features, int depth,
                                   int epilogue, float softcap, cudaStream_t stream) {
  HX_REQUIRE(softcap >= 0.0f && (softcap == 0.0f || epilogue == EPI_STORE_F32),
             "hx_gemm_simt: a softcap belongs to a float32 store");
  HX_REQUIRE(tokens >= 0 && features > 0 && depth > 0, "hx_gemm_simt: bad sizes");
  HX_REQUIRE(ldx >= depth && ldw >= depth && ldo >= features, "hx_gemm_simt: bad strides");
  // (tiles of fewer than 64 tokens are for products with fewer tiles of 64 than SMs)
  HX_REQUIRE((tokens + 63) / 64 <= 65535, "hx_gemm_simt: too many rows (%d)", tokens);
  if (tokens == 0) return HX_OK;
  const SimtArgs a{x, ldx, w, ldw, out, ldo, tokens, features, depth, softcap};
  int rc;
  if (dtype == HX_F32) {
    rc = launch<float>(a, epilogue, stream);
  } else if (dtype == HX_BF16) {
    rc = launch<__nv_bfloat16>(a, epilogue, stream);
  } else {
    HX_REQUIRE(false, "hx_gemm_simt: unknown dtype %d", dtype);
  }
  if (rc != HX_OK) return rc;
  HX_CHECK_LAUNCH("hx_gemm_simt");
  return HX_OK;
}

HX_API int hx_gemm_simt(const void* x, int ldx, const void* w, int ldw, void* out, int ldo,
                        int dtype, int tokens, int features, int depth, int epilogue,
                        cudaStream_t stream) {
  return hx_gemm_simt_softcapped(x, ldx, w, ldw, out, ldo, dtype, tokens, features, depth, epilogue,
                                 0.0f, stream);
}
