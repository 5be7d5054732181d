// A few float32 tokens by a float32 matrix: out[t, o] (+)= sum_k x[t, k] * w[o, k] in float32 multiply-adds.
//
// The stream of the weights is the bound, and with an output a thread (hx_gemm_simt.cu) two 16-byte reads of shared
// memory for four multiply-adds are far above it.  Here the lanes of a warp split the depth instead: a warp owns four
// features and every token of its tile, a lane four neighbouring k of each 128, so that a step takes 4 + TOKENS reads
// for 16 TOKENS multiply-adds, all side by side.  Two warps share four features' depth (128 k each of a stage of
// 256); lanes and then the two warps are summed in a fixed order that no size but the depth enters, so here, too, a
// value does not depend on the other rows of the call.  A CTA an SM goes through its tiles in one stream of stages,
// 100 KB and more of them on their way; a tile has as many features (up to 32) as let the last round fill.
//
// Measured (one B200, operands out of the L2, us, hx_gemm_simt.cu or hx_gemm_split.cu / here):
//   tokens                    1              4              8              16             32
//   [17,280 x 3,200]     69.6 / 51.2    77.8 / 54.0   114.7 / 56.1   120.8 / 78.8
//   [3,200 x 8,640]      98.3 / 28.7    98.3 / 30.8   130.1 / 33.8   131.1 / 44.0   150.5 / 83.0
//   [4,096 x 4,096]      50.3 / 20.5    51.2 / 22.6    65.5 / 22.6    65.6 / 29.6    80.7 / 49.2
//   [64 x 4,096]         49.2 / 14.3    49.2 / 16.4                   63.5 / 20.5
// One token is the stream (221 MB in 51 us with its launch, 4.3 TB/s); at 16 the reads of shared memory and the
// multiply-adds are each about the stream's time.  With divisions for each stage's addresses 16 tokens by
// [17,280 x 3,200] took 92.0 us; a CTA a tile, three stages and two CTAs an SM, one token by [3,200 x 8,640] 37.6.
// Errors against 64 bits (rms, relative) 1.0e-6 -> 1.4e-7 at a depth of 3,200, 1.7e-6 -> 2.2e-7 at 8,640.
#include "hx_mma.cuh"

#include <algorithm>
#include <mutex>

namespace {

enum Epilogue : int { EPI_STORE = 0, EPI_STORE_F32 = 1, EPI_ADD_F32 = 2 };

struct FewArgs {
  const float* x;
  int ldx;
  const float* w;
  int ldw;
  float* out;
  int ldo, tokens, features, depth;
  float softcap;
  int rows, token_tiles, tiles;      // features of a tile (a multiple of four, FEW_ROWS at most); tiles in all
};

constexpr int FEW_DEPTH = 256, FEW_ROWS = 32, FEW_THREADS = 512, FEW_WARP_ROWS = 4, FEW_SLICES = 2;

template <int TOKENS>
struct FewConfig {
  static constexpr int kStageFloats = (TOKENS + FEW_ROWS) * FEW_DEPTH;
  static constexpr int kStages = TOKENS <= 4 ? 6 : TOKENS <= 8 ? 5 : 4;
  static constexpr int kSums = FEW_SLICES * TOKENS * FEW_ROWS;
  static constexpr int kBytes = (kStages * kStageFloats + kSums) * 4;
  static_assert(kBytes <= 227 * 1024 && TOKENS * FEW_ROWS <= FEW_THREADS, "shared memory, and an output a thread");
};

// Sums over the lanes of a warp of V values each: while there are several, each half of the lanes keeps half of them.
template <int V, int APART>
__device__ __forceinline__ void sum_lanes(float* acc, int lane) {
  if constexpr (V > 1) {
    const bool upper = (lane & APART) != 0;
#pragma unroll
    for (int i = 0; i < V / 2; ++i) {
      const float send = upper ? acc[i] : acc[i + V / 2], keep = upper ? acc[i + V / 2] : acc[i];
      acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, APART);
    }
  } else {
    acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], APART);
  }
  if constexpr (APART > 1) sum_lanes<(V > 1 ? V / 2 : 1), APART / 2>(acc, lane);
}

template <int TOKENS, int EPI>
__global__ __launch_bounds__(FEW_THREADS, 1) void gemm_few_kernel(const FewArgs a) {
  using Config = FewConfig<TOKENS>;
  constexpr int kPieces = FEW_DEPTH / 4, kStages = Config::kStages, R = FEW_WARP_ROWS;
  extern __shared__ float4 few_stages[];
  float* stages = reinterpret_cast<float*>(few_stages);
  hx_pdl_prologue();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int slice = warp % FEW_SLICES, row0 = warp / FEW_SLICES * R;
  const int steps = (a.depth + FEW_DEPTH - 1) / FEW_DEPTH;
  float* sums = stages + kStages * Config::kStageFloats;      // [slice][token][feature of the tile]

  // a stage: the tile's weight rows, then its tokens, FEW_DEPTH values of each; zeros where there is no row or no k
  const int piece = threadIdx.x % kPieces, first = threadIdx.x / kPieces;
  constexpr int kApart = FEW_THREADS / kPieces;      // rows between a thread's
  const uint32_t fill_to = hx_shared_address(stages + first * FEW_DEPTH + 4 * piece);
  int fill_tile = blockIdx.x, fill_k = 4 * piece, fill_stage = 0;
  const float *fill_w = nullptr, *fill_x = nullptr;      // the thread's first row of each, at fill_k
  int fill_features = 0, fill_tokens = 0;                // rows from there on that are the tile's
  auto fill_from = [&] {
    const int token0 = fill_tile % a.token_tiles * TOKENS + first, feature0 = fill_tile / a.token_tiles * a.rows;
    fill_k = 4 * piece;
    fill_w = a.w + static_cast<size_t>(feature0 + first) * a.ldw + fill_k;
    fill_x = a.x + static_cast<size_t>(token0) * a.ldx + fill_k;
    fill_features = min(a.rows, a.features - feature0) - first;
    fill_tokens = a.tokens - token0;
  };
  if (fill_tile < a.tiles) fill_from();
  auto fill = [&] {
    if (fill_tile < a.tiles) {
      const uint32_t to = fill_to + fill_stage * (Config::kStageFloats * 4);
      const int live = max(0, min(4, a.depth - fill_k)) * 4;
#pragma unroll
      for (int i = 0; i < FEW_ROWS / kApart; ++i) {
        const bool there = live > 0 && i * kApart < fill_features;
        hx_cp_async_16(to + i * kApart * FEW_DEPTH * 4, there ? fill_w + static_cast<size_t>(i * kApart) * a.ldw : a.w,
                       there ? live : 0);
      }
#pragma unroll
      for (int i = 0; i < (TOKENS + kApart - 1) / kApart; ++i) {
        const bool there = live > 0 && i * kApart < fill_tokens;
        if (TOKENS >= kApart || first < TOKENS)
          hx_cp_async_16(to + (FEW_ROWS + i * kApart) * FEW_DEPTH * 4,
                         there ? fill_x + static_cast<size_t>(i * kApart) * a.ldx : a.x, there ? live : 0);
      }
      fill_stage = fill_stage + 1 == kStages ? 0 : fill_stage + 1;
      fill_k += FEW_DEPTH;
      fill_w += FEW_DEPTH;
      fill_x += FEW_DEPTH;
      if (fill_k - 4 * piece >= a.depth) {
        fill_tile += gridDim.x;
        if (fill_tile < a.tiles) fill_from();
      }
    }
    hx_cp_async_commit();      // an empty group keeps the count
  };

#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) fill();
  int at = 0;
  for (int tile = blockIdx.x; tile < a.tiles; tile += gridDim.x) {
    float acc[TOKENS * R];
#pragma unroll
    for (int i = 0; i < TOKENS * R; ++i) acc[i] = 0.0f;
    for (int step = 0; step < steps; ++step) {
      hx_cp_async_wait<kStages - 2>();
      __syncthreads();      // this step's rows are there, and the last step's stage is free
      fill();
      const float* stage = stages + at * Config::kStageFloats + slice * 128 + 4 * lane;
      at = at + 1 == kStages ? 0 : at + 1;
      if (row0 < a.rows) {
        float4 b[R];
#pragma unroll
        for (int j = 0; j < R; ++j) b[j] = *reinterpret_cast<const float4*>(stage + (row0 + j) * FEW_DEPTH);
#pragma unroll
        for (int t = 0; t < TOKENS; ++t) {
          const float4 v = *reinterpret_cast<const float4*>(stage + (FEW_ROWS + t) * FEW_DEPTH);
#pragma unroll
          for (int j = 0; j < R; ++j) acc[t * R + j] = fmaf(v.x, b[j].x, acc[t * R + j]);
#pragma unroll
          for (int j = 0; j < R; ++j) acc[t * R + j] = fmaf(v.y, b[j].y, acc[t * R + j]);
#pragma unroll
          for (int j = 0; j < R; ++j) acc[t * R + j] = fmaf(v.z, b[j].z, acc[t * R + j]);
#pragma unroll
          for (int j = 0; j < R; ++j) acc[t * R + j] = fmaf(v.w, b[j].w, acc[t * R + j]);
        }
      }
    }

    constexpr int V = TOKENS * R;
    constexpr int kHeld = V >= 32 ? V / 32 : 1, kLanes = V / kHeld;      // values a lane holds, lanes that differ
    sum_lanes<V, 16>(acc, lane);
    if (lane % (32 / kLanes) == 0) {
#pragma unroll
      for (int i = 0; i < kHeld; ++i) {
        const int value = lane / (32 / kLanes) * kHeld + i;
        sums[(slice * TOKENS + value / R) * FEW_ROWS + row0 + value % R] = acc[i];
      }
    }
    __syncthreads();      // (and one more comes before the next tile's sums are written)
    const int row = threadIdx.x % FEW_ROWS;
    const int token = tile % a.token_tiles * TOKENS + threadIdx.x / FEW_ROWS;
    const int feature = tile / a.token_tiles * a.rows + row;
    if (threadIdx.x < TOKENS * FEW_ROWS && row < a.rows && token < a.tokens && feature < a.features) {
      const float sum = sums[threadIdx.x] + sums[TOKENS * FEW_ROWS + threadIdx.x];
      float* out = a.out + static_cast<size_t>(token) * a.ldo + feature;
      if (EPI == EPI_ADD_F32) {
        *out += sum;
      } else {
        *out = a.softcap > 0.0f ? a.softcap * tanhf(sum / a.softcap) : sum;
      }
    }
  }
}

template <int TOKENS, int EPI>
int launch_few(FewArgs a, cudaStream_t stream) {
  constexpr int kBytes = FewConfig<TOKENS>::kBytes;
  static std::once_flag once;
  static cudaError_t configured = cudaSuccess;
  std::call_once(once, [] {
    configured = cudaFuncSetAttribute(gemm_few_kernel<TOKENS, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes);
    if (configured != cudaSuccess) cudaGetLastError();
  });
  if (configured != cudaSuccess) {
    hx_set_error("hx_gemm_few: cannot reserve %d bytes of shared memory", kBytes);
    return HX_ERR_LAUNCH;
  }
  const int sms = hx_device_sm_count();
  if (sms <= 0) return HX_ERR_LAUNCH;
  a.token_tiles = (a.tokens + TOKENS - 1) / TOKENS;
  const long long rows = static_cast<long long>(a.token_tiles) * a.features;
  const long long rounds = (rows + FEW_ROWS * sms - 1) / (FEW_ROWS * sms);
  a.rows = std::min<long long>(FEW_ROWS, (rows + rounds * sms * 4 - 1) / (rounds * sms * 4) * 4);
  a.tiles = (a.features + a.rows - 1) / a.rows * a.token_tiles;
  hx_launch(gemm_few_kernel<TOKENS, EPI>, dim3(std::min(a.tiles, sms)), FEW_THREADS, kBytes, stream, a);
  return HX_OK;
}

template <int EPI>
int launch_tokens(const FewArgs& a, cudaStream_t stream) {
  if (a.tokens == 1) return launch_few<1, EPI>(a, stream);
  if (a.tokens == 2) return launch_few<2, EPI>(a, stream);
  if (a.tokens <= 4) return launch_few<4, EPI>(a, stream);
  if (a.tokens <= 8) return launch_few<8, EPI>(a, stream);
  return launch_few<16, EPI>(a, stream);
}

}  // namespace

// Whether the product runs here, and is the faster road: every 16 tokens read and multiply all weights again, so
// behind 16 tokens only while the tiles are few rounds of the SMs.  Measured (us, tensor cores / here): 9,600 features of
// 3,200 with 32 tokens, 5 rounds, 111 / 94, 48, 7 rounds, 111 / 129; 17,280 with 17, 8 rounds, 120 / 150; 4,096 of 4,096 with
// 48, 3 rounds, 81 / 72, 64, 4 rounds, 81 / 92; 3,200 of 8,640 with 64, 3 rounds, 150 / 137; 1,024 of 4,096 with 128, 2
// rounds, 77 / 50.  A depth below a stage is mostly zeros here (9,000 of 128 with 16 tokens 10 / 12).  The line at 128 tokens is
// only where the measurements end: 16 of 2,048 take 7.2 us with 128 tokens and, as one chain, 58 with 129.
HX_API int hx_gemm_few_takes(const void* x, int ldx, const void* w, int ldw, int tokens, int features, int depth) {
  if (tokens <= 0 || tokens > 128 || features <= 0 || depth < FEW_DEPTH || ldx % 4 != 0 || ldw % 4 != 0 ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) != 0)
    return 0;
  const long long rows = static_cast<long long>((tokens + 15) / 16) * features;
  const long long round = static_cast<long long>(FEW_ROWS) * hx_device_sm_count();
  return tokens <= 16 || rows <= 3 * round || (tokens <= 32 && rows <= 5 * round);
}

// float32 x [tokens, ldx], w [features, ldw], out [tokens, ldo]; epilogues and softcap as hx_gemm_simt_softcapped.
HX_API int hx_gemm_few(const float* x, int ldx, const float* w, int ldw, float* out, int ldo, int tokens, int features,
                       int depth, int epilogue, float softcap, cudaStream_t stream) {
  HX_REQUIRE(tokens > 0 && features > 0 && depth > 0, "hx_gemm_few: bad sizes");
  HX_REQUIRE(softcap >= 0.0f && (softcap == 0.0f || epilogue == EPI_STORE_F32),
             "hx_gemm_few: a softcap belongs to a float32 store");
  HX_REQUIRE(ldx >= depth && ldw >= depth && ldo >= features, "hx_gemm_few: bad strides");
  HX_REQUIRE(hx_gemm_few_takes(x, ldx, w, ldw, tokens, features, depth),
             "hx_gemm_few: %d tokens by %d features of %d in rows of %d and %d are not supported", tokens, features, depth, ldx,
             ldw);
  const FewArgs a{x, ldx, w, ldw, out, ldo, tokens, features, depth, softcap, 0, 0, 0};
  int rc;
  switch (epilogue) {
    case EPI_STORE:      // (the storage type is float32)
    case EPI_STORE_F32: rc = launch_tokens<EPI_STORE_F32>(a, stream); break;
    case EPI_ADD_F32: rc = launch_tokens<EPI_ADD_F32>(a, stream); break;
    default: HX_REQUIRE(false, "hx_gemm_few: unknown epilogue %d", epilogue); return HX_ERR_ARGUMENT;
  }
  if (rc != HX_OK) return rc;
  HX_CHECK_LAUNCH("hx_gemm_few");
  return HX_OK;
}
