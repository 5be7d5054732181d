// float32 products of many tokens on the tensor cores: out[t, o] (+)= sum_k x[t, k] * w[o, k].
//
// Every operand goes in as three bfloat16 terms, 2^16 x = x0 + x1 + x2, each the nearest to what the ones
// before it leave: 24 bits, all that a float32 holds.  (Times 2^16 because bfloat16 ends at 2^-133: the last
// bit of every float32, 2^-149 at least, is then one of a term.  Blocks of sums are divided by 2^32 as they
// are added.)  Of the nine products the three below 2^-25 of the
// whole (x1 w2, x2 w1, x2 w2) are left out.  The tensor cores add in float32 but do not round to nearest,
// so a sum stays in tensor memory for one block of 64 k only, the products of the small terms first, and
// the blocks are added in registers.  The sums are closer to those of 64 bits than a chain of float32
// multiply-adds is: measured, relative 2-norm, here and the chain, normal operands: depth 64 7.7e-8 and 1.4e-7,
// 256 8.8e-8 and 2.9e-7, 3,200 1.5e-7 and 1.0e-6, 8,640 2.2e-7 and 1.7e-6; positive operands alike.  (Where a few
// products are the whole sum, operands e^(4 n): 1.8e-8 and 1.7e-8, 1.3e-7 and 1.1e-7 at the last two.)
//
// A sum that is not finite (an operand is not, or 2^16 times it leaves float32, or 2^32 times a block's
// sum does: operands from 2^112 and sums from 2^96 on) is taken again as that chain, which says what it is.
//
// What bounds it: the conversion.  A block of 64 k of a tile of 128 x 128 takes about 4,000 cycles; with one
// of the six products it takes as long, without the loads 3,300 (ncu: issue slots 54 % busy, tensor pipe 38 %):
// eight warps that load, cut and store 16 pieces of four numbers each a block, two warps a scheduler.
// Slower: sixteen such warps (too few registers for loads in flight: 463 -> 502 us), all warps converting
// and summing in turn (539), the weights' lines asked for ahead (4 % faster alone, 3 % slower in place).
// Measured (us, tiles of multiply-adds before): 512 tokens by [17,280 x 3,200] 1,581 -> 434, by [3,200 x 8,640] 947 ->
// 287, by [4,096 x 4,096] 522 -> 157; 33 by the first 248 -> 117.  (With the next block's tokens asked for in front
// of the proxy fence, which waits for loads too: 459 and 311.)
//
// Every wait on an mbarrier is bounded; a wait that runs out sets a status bit, the CTA skips its
// remaining work, frees its tensor memory and returns.
#include "hx_tcgen05.cuh"

#include <cfloat>
#include <mutex>

namespace {

enum Epilogue : int { EPI_STORE = 0, EPI_STORE_F32 = 1, EPI_ADD_F32 = 2 };

constexpr int TILE = 128;           // tokens and features of a CTA
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int TERM_BYTES = TILE * BK * 2;
constexpr int STAGE_BYTES = 6 * TERM_BYTES;      // x0 x1 x2 w0 w1 w2
constexpr int STAGES = 2;
constexpr int SUM_WARPS = 8;        // two for each quarter of the tile's tokens, half of the features each
constexpr int COPY_WARPS = 8;
constexpr int THREADS = 32 * (SUM_WARPS + COPY_WARPS);
constexpr int COPY_THREADS = 32 * COPY_WARPS;
constexpr int PASS_ROWS = COPY_THREADS / (BK / 4);      // rows that the copying threads take at a time
constexpr int PASSES = TILE / PASS_ROWS;
constexpr int COLUMNS = TILE / 2;   // of a summing thread
// A thread's registers: 128 at launch, of which the summing warps need fewer and the others, with 64
// loaded numbers on their way, more.
constexpr int SUM_REGISTERS = 104, COPY_REGISTERS = 152;
static_assert(SUM_WARPS * SUM_REGISTERS + COPY_WARPS * COPY_REGISTERS <= 128 * (SUM_WARPS + COPY_WARPS),
              "what one side takes the other has given back");
constexpr int TMEM_COLUMNS = 2 * TILE;
constexpr float OPERAND_SCALE = 65536.0f, SUM_SCALE = 1.0f / (OPERAND_SCALE * OPERAND_SCALE);
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*alignment*/ + 256 /*barriers*/;

struct SplitArgs {
  const float* x;
  int ldx;
  const float* w;
  int ldw;
  float* out;
  int ldo, tokens, features, depth;
  float softcap;
  int* status;
};

__device__ __forceinline__ uint32_t two_terms(float a, float b) {
  uint32_t packed;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(packed) : "f"(b), "f"(a));
  return packed;
}
// What two packed terms leave of a and b.
__device__ __forceinline__ void leave(uint32_t terms, float& a, float& b) {
  a -= __uint_as_float(terms << 16);
  b -= __uint_as_float(terms & 0xffff0000u);
}

// The terms of four numbers, 8 bytes each, to `at` in the three matrices of terms.
__device__ __forceinline__ void store_terms(uint8_t* at, float4 v) {
  asm("{\n\t.reg .b64 s, p, q;\n\t"
      "mov.b64 s, {%4, %4};\n\tmov.b64 p, {%0, %1};\n\tmov.b64 q, {%2, %3};\n\t"
      "mul.rn.f32x2 p, p, s;\n\tmul.rn.f32x2 q, q, s;\n\t"
      "mov.b64 {%0, %1}, p;\n\tmov.b64 {%2, %3}, q;\n\t}"
      : "+f"(v.x), "+f"(v.y), "+f"(v.z), "+f"(v.w)
      : "f"(OPERAND_SCALE));
#pragma unroll
  for (int term = 0; term < 3; ++term) {
    const uint2 packed = make_uint2(two_terms(v.x, v.y), two_terms(v.z, v.w));
    *reinterpret_cast<uint2*>(at + term * TERM_BYTES) = packed;
    leave(packed.x, v.x, v.y);
    leave(packed.y, v.z, v.w);
  }
}

// The sum as a chain of float32 multiply-adds.
__device__ __noinline__ float chained_sum(const float* x, const float* w, int depth) {
  float sum = 0.0f;
  for (int k = 0; k < depth && !isnan(sum); ++k) sum = fmaf(x[k], w[k], sum);
  return sum;
}

template <int EPI>
__global__ __launch_bounds__(THREADS, 1) void gemm_split_kernel(const SplitArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* sum_full_bar = empty_bar + STAGES;      // [2]
  uint64_t* sum_empty_bar = sum_full_bar + 2;       // [2]
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(sum_empty_bar + 2);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int token0 = blockIdx.x * TILE, feature0 = blockIdx.y * TILE;
  const int blocks = (a.depth + BK - 1) / BK;
  hx_pdl_trigger();
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], COPY_WARPS);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sum_full_bar[b], 1);
      mbar_init(&sum_empty_bar[b], SUM_WARPS);
    }
    *failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(tmem_holder, TMEM_COLUMNS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  hx_pdl_wait();
  auto give_up = [&]() {
    atomicOr(a.status, HX_FLAG_WAIT_TIMEOUT);
    *failed = 1;
  };

  // The products of a block, by one thread.
  auto multiply = [&](int kb) {
    const int s = kb % STAGES, buffer = kb & 1;
    if (*failed || !mbar_wait(&sum_empty_bar[buffer], ((kb >> 1) & 1u) ^ 1u) ||
        !mbar_wait(&full_bar[s], (kb / STAGES) & 1u)) {
      give_up();
      return;
    }
    tc_fence_after();
    constexpr uint32_t idesc = make_idesc(TILE, TILE);
    const uint32_t stage = smem_u32(smem + s * STAGE_BYTES);
    const uint32_t sums = tmem_base + buffer * TILE;
    // term of x, term of w: the smallest products first
    constexpr int X[6] = {2, 0, 1, 1, 0, 0}, W[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const uint64_t desc_x = make_smem_desc(stage + X[i] * TERM_BYTES);
      const uint64_t desc_w = make_smem_desc(stage + (3 + W[i]) * TERM_BYTES);
#pragma unroll
      for (int k = 0; k < BK / UMMA_K; ++k) {
        const uint64_t step = static_cast<uint64_t>(k * UMMA_K * 2 >> 4);
        umma_bf16(sums, desc_x + step, desc_w + step, idesc, i > 0 || k > 0 ? 1u : 0u);
      }
    }
    umma_commit(&empty_bar[s]);
    umma_commit(&sum_full_bar[buffer]);
  };

  if (warp >= SUM_WARPS) {
    // ------------------------------------------- operands: loaded, cut into terms, stored swizzled
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(COPY_REGISTERS));
    const int thread = threadIdx.x - 32 * SUM_WARPS;
    const int piece = thread % (BK / 4), row0 = thread / (BK / 4);      // four k of rows row0 + PASS_ROWS p
    const float* x = a.x + static_cast<size_t>(token0) * a.ldx + 4 * piece;
    const float* w = a.w + static_cast<size_t>(feature0) * a.ldw + 4 * piece;
    const int x_rows = a.tokens - token0, w_rows = a.features - feature0;
    auto load = [&](float4 (&v)[PASSES], const float* from, int ld, int rows, int kb) {
      const bool inside = kb * BK + 4 * piece < a.depth;      // the depth is a multiple of four
#pragma unroll
      for (int p = 0; p < PASSES; ++p) {
        const int row = row0 + PASS_ROWS * p;
        v[p] = inside && row < rows
                   ? *reinterpret_cast<const float4*>(from + static_cast<size_t>(row) * ld + kb * BK)
                   : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
    };
    auto store = [&](uint8_t* terms, const float4 (&v)[PASSES]) {
#pragma unroll
      for (int p = 0; p < PASSES; ++p) {
        const int row = row0 + PASS_ROWS * p;
        store_terms(terms + row * (BK * 2) + (((piece >> 1) ^ (row & 7)) << 4) + ((piece & 1) << 3), v[p]);
      }
    };
    float4 xv[PASSES], wv[PASSES];
    load(xv, x, a.ldx, x_rows, 0);
    for (int kb = 0; kb < blocks && !*failed; ++kb) {
      const int s = kb % STAGES;
      load(wv, w, a.ldw, w_rows, kb);
      bool ok = true;
      if (lane == 0) ok = mbar_wait(&empty_bar[s], ((kb / STAGES) & 1u) ^ 1u);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) {
        if (lane == 0) give_up();
        break;
      }
      uint8_t* stage = smem + s * STAGE_BYTES;
      store(stage, xv);
      store(stage + 3 * TERM_BYTES, wv);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&full_bar[s]);
      // (not in front of the fence, which waits for loads too)
      if (kb + 1 < blocks) load(xv, x, a.ldx, x_rows, kb + 1);
    }
  } else {
    // ------------------------------------- products, sums of the blocks, and the epilogue
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(SUM_REGISTERS));
    const int quarter = warp & 3, half = warp >> 2;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + half * COLUMNS;
    float sum[COLUMNS];
#pragma unroll
    for (int j = 0; j < COLUMNS; ++j) sum[j] = 0.0f;
    bool ok = true;
    if (warp == 0) {
      if (hx_elect_one()) multiply(0);
      __syncwarp();
    }
    for (int kb = 0; kb < blocks; ++kb) {
      const int buffer = kb & 1;
      // the first warp has the next block multiplied while it waits for this one
      if (warp == 0 && kb + 1 < blocks) {
        if (hx_elect_one()) multiply(kb + 1);
        __syncwarp();
      }
      if (lane == 0) ok = !*failed && mbar_wait(&sum_full_bar[buffer], (kb >> 1) & 1u);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) {
        if (lane == 0) give_up();
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int column = 0; column < COLUMNS; column += 16) {
        float v[16];
        tmem_load16(lane_base + buffer * TILE + column, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) sum[column + j] = fmaf(v[j], SUM_SCALE, sum[column + j]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sum_empty_bar[buffer]);
    }
    const int token = token0 + quarter * 32 + lane, column0 = feature0 + half * COLUMNS;
    const int live = min(COLUMNS, a.features - column0);
    if (ok && token < a.tokens && live > 0) {
      float* out = a.out + static_cast<size_t>(token) * a.ldo + column0;
      const bool wide = a.ldo % 4 == 0 && (reinterpret_cast<uintptr_t>(a.out) & 15) == 0 && live == COLUMNS;
#pragma unroll
      for (int j = 0; j < COLUMNS; ++j)
        if (!(fabsf(sum[j]) <= FLT_MAX) && j < live)
          sum[j] = chained_sum(a.x + static_cast<size_t>(token) * a.ldx,
                               a.w + static_cast<size_t>(column0 + j) * a.ldw, a.depth);
      if (EPI == EPI_STORE_F32 && a.softcap > 0.0f) {
#pragma unroll
        for (int j = 0; j < COLUMNS; ++j) sum[j] = a.softcap * tanhf(sum[j] / a.softcap);
      }
      if (wide) {
#pragma unroll
        for (int j = 0; j < COLUMNS; j += 4) {
          float4 v = make_float4(sum[j], sum[j + 1], sum[j + 2], sum[j + 3]);
          if (EPI == EPI_ADD_F32) {
            const float4 old = *reinterpret_cast<const float4*>(out + j);
            v.x += old.x;
            v.y += old.y;
            v.z += old.z;
            v.w += old.w;
          }
          *reinterpret_cast<float4*>(out + j) = v;
        }
      } else {
#pragma unroll
        for (int j = 0; j < COLUMNS; ++j) {
          if (j < live) {
            if (EPI == EPI_ADD_F32) out[j] += sum[j];
            else out[j] = sum[j];
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLUMNS);
  }
}

template <int EPI>
int launch_split(const SplitArgs& a, cudaStream_t stream) {
  static std::once_flag once;
  static bool configured = false;
  std::call_once(once, [] {
    configured = cudaFuncSetAttribute(gemm_split_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      SMEM_BYTES) == cudaSuccess;
    if (!configured) cudaGetLastError();
  });
  if (!configured) {
    hx_set_error("hx_gemm_split: cannot reserve %d bytes of shared memory", SMEM_BYTES);
    return HX_ERR_LAUNCH;
  }
  const dim3 grid((a.tokens + TILE - 1) / TILE, (a.features + TILE - 1) / TILE);
  hx_launch(gemm_split_kernel<EPI>, grid, THREADS, SMEM_BYTES, stream, a);
  return HX_OK;
}

}  // namespace

// Whether the product runs here: rows of both operands begin on 16 bytes and hold a multiple of four.
HX_API int hx_gemm_split_supports(const void* x, int ldx, const void* w, int ldw, int features, int depth) {
  return depth > 0 && features > 0 && depth % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && (features + TILE - 1) / TILE <= 65535 &&
         ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
}

// Whether it is the faster road for this many tokens: with few tiles either road is one round of CTAs that
// walk the depth alone, 2.0 us a block of 64 k on the CUDA cores (32 x 32 a tile, several CTAs an SM) against
// 2.2 here, so the CUDA cores need more than two such tiles an SM to be slower.  Measured (us, CUDA cores / here):
// 9,600 features of 3,200 17 tokens 141 / 111; 4,096 of 4,096 64 tokens 131 / 143, 100 188 / 146; 3,200 of 8,640 64
// 266 / 289, 100 375 / 294.
HX_API int hx_gemm_split_pays(int tokens, int features) {
  const long long small = static_cast<long long>((tokens + 31) / 32) * ((features + 31) / 32);
  return tokens > 16 && small >= 2ll * hx_device_sm_count();
}

// float32 x [tokens, ldx], w [features, ldw], out [tokens, ldo]; epilogues and softcap as hx_gemm_simt_softcapped.
HX_API int hx_gemm_split(const float* x, int ldx, const float* w, int ldw, float* out, int ldo, int tokens,
                         int features, int depth, int epilogue, float softcap, int* status, cudaStream_t stream) {
  HX_REQUIRE(tokens >= 0 && features > 0 && depth > 0, "hx_gemm_split: bad sizes");
  HX_REQUIRE(softcap >= 0.0f && (softcap == 0.0f || epilogue == EPI_STORE_F32),
             "hx_gemm_split: a softcap belongs to a float32 store");
  HX_REQUIRE(ldx >= depth && ldw >= depth && ldo >= features, "hx_gemm_split: bad strides");
  HX_REQUIRE(hx_gemm_split_supports(x, ldx, w, ldw, features, depth),
             "hx_gemm_split: rows of %d and %d for a depth of %d are not supported", ldx, ldw, depth);
  HX_REQUIRE(status != nullptr, "hx_gemm_split: status word missing");
  if (tokens == 0) return HX_OK;
  const SplitArgs a{x, ldx, w, ldw, out, ldo, tokens, features, depth, softcap, status};
  int rc;
  switch (epilogue) {
    case EPI_STORE: rc = launch_split<EPI_STORE>(a, stream); break;
    case EPI_STORE_F32: rc = launch_split<EPI_STORE_F32>(a, stream); break;
    case EPI_ADD_F32: rc = launch_split<EPI_ADD_F32>(a, stream); break;
    default:
      hx_set_error("hx_gemm_split: unknown epilogue %d", epilogue);
      return HX_ERR_ARGUMENT;
  }
  if (rc != HX_OK) return rc;
  HX_CHECK_LAUNCH("hx_gemm_split");
  return HX_OK;
}
