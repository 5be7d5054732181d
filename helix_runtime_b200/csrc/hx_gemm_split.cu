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
// Two kernels: one CTA a tile, for shallow products and callers without scratch, and below, with scratch, pairs of
// CTAs (hx_gemm_split_scratch_pays says where the line lies).
//
// What bounds the first: the conversion.  A block of 64 k of a tile of 128 x 128 takes about 4,000 cycles; with one
// of the six products it takes as long, without the loads 3,300 (ncu: issue slots 54 % busy, tensor pipe 38 %):
// eight warps that load, cut and store 16 pieces of four numbers each a block, two warps a scheduler.
// Slower: sixteen such warps (too few registers for loads in flight: 463 -> 502 us), all warps converting
// and summing in turn (539), the weights' lines asked for ahead (4 % faster alone, 3 % slower in place).
// Measured (us, tiles of multiply-adds / one CTA a tile; deep products, which pairs take now): 512 tokens by
// [17,280 x 3,200] 1,581 / 434, by [3,200 x 8,640] 947 / 287, by [4,096 x 4,096] 522 / 157; 33 by the first 248 / 117.
// (With the next block's tokens asked for in front of the proxy fence, which waits for loads too: 459 and 311.)
//
// Every wait on an mbarrier is bounded; a wait that runs out sets a status bit, the CTA skips its
// remaining work, frees its tensor memory and returns.
#include "hx_tcgen05.cuh"
#include "hx_tensor_map.cuh"

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

// The products of a block, term of x and term of w: the smallest first.
__device__ constexpr int TERM_OF_X[6] = {2, 0, 1, 1, 0, 0}, TERM_OF_W[6] = {0, 2, 1, 0, 1, 0};

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

// The terms of four numbers, 8 bytes each, to `at` in the three matrices of terms, term_bytes apart.
__device__ __forceinline__ void store_terms(uint8_t* at, float4 v, size_t term_bytes = TERM_BYTES) {
  asm("{\n\t.reg .b64 s, p, q;\n\t"
      "mov.b64 s, {%4, %4};\n\tmov.b64 p, {%0, %1};\n\tmov.b64 q, {%2, %3};\n\t"
      "mul.rn.f32x2 p, p, s;\n\tmul.rn.f32x2 q, q, s;\n\t"
      "mov.b64 {%0, %1}, p;\n\tmov.b64 {%2, %3}, q;\n\t}"
      : "+f"(v.x), "+f"(v.y), "+f"(v.z), "+f"(v.w)
      : "f"(OPERAND_SCALE));
#pragma unroll
  for (int term = 0; term < 3; ++term) {
    const uint2 packed = make_uint2(two_terms(v.x, v.y), two_terms(v.z, v.w));
    *reinterpret_cast<uint2*>(at + term * term_bytes) = packed;
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

// A summing thread's columns to the output (or added to it).
template <int EPI>
__device__ __forceinline__ void write_sums(const SplitArgs& a, float (&sum)[COLUMNS], int token, int column0) {
  const int live = min(COLUMNS, a.features - column0);
  if (token >= a.tokens || live <= 0) return;
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
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const uint64_t desc_x = make_smem_desc(stage + TERM_OF_X[i] * TERM_BYTES);
      const uint64_t desc_w = make_smem_desc(stage + (3 + TERM_OF_W[i]) * TERM_BYTES);
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
    if (ok) write_sums<EPI>(a, sum, token0 + quarter * 32 + lane, feature0 + half * COLUMNS);
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLUMNS);
  }
}

// ------------------------------------------------------------------ with scratch: pairs of CTAs
//
// Above, every tile cuts its tokens again, for each of its 128 features once: with 512 tokens by [17,280 x
// 3,200] the conversion of the tokens is done 135 times.  Here split_cut_kernel cuts the tokens once (6 bytes a
// number to scratch, which the copy engine brings in swizzled), and two CTAs share a tile of 256 tokens by 128
// features (tcgen05.mma.cta_group::2): each cuts 64 of the weight rows a block, a quarter of the numbers that a
// CTA above cuts for as many products.  Two groups of four warps cut alternate blocks, so a group's loads
// have two blocks' time to arrive.  Persistent: the ring of stages runs on from tile to tile, and the next
// tile's first products run while this one's sums are stored.  Sums of four blocks lie in tensor memory, so
// that the summing warps' round trip is hidden.  The sums are those of the kernel above, bit for bit.
//
// Measured (us, that kernel and this one with its cut): 512 tokens by [17,280 x 3,200] 434 -> 251, by [3,200 x
// 8,640] 287 -> 156.  A block takes 2,300 cycles, its products 1,540 of them; with one product of six 2,000: the
// ring of three stages (72 KB each) hardly covers the tokens' way from the L2, 48 KB a block and CTA.
// Slower: arrivals at the leader's barriers that release all memory (349 us, see mbar_arrive_pair), two
// blocks of weights on their way in registers (318), all eight warps on one block (296), terms kept in registers
// until their stage is free (255 to 282), sums of two blocks (257).
constexpr int PAIR_TOKENS = 2 * TILE;
constexpr int PAIR_ROWS = TILE / 2;                     // weight rows of a CTA
constexpr int PAIR_X_BYTES = TILE * BK * 2, PAIR_W_BYTES = PAIR_ROWS * BK * 2;      // a term
constexpr int PAIR_STAGE_BYTES = 3 * (PAIR_X_BYTES + PAIR_W_BYTES);
constexpr int PAIR_STAGES = 3;
constexpr int PAIR_BUFFERS = 4;                         // of a block's sums
constexpr int PAIR_TMEM_COLUMNS = PAIR_BUFFERS * TILE;
constexpr int PAIR_GROUPS = 2, PAIR_GROUP_WARPS = 8 / PAIR_GROUPS;
constexpr int PAIR_TMA_WARP = SUM_WARPS + PAIR_GROUPS * PAIR_GROUP_WARPS, PAIR_MMA_WARP = PAIR_TMA_WARP + 1;
constexpr int PAIR_THREADS = 32 * (PAIR_TMA_WARP + 4);      // whole warpgroups, whose registers are dealt anew
// At launch 96 a thread; those that issue copies and products need few, the others take what they leave.
constexpr int PAIR_REGISTERS = 96, PAIR_WORK_REGISTERS = 112, PAIR_ISSUE_REGISTERS = 32;
static_assert((PAIR_THREADS / 128 - 1) * PAIR_WORK_REGISTERS + PAIR_ISSUE_REGISTERS <=
                  PAIR_THREADS / 128 * PAIR_REGISTERS,
              "what one side takes the other has given back");
constexpr int PAIR_PASS_ROWS = 32 * PAIR_GROUP_WARPS / (BK / 4), PAIR_PASSES = PAIR_ROWS / PAIR_PASS_ROWS;
constexpr int PAIR_SMEM_BYTES = PAIR_STAGES * PAIR_STAGE_BYTES + 1024 /*alignment*/ + 256 /*barriers*/;

// x [tokens, depth] as three matrices of terms [tokens, ldt], zeros behind the depth.
constexpr int CUT_THREADS = 256;
__global__ __launch_bounds__(CUT_THREADS) void split_cut_kernel(const float* x, int ldx, __nv_bfloat16* terms,
                                                                int ldt, int tokens, int depth) {
  hx_pdl_prologue();
  const int pieces = ldt / 4;
  const size_t term_bytes = static_cast<size_t>(tokens) * ldt * 2;
  for (int token = blockIdx.y; token < tokens; token += gridDim.y) {
    const int piece = blockIdx.x * CUT_THREADS + threadIdx.x;
    if (piece >= pieces) continue;
    const float4 v = 4 * piece < depth
                         ? *reinterpret_cast<const float4*>(x + static_cast<size_t>(token) * ldx + 4 * piece)
                         : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    store_terms(reinterpret_cast<uint8_t*>(terms + static_cast<size_t>(token) * ldt + 4 * piece), v, term_bytes);
  }
}

template <int EPI>
__global__ __cluster_dims__(2, 1, 1) __launch_bounds__(PAIR_THREADS, 1) void gemm_split_pair_kernel(
    const __grid_constant__ CUtensorMap map_terms, const SplitArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + PAIR_STAGES * PAIR_STAGE_BYTES);      // leader's count
  uint64_t* empty_bar = full_bar + PAIR_STAGES;
  uint64_t* sum_full_bar = empty_bar + PAIR_STAGES;
  uint64_t* sum_empty_bar = sum_full_bar + PAIR_BUFFERS;      // leader's count
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(sum_empty_bar + PAIR_BUFFERS);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_rank());
  const int worker = blockIdx.x >> 1, workers = gridDim.x >> 1;
  const int blocks = (a.depth + BK - 1) / BK;
  const int token_tiles = (a.tokens + PAIR_TOKENS - 1) / PAIR_TOKENS;
  const int units = token_tiles * ((a.features + TILE - 1) / TILE);
  const int own_units = worker < units ? (units - worker - 1) / workers + 1 : 0;
  const int fills = own_units * blocks;      // blocks of all its tiles
  // the tile that the i-th of them is, the tokens of a feature tile one after the other
  auto tile_at = [&](int i, int& token0, int& feature0) {
    const int unit = worker + i * workers;
    token0 = unit % token_tiles * PAIR_TOKENS + rank * TILE;
    feature0 = unit / token_tiles * TILE;
  };
  hx_pdl_trigger();
  if (threadIdx.x == 0) {
    for (int s = 0; s < PAIR_STAGES; ++s) {
      mbar_init(&full_bar[s], 1 + 2 * PAIR_GROUP_WARPS);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < PAIR_BUFFERS; ++b) {
      mbar_init(&sum_full_bar[b], 1);
      mbar_init(&sum_empty_bar[b], 2 * SUM_WARPS);
    }
    *failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == PAIR_MMA_WARP) tmem_alloc_pair(tmem_holder, PAIR_TMEM_COLUMNS);
  tc_fence_before();
  __syncthreads();
  cluster_sync();      // nothing arrives at the other CTA's barriers before they are there
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  auto give_up = [&]() {
    atomicOr(a.status, HX_FLAG_WAIT_TIMEOUT);
    *failed = 1;
  };

  if (warp < SUM_WARPS) {
    // ------------------------------------------------------- sums of the blocks, and the epilogue
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(PAIR_WORK_REGISTERS));
    hx_pdl_wait();
    const int quarter = warp & 3, half = warp >> 2;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + half * COLUMNS;
    uint32_t block = 0;
    bool ok = true;
    for (int i = 0; i < own_units && ok; ++i) {
      float sum[COLUMNS];
#pragma unroll
      for (int j = 0; j < COLUMNS; ++j) sum[j] = 0.0f;
      for (int kb = 0; kb < blocks; ++kb, ++block) {
        const int buffer = block % PAIR_BUFFERS;
        if (lane == 0) ok = !*failed && mbar_wait(&sum_full_bar[buffer], (block / PAIR_BUFFERS) & 1u);
        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        if (!ok) {
          if (lane == 0) give_up();
          break;
        }
        tc_fence_after();
#pragma unroll
        for (int column = 0; column < COLUMNS; column += 32) {
          uint32_t v[2][16];
          tmem_load16_issue(lane_base + buffer * TILE + column, v[0]);
          tmem_load16_issue(lane_base + buffer * TILE + column + 16, v[1]);
          tmem_load_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j)
            sum[column + j] = fmaf(__uint_as_float(v[j / 16][j % 16]), SUM_SCALE, sum[column + j]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_pair(cluster_address(&sum_empty_bar[buffer], 0));
      }
      int token0, feature0;
      tile_at(i, token0, feature0);
      if (ok) write_sums<EPI>(a, sum, token0 + quarter * 32 + lane, feature0 + half * COLUMNS);
    }
  } else if (warp < PAIR_TMA_WARP) {
    // -------------------------------- weights (no kernel of a step writes them: no wait for the one before)
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(PAIR_WORK_REGISTERS));
    const int thread = (threadIdx.x - 32 * SUM_WARPS) % (32 * PAIR_GROUP_WARPS);
    const int piece = thread % (BK / 4), row0 = thread / (BK / 4);
    float4 v[PAIR_PASSES];
    auto load = [&](int fill) {
      int token0, feature0;
      tile_at(fill / blocks, token0, feature0);
      const int first = feature0 + rank * PAIR_ROWS, k = fill % blocks * BK + 4 * piece;
      const float* from = a.w + static_cast<size_t>(first) * a.ldw + k;
#pragma unroll
      for (int p = 0; p < PAIR_PASSES; ++p) {
        const int row = row0 + PAIR_PASS_ROWS * p;
        v[p] = k < a.depth && first + row < a.features      // the depth is a multiple of four
                   ? *reinterpret_cast<const float4*>(from + static_cast<size_t>(row) * a.ldw)
                   : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
    };
    int fill = (warp - SUM_WARPS) / PAIR_GROUP_WARPS;
    if (fill < fills) load(fill);
    for (; fill < fills; fill += PAIR_GROUPS) {
      const int s = fill % PAIR_STAGES;
      bool ok = true;
      if (lane == 0) ok = !*failed && mbar_wait(&empty_bar[s], ((fill / PAIR_STAGES) & 1u) ^ 1u);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) {
        if (lane == 0) give_up();
        break;
      }
      uint8_t* terms = smem + s * PAIR_STAGE_BYTES + 3 * PAIR_X_BYTES;
#pragma unroll
      for (int p = 0; p < PAIR_PASSES; ++p) {
        const int row = row0 + PAIR_PASS_ROWS * p;
        store_terms(terms + row * (BK * 2) + (((piece >> 1) ^ (row & 7)) << 4) + ((piece & 1) << 3), v[p],
                    PAIR_W_BYTES);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_pair(cluster_address(&full_bar[s], 0));
      if (fill + PAIR_GROUPS < fills) load(fill + PAIR_GROUPS);
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(PAIR_ISSUE_REGISTERS));
    if (warp == PAIR_TMA_WARP) {
      // ------------------------------------------------------------------ the tokens' terms
      hx_pdl_wait();
      if (hx_elect_one()) {
        int fill = 0;
        for (int i = 0; i < own_units && !*failed; ++i) {
          int token0, feature0;
          tile_at(i, token0, feature0);
          for (int kb = 0; kb < blocks; ++kb, ++fill) {
            const int s = fill % PAIR_STAGES;
            if (!mbar_wait(&empty_bar[s], ((fill / PAIR_STAGES) & 1u) ^ 1u)) {
              give_up();
              break;
            }
            if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * 3 * PAIR_X_BYTES);
            const uint32_t bar = cluster_address(&full_bar[s], 0);
#pragma unroll
            for (int term = 0; term < 3; ++term)
              tma_load_2d_pair(smem + s * PAIR_STAGE_BYTES + term * PAIR_X_BYTES, &map_terms, bar, kb * BK,
                               term * a.tokens + token0);
          }
        }
        // the leader's last arrivals at this CTA's barriers, before the CTA may end
        for (int last = fill > PAIR_STAGES ? fill - PAIR_STAGES : 0; last < fill && !*failed; ++last)
          if (!mbar_wait(&empty_bar[last % PAIR_STAGES], (last / PAIR_STAGES) & 1u)) give_up();
      }
    } else if (warp == PAIR_MMA_WARP && rank == 0 && hx_elect_one()) {
      // ---------------------------------------------------------------- products, for both CTAs
      constexpr uint32_t idesc = make_idesc(PAIR_TOKENS, TILE);
      for (int fill = 0; fill < fills && !*failed; ++fill) {
        const int s = fill % PAIR_STAGES, buffer = fill % PAIR_BUFFERS;
        if (!mbar_wait(&sum_empty_bar[buffer], ((fill / PAIR_BUFFERS) & 1u) ^ 1u) ||
            !mbar_wait(&full_bar[s], (fill / PAIR_STAGES) & 1u)) {
          give_up();
          break;
        }
        tc_fence_after();
        const uint32_t stage = smem_u32(smem + s * PAIR_STAGE_BYTES);
        const uint32_t sums = tmem_base + buffer * TILE;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
          const uint64_t desc_x = make_smem_desc(stage + TERM_OF_X[i] * PAIR_X_BYTES);
          const uint64_t desc_w = make_smem_desc(stage + 3 * PAIR_X_BYTES + TERM_OF_W[i] * PAIR_W_BYTES);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t step = static_cast<uint64_t>(k * UMMA_K * 2 >> 4);
            umma_bf16_pair(sums, desc_x + step, desc_w + step, idesc, i > 0 || k > 0 ? 1u : 0u);
          }
        }
        umma_commit_pair(&empty_bar[s]);
        umma_commit_pair(&sum_full_bar[buffer]);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync();      // neither CTA's memory is read or arrived at any more
  if (warp == PAIR_MMA_WARP) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, PAIR_TMEM_COLUMNS);
  }
}

// Numbers of a row of terms: rows of a tensor map begin on 16 bytes.
int terms_row(int depth) { return (depth + 7) / 8 * 8; }

template <int EPI>
int launch_split(const SplitArgs& a, __nv_bfloat16* terms, cudaStream_t stream) {
  static std::once_flag once;
  static bool configured = false;
  std::call_once(once, [] {
    configured = cudaFuncSetAttribute(gemm_split_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      SMEM_BYTES) == cudaSuccess &&
                 cudaFuncSetAttribute(gemm_split_pair_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      PAIR_SMEM_BYTES) == cudaSuccess;
    if (!configured) cudaGetLastError();
  });
  if (!configured) {
    hx_set_error("hx_gemm_split: cannot reserve %d bytes of shared memory", SMEM_BYTES);
    return HX_ERR_LAUNCH;
  }
  const int pairs = hx_device_sm_count() / 2;
  const long long units = static_cast<long long>((a.tokens + PAIR_TOKENS - 1) / PAIR_TOKENS) *
                          ((a.features + TILE - 1) / TILE);
  // (a pair counts its blocks in 32 bits, a tensor map the rows of all three terms)
  if (terms != nullptr && (units / pairs + 1) * ((a.depth + BK - 1) / BK) < (1ll << 30) && a.tokens < (1 << 29)) {
    const int ldt = terms_row(a.depth);
    CUtensorMap map;
    const int rc = hx_tensor_map("hx_gemm_split", terms, 3ull * a.tokens, ldt, ldt, TILE, BK, true, &map);
    if (rc != HX_OK) return rc;
    const int piece_blocks = (ldt / 4 + CUT_THREADS - 1) / CUT_THREADS;
    hx_launch(split_cut_kernel, dim3(piece_blocks, a.tokens < 65535 ? a.tokens : 65535), CUT_THREADS, 0, stream,
              a.x, a.ldx, terms, ldt, a.tokens, a.depth);
    HX_CHECK_LAUNCH("hx_gemm_split (terms)");
    hx_launch(gemm_split_pair_kernel<EPI>, 2 * static_cast<int>(units < pairs ? units : pairs), PAIR_THREADS,
              PAIR_SMEM_BYTES, stream, map, a);
    return HX_OK;
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

// Whether it is the faster road for this many tokens, without scratch: with few tiles either road is one round of CTAs that
// walk the depth alone, 2.0 us a block of 64 k on the CUDA cores (32 x 32 a tile, several CTAs an SM) against
// 2.2 here, so the CUDA cores need more than two such tiles an SM to be slower.  Measured (us, CUDA cores / here):
// 9,600 features of 3,200 17 tokens 141 / 111; 4,096 of 4,096 64 tokens 131 / 143, 100 188 / 146; 3,200 of 8,640 64
// 266 / 289, 100 375 / 294.
HX_API int hx_gemm_split_pays(int tokens, int features) {
  const long long small = static_cast<long long>((tokens + 31) / 32) * ((features + 31) / 32);
  return tokens > 16 && small >= 2ll * hx_device_sm_count();
}

// The same for a caller with scratch.  The cut is a launch of its own, and a pair's way through its first blocks is
// longer: 6 to 8 us more than the CUDA cores take for a shallow product, 2 more than one CTA a tile, which a deep
// product or several rounds of tiles bring back.  Measured (us, the road without scratch / here):
//   fewer tiles of 32 x 32 than SMs: 129 tokens by [700 x 64] 3.6 / 12.2, x 512 17.0 / 18.3, x 768 24.3 / 23.0;
//   fewer than two an SM: 256 by [700 x 256] 11.9 / 18.3, 129 by [1,500 x 256] 13.4 / 16.1, x 512 24.6 / 19.1, 64 by [4,000 x
//   128] 8.4 / 10.1, x 256 14.5 / 12.2;
//   more (without scratch one CTA a tile): 256 by [9,000 x 64] 9.7 / 12.7, 512 18.6 / 17.2, 512 by [4,000 x 128] 12.4 / 13.7, 1,024
//   23.6 / 20.0, 256 by [4,000 x 256] 16.8 / 14.6, 2,048 by [300 x 256] 15.7 / 16.5, x 512 23.3 / 20.2.
// 17 tokens by [17,280 x 3,200] 123 / 120, by [3,200 x 8,640] 248 / 151.  (Up to 16 tokens, and up to 128 of few
// features, are hx_gemm_few.cu's.)
HX_API int hx_gemm_split_scratch_pays(int tokens, int features, int depth) {
  const long long small = static_cast<long long>((tokens + 31) / 32) * ((features + 31) / 32);
  const int sms = hx_device_sm_count();
  if (tokens <= 16 || small < 32) return 0;
  if (small < 2ll * sms) return depth >= (small < sms ? 640 : tokens > 64 ? 512 : 256);
  const long long units = static_cast<long long>((tokens + PAIR_TOKENS - 1) / PAIR_TOKENS) *
                          ((features + TILE - 1) / TILE);
  return depth >= 512 || units > sms / 2 || (depth >= 256 && tokens <= 4ll * features);
}

// Numbers of bfloat16 scratch (on 16 bytes) that hx_gemm_split_scratch has a use for.
HX_API long long hx_gemm_split_terms(int tokens, int depth) {
  return tokens > 0 && hx_device_sm_count() >= 2 ? 3ll * tokens * terms_row(depth) : 0;
}

// float32 x [tokens, ldx], w [features, ldw], out [tokens, ldo]; epilogues and softcap as hx_gemm_simt_softcapped.
// `terms`: scratch of hx_gemm_split_terms() numbers, or null.
HX_API int hx_gemm_split_scratch(const float* x, int ldx, const float* w, int ldw, float* out, int ldo, int tokens,
                                 int features, int depth, int epilogue, float softcap, void* terms,
                                 long long terms_size, int* status, cudaStream_t stream) {
  HX_REQUIRE(tokens >= 0 && features > 0 && depth > 0, "hx_gemm_split: bad sizes");
  HX_REQUIRE(softcap >= 0.0f && (softcap == 0.0f || epilogue == EPI_STORE_F32),
             "hx_gemm_split: a softcap belongs to a float32 store");
  HX_REQUIRE(ldx >= depth && ldw >= depth && ldo >= features, "hx_gemm_split: bad strides");
  HX_REQUIRE(hx_gemm_split_supports(x, ldx, w, ldw, features, depth),
             "hx_gemm_split: rows of %d and %d for a depth of %d are not supported", ldx, ldw, depth);
  HX_REQUIRE(status != nullptr, "hx_gemm_split: status word missing");
  if (tokens == 0) return HX_OK;
  __nv_bfloat16* cut = nullptr;
  const long long needed = hx_gemm_split_terms(tokens, depth);
  if (terms != nullptr && needed > 0) {
    HX_REQUIRE(terms_size >= needed && (reinterpret_cast<uintptr_t>(terms) & 15) == 0,
               "hx_gemm_split: scratch of %lld numbers for %lld, or not on 16 bytes", terms_size, needed);
    cut = static_cast<__nv_bfloat16*>(terms);
  }
  const SplitArgs a{x, ldx, w, ldw, out, ldo, tokens, features, depth, softcap, status};
  int rc;
  switch (epilogue) {
    case EPI_STORE: rc = launch_split<EPI_STORE>(a, cut, stream); break;
    case EPI_STORE_F32: rc = launch_split<EPI_STORE_F32>(a, cut, stream); break;
    case EPI_ADD_F32: rc = launch_split<EPI_ADD_F32>(a, cut, stream); break;
    default:
      hx_set_error("hx_gemm_split: unknown epilogue %d", epilogue);
      return HX_ERR_ARGUMENT;
  }
  if (rc != HX_OK) return rc;
  HX_CHECK_LAUNCH("hx_gemm_split");
  return HX_OK;
}

HX_API int hx_gemm_split(const float* x, int ldx, const float* w, int ldw, float* out, int ldo, int tokens,
                         int features, int depth, int epilogue, float softcap, int* status, cudaStream_t stream) {
  return hx_gemm_split_scratch(x, ldx, w, ldw, out, ldo, tokens, features, depth, epilogue, softcap, nullptr, 0,
                               status, stream);
}
