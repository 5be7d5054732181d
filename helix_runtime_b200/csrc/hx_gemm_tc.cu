// bfloat16 matrix product on the 5th-generation tensor cores (tcgen05, sm_100a).
//
//   out[t, f] (+)= sum_k x[t, k] * w[f, k]        x: [tokens, K]   w: [features, K]
//
// Both operands are K-major, which is how the checkpoint stores its matrices, so no
// transposed copy is ever made (the reference keeps [in, out] and multiplies with a
// 16x16 shared-memory kernel, src/kernels/cuda/matmul.cu:36-71).
//
// Mapping.  The WEIGHT tile is the MMA's M operand (128 features per CTA) and the
// TOKEN tile its N operand (BN = 16 ... 256 tokens), so one kernel covers decoding
// (a handful of tokens, pure weight streaming) and prompt portions (256-token
// tiles).  The accumulator lives in tensor memory as [128 feature lanes x BN token
// columns] float32.  Warp roles:
//   warp 0      one lane issues the TMA loads of both operand tiles, STAGES deep;
//   warp 1      allocates tensor memory; one lane issues tcgen05.mma and commits;
//   warps 2..5  epilogue: tcgen05.ld their 32-lane quarter, apply the epilogue, store.
// Shared-memory tiles are [rows x 64] bfloat16 with the 128-byte swizzle that both
// TMA and the MMA descriptors understand.
//
// Epilogues: store bf16, store f32 (logits), add into f32 (the residual stream; with
// split-K through float32 atomics), and SwiGLU, where the CTA multiplies the same
// token tile with a gate tile and an up tile of the fused [2I, K] matrix into two
// accumulators and writes silu(gate) * up.  For prompt portions the fused QKV product can
// also rotate queries and keys and put keys and values into the cache pages in its epilogue
// (hx_gemm_tc_rope_append), which saves the separate pass over the projected rows.
//
// Every wait on an mbarrier is bounded; a wait that runs out sets a status bit, the
// CTA skips its remaining work, frees its tensor memory and returns.
#include "hx_tcgen05.cuh"
#include "hx_tensor_map.cuh"

#include <cmath>
#include <type_traits>

namespace {

constexpr int BM = 128;        // features per CTA (MMA M)
constexpr int BK = 64;         // k elements per stage: 128 bytes, one swizzle span
constexpr int UMMA_K = 16;     // k elements per tcgen05.mma of kind::f16
constexpr int THREADS = 192;

enum Epilogue : int {
  EPI_STORE_BF16 = 0, EPI_STORE_F32 = 1, EPI_ADD_F32 = 2, EPI_SWIGLU = 3,
  EPI_ROPE_APPEND = 4      // persistent kernel only, see RopeArgs
};

// Where the [128 rows x 64 k] box of the weights that begins at row `row`, k-block `kb`, is.
// Row-major weights: a box is 128 row segments of 128 bytes, one per row of the matrix.  Tiled
// weights (k_tiles > 0) store every such box as 16 contiguous kilobytes, box after box along
// k, then along the rows: a product that streams its weights once then reads DRAM in long
// runs instead of 128-byte pieces (measured: 4 % less time for the decode products).
__device__ __forceinline__ void load_weight_box(void* dst, const CUtensorMap* map, uint64_t* bar,
                                                int row, int kb, int k_tiles) {
  if (k_tiles > 0) {
    tma_load_2d(dst, map, bar, 0, ((row / BM) * k_tiles + kb) * BM);
  } else {
    tma_load_2d(dst, map, bar, kb * BK, row);
  }
}

// A float32 store may let the sums run into a level: cap * tanh(x / cap) (cap 0: as they are).
__device__ __forceinline__ float level_off(float x, float cap) {
  return cap > 0.0f ? cap * tanhf(x / cap) : x;
}

// This thread's feature of 16 tokens from token0 on, as the epilogue stores it.
template <int EPI>
__device__ __forceinline__ void store_columns(void* out, int ldo, int tokens, int token0, int feature,
                                              const float (&acc)[16], float softcap) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const int token = token0 + j;
    if (token < tokens) {
      const size_t index = static_cast<size_t>(token) * ldo + feature;
      if (EPI == EPI_STORE_BF16 || EPI == EPI_SWIGLU) {
        static_cast<__nv_bfloat16*>(out)[index] = __float2bfloat16_rn(acc[j]);
      } else if (EPI == EPI_STORE_F32) {
        static_cast<float*>(out)[index] = level_off(acc[j], softcap);
      } else {
        // a reduction at the memory side: nothing to wait for.  With one writer per
        // element the sum is still deterministic.
        atomicAdd(static_cast<float*>(out) + index, acc[j]);
      }
    }
  }
}

// One epilogue warp's share of a finished tile: its 32 features (tensor-memory lanes) for all
// BN token columns, 16 columns at a time.  With SwiGLU the up accumulator sits BN columns on.
template <int BN, int EPI>
__device__ __forceinline__ void write_tile(void* out, int ldo, int tokens, int features,
                                           uint32_t lane_address, int feature, int token0,
                                           int activation, float gate_limit,
                                           const float* gate_bias, const float* up_bias,
                                           float softcap) {
  const bool feature_ok = feature < features;
  // this thread's feature is one row of the gate and one of the up matrix: one bias each
  const float gate_b = EPI == EPI_SWIGLU && gate_bias != nullptr && feature_ok ? gate_bias[feature] : 0.0f;
  const float up_b = EPI == EPI_SWIGLU && up_bias != nullptr && feature_ok ? up_bias[feature] : 0.0f;
#pragma unroll 1
  for (int column = 0; column < BN; column += 16) {
    if (token0 + column >= tokens) break;   // uniform over the warp
    float acc[16];
    tmem_load16(lane_address + column, acc);
    if (EPI == EPI_SWIGLU) {
      float up[16];
      tmem_load16(lane_address + BN + column, up);
#pragma unroll
      for (int j = 0; j < 16; ++j)
        acc[j] = hx_gated_fast(acc[j] + gate_b, up[j] + up_b, activation, gate_limit);
    }
    if (feature_ok) store_columns<EPI>(out, ldo, tokens, token0 + column, feature, acc, softcap);
  }
}

// ---------------------------------------------------------------------- kernel

template <int BN, bool DUAL>
struct TileConfig {
  static constexpr int kWeightBytes = BM * BK * 2 * (DUAL ? 2 : 1);
  static constexpr int kTokenBytes = BN * BK * 2;
  static constexpr int kStageBytes = kWeightBytes + kTokenBytes;
  // Token tiles up to 128 are the weight-streaming case (decoding, short prompt portions):
  // two CTAs share an SM so that one CTA's pipeline fill and epilogue overlap the other's
  // loads (with 128 tokens that leaves three stages of 32 KB each, and still wins: steps of
  // 65 to 128 tokens take 9 % less time than with one CTA of six stages).  Larger tiles take
  // the SM.
  static constexpr int kBudget = (BN <= 128 && !DUAL) ? 100 * 1024 : 200 * 1024;
  static constexpr int kStagesRaw = kBudget / kStageBytes;
  static constexpr int kStages = kStagesRaw > 8 ? 8 : kStagesRaw;
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*alignment*/ + 256 /*barriers*/;
  static constexpr int kAccumulatorColumns = BN * (DUAL ? 2 : 1);
  static constexpr int kTmemColumns =
      kAccumulatorColumns <= 32 ? 32
      : kAccumulatorColumns <= 64 ? 64
      : kAccumulatorColumns <= 128 ? 128
      : kAccumulatorColumns <= 256 ? 256 : 512;
};

struct GemmArgs {
  void* out;
  int ldo;
  int tokens;
  int features;     // rows of the output the epilogue may write
  int depth;        // K
  int up_row_offset;  // SwiGLU: row of the first up-projection feature in the weight matrix
  int k_blocks_per_split;
  int k_tiles;        // > 0: the weights are stored as tiles, this many along k
  int* status;
  int activation;     // gated epilogue: what the gate passes through (HxGateActivation)
  // Grouped product: token tile t multiplies with the rows of group tile_group[t] of the
  // weight matrix (group g's rows start at g * group_rows); a negative group skips the tile.
  // The list lies in device memory and is written by an earlier kernel of the stream.
  const int* tile_group = nullptr;
  int group_rows = 0;
  float gate_limit = 0.0f;    // gated epilogue: the limit of HX_GATE_CLAMPED_SIGMOID
  // gated epilogue: float32 biases of the gate and the up rows, [features] each (null: none)
  const float* gate_bias = nullptr;
  const float* up_bias = nullptr;
  float softcap = 0.0f;       // float32 store: see level_off
  // Store epilogues: > 1 where the CTAs of a tile, one for each run of k-blocks, are a cluster that adds its
  // sums up (see gather_parts).
  int cluster = 1;
};

// A product that is stored cannot be cut along the reduction into atomic adds, and one with few tiles (a
// router of 16 features, a projection of 1,280) was a few CTAs that walked the whole depth, 0.25 us a block
// of 64.  Here the CTAs that share a tile's depth form a cluster: each leaves its sums in its own shared memory
// (the ring is empty by then), [column][feature], and every 16 columns are added up by one of them, in the order of
// the ranks, and stored.  Measured (us, in a chain of launches, a CTA a tile before): 1 token by [16 x 4,096] 13.1 ->
// 7.2, 64 16.0 -> 8.6, 100 20.4 -> 10.4, 1,024 13.8 -> 11.6; by [1,280 x 4,096] 13.2 -> 7.6, 16.3 -> 9.9, 25.7 -> 12.5
// (1, 64, 100 tokens); by [4,096 x 4,096] 13.2 -> 8.8, 15.4 -> 11.6, 22.4 -> 15.8.
template <int BN>
__device__ __forceinline__ void leave_part(float* part, uint32_t lane_address, int row, int columns) {
#pragma unroll 1
  for (int column = 0; column < columns; column += 16) {
    float acc[16];
    tmem_load16(lane_address + column, acc);
#pragma unroll
    for (int j = 0; j < 16; ++j) part[(column + j) * BM + row] = acc[j];
  }
}

template <int BN, int EPI>
__device__ __forceinline__ void gather_parts(const GemmArgs& a, const float* part, int rank, int row, int feature,
                                             int token0) {
#pragma unroll 1
  for (int column = 16 * rank; column < BN && token0 + column < a.tokens; column += 16 * a.cluster) {
    float sums[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) sums[j] = 0.0f;
    for (int r = 0; r < a.cluster; ++r) {
      const uint32_t from = cluster_address(part + column * BM + row, r);
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        float x;
        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(from + j * BM * 4));
        sums[j] += x;
      }
    }
    if (feature >= a.features) continue;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int token = token0 + column + j;
      if (token >= a.tokens) break;
      const size_t index = static_cast<size_t>(token) * a.ldo + feature;
      if (EPI == EPI_STORE_BF16) static_cast<__nv_bfloat16*>(a.out)[index] = __float2bfloat16_rn(sums[j]);
      else static_cast<float*>(a.out)[index] = level_off(sums[j], a.softcap);
    }
  }
}

// A grouped product of a few tiles of 16 tokens (experts of one to three tokens) with float32 sums leaves them in
// tensor memory for one block of 64 k only: the tensor cores do not round to nearest, and a chain over a depth of
// 2,816 is off by 3.0e-6 (relative 2-norm), where a product a pair on the CUDA cores (hx_expert_down), which such
// experts would else take, is off by 8.6e-8.  Four blocks are a turn, two turns share tensor memory; the blocks are
// added here in registers, with what each addition rounds away: 7.0e-8.  Measured (us, the chain / here): 4 tiles by
// [4,096 x 2,816] 20.0 / 21.5, 2 by [4,096 x 4,096] 20.0 / 22.7; turns of one block 23.8 and 30.2.
constexpr int TURN_BLOCKS = 4, TURN_COLUMNS = 16 * TURN_BLOCKS, TURNS = 2;

__device__ __forceinline__ void sum_blocks(const GemmArgs& a, uint32_t lane_address, uint64_t* turn_full_bar,
                                           uint64_t* turn_empty_bar, int blocks, int feature, int token0) {
  const int lane = threadIdx.x & 31;
  float sum[16], lost[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) sum[j] = lost[j] = 0.0f;
  for (int turn = 0; turn * TURN_BLOCKS < blocks; ++turn) {
    const int buffer = turn % TURNS;
    bool ok = true;
    if (lane == 0) ok = mbar_wait(&turn_full_bar[buffer], static_cast<uint32_t>(turn / TURNS) & 1u);
    ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
    if (!ok) {
      if (lane == 0) atomicOr(a.status, HX_FLAG_WAIT_TIMEOUT);
      return;
    }
    tc_fence_after();
#pragma unroll
    for (int half = 0; half < TURN_BLOCKS; half += 2) {
      uint32_t block[2][16];
      tmem_load16_issue(lane_address + buffer * TURN_COLUMNS + 16 * half, block[0]);
      tmem_load16_issue(lane_address + buffer * TURN_COLUMNS + 16 * half + 16, block[1]);
      tmem_load_wait();
      if (half + 2 == TURN_BLOCKS) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&turn_empty_bar[buffer]);
      }
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        if (turn * TURN_BLOCKS + half + b >= blocks) break;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float x = __uint_as_float(block[b][j]), before = sum[j];
          sum[j] = before + x;
          const float added = sum[j] - before;
          lost[j] += (before - (sum[j] - added)) + (x - added);
        }
      }
    }
  }
  if (feature >= a.features) return;
#pragma unroll
  for (int j = 0; j < 16; ++j)
    if (isfinite(sum[j])) sum[j] += lost[j];      // (an infinite sum has lost what is no number)
  store_columns<EPI_STORE_F32>(a.out, a.ldo, a.tokens, token0, feature, sum, a.softcap);
}

// IN_BLOCKS: see sum_blocks; a kernel of its own because of its registers (79 a thread, 40 without).
template <int BN, int EPI, bool IN_BLOCKS = false>
__global__ __launch_bounds__(THREADS) void gemm_tc_kernel(
    const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
    const GemmArgs args) {
  constexpr bool DUAL = EPI == EPI_SWIGLU;
  using Config = TileConfig<BN, DUAL>;
  constexpr int STAGES = Config::kStages;
  static_assert(!IN_BLOCKS || (BN == 16 && EPI == EPI_STORE_F32), "sum_blocks is for tiles of 16 tokens");
  constexpr bool CLUSTERS = (EPI == EPI_STORE_BF16 || EPI == EPI_STORE_F32) && BN <= 128;
  static_assert(!CLUSTERS || BN * BM * 4 <= STAGES * Config::kStageBytes, "a part lies where the ring was");

  hx_pdl_trigger();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * Config::kStageBytes);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* accum_bar = empty_bar + STAGES;
  uint64_t* turn_full_bar = accum_bar + 1;      // [TURNS] a turn's sums are complete
  uint64_t* turn_empty_bar = turn_full_bar + TURNS;      // [TURNS] they are read
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(turn_empty_bar + TURNS);
  static_assert((2 * STAGES + 1 + 2 * TURNS) * 8 + 4 <= 256, "the barriers' place");
  constexpr int TMEM_COLUMNS = IN_BLOCKS ? TURNS * TURN_COLUMNS : Config::kTmemColumns;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // token tiles vary fastest: the CTAs that run side by side share a weight tile, which then
  // comes from DRAM once and from the L2 for the rest; the token tiles are L2-resident anyway
  const int feature0 = blockIdx.y * BM;
  const int token0 = blockIdx.x * BN;
  const int total_k_blocks = (args.depth + BK - 1) / BK;
  const int kb_begin = blockIdx.z * args.k_blocks_per_split;
  const int kb_end = min(kb_begin + args.k_blocks_per_split, total_k_blocks);
  int weight_row0 = feature0;      // row of the weight matrix that feature0 is
  bool skipped = false;
  if (args.tile_group != nullptr) {
    hx_pdl_wait();                 // the list is the work of a kernel before this one
    const int group = args.tile_group[blockIdx.x];
    skipped = group < 0;
    weight_row0 = (skipped ? 0 : group * args.group_rows) + feature0;
  }
  const int n_k_blocks = skipped ? 0 : kb_end - kb_begin;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(accum_bar, 1);
    if (IN_BLOCKS) {
      for (int b = 0; b < TURNS; ++b) {
        mbar_init(&turn_full_bar[b], 1);
        mbar_init(&turn_empty_bar[b], 4);      // one arrival per epilogue warp
      }
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_holder, TMEM_COLUMNS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  if (n_k_blocks > 0) {
    if (warp == 0) {
      // ------------------------------------------------------------ TMA producer
      if (hx_elect_one()) {
        // The weight tiles do not depend on the kernel before this one: the first STAGES of
        // them are requested at once, before the dependency wait, so that weights stream
        // across the kernel boundary.  The token tiles follow after the wait.
        const int eager = n_k_blocks < STAGES ? n_k_blocks : STAGES;
        for (int i = 0; i < eager; ++i) {
          uint8_t* stage = smem + i * Config::kStageBytes;
          mbar_expect_tx(&full_bar[i], Config::kStageBytes);
          load_weight_box(stage, &map_w, &full_bar[i], weight_row0, kb_begin + i, args.k_tiles);
          if (DUAL)
            load_weight_box(stage + BM * BK * 2, &map_w, &full_bar[i],
                            args.up_row_offset + weight_row0, kb_begin + i, args.k_tiles);
        }
        hx_pdl_wait();
        for (int i = 0; i < eager; ++i) {
          uint8_t* stage = smem + i * Config::kStageBytes;
          tma_load_2d(stage + Config::kWeightBytes, &map_x, &full_bar[i], (kb_begin + i) * BK,
                      token0);
        }
        for (int i = eager; i < n_k_blocks; ++i) {
          const int s = i % STAGES;
          const uint32_t round = static_cast<uint32_t>(i / STAGES);
          if (!mbar_wait(&empty_bar[s], (round & 1u) ^ 1u)) {
            atomicOr(args.status, HX_FLAG_WAIT_TIMEOUT);
            break;
          }
          uint8_t* stage = smem + s * Config::kStageBytes;
          mbar_expect_tx(&full_bar[s], Config::kStageBytes);
          const int k = (kb_begin + i) * BK;
          load_weight_box(stage, &map_w, &full_bar[s], weight_row0, kb_begin + i, args.k_tiles);
          if (DUAL)
            load_weight_box(stage + BM * BK * 2, &map_w, &full_bar[s],
                            args.up_row_offset + weight_row0, kb_begin + i, args.k_tiles);
          tma_load_2d(stage + Config::kWeightBytes, &map_x, &full_bar[s], k, token0);
        }
      }
    } else if (warp == 1) {
      // -------------------------------------------------------------- MMA issuer
      if (hx_elect_one()) {
        constexpr uint32_t idesc = make_idesc(BM, BN);
        bool ok = true;
        for (int i = 0; i < n_k_blocks && ok; ++i) {
          const int s = i % STAGES;
          const uint32_t round = static_cast<uint32_t>(i / STAGES);
          const int turn = i / TURN_BLOCKS;
          if (!mbar_wait(&full_bar[s], round & 1u) ||
              (IN_BLOCKS && i % TURN_BLOCKS == 0 &&
               !mbar_wait(&turn_empty_bar[turn % TURNS], (static_cast<uint32_t>(turn / TURNS) & 1u) ^ 1u))) {
            atomicOr(args.status, HX_FLAG_WAIT_TIMEOUT);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sums = tmem_base + (IN_BLOCKS ? i % (TURNS * TURN_BLOCKS) * 16 : 0);
          const uint32_t stage = smem_u32(smem + s * Config::kStageBytes);
          const uint64_t desc_w = make_smem_desc(stage);
          const uint64_t desc_w2 = make_smem_desc(stage + BM * BK * 2);
          const uint64_t desc_x = make_smem_desc(stage + Config::kWeightBytes);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            // stepping 16 k-elements = 32 bytes inside the swizzle span: +2 in 16-byte units
            const uint64_t step = static_cast<uint64_t>(k * UMMA_K * 2 >> 4);
            const uint32_t accumulate = ((i > 0 && !IN_BLOCKS) || k > 0) ? 1u : 0u;
            umma_bf16(sums, desc_w + step, desc_x + step, idesc, accumulate);
            if (DUAL) umma_bf16(sums + BN, desc_w2 + step, desc_x + step, idesc, accumulate);
          }
          umma_commit(&empty_bar[s]);   // the stage may be refilled once these MMAs have read it
          if (IN_BLOCKS && (i % TURN_BLOCKS == TURN_BLOCKS - 1 || i + 1 == n_k_blocks))
            umma_commit(&turn_full_bar[turn % TURNS]);
        }
        umma_commit(accum_bar);         // the accumulator is complete
      }
    } else {
      // ---------------------------------------------------------------- epilogue
      hx_pdl_wait();                    // the output may be something the last kernel read
      const int quarter = warp & 3;     // tensor-memory lanes [32 * quarter, 32 * quarter + 32)
      const int feature = feature0 + quarter * 32 + lane;
      const uint32_t lane_address = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
      if constexpr (IN_BLOCKS)
        sum_blocks(args, lane_address, turn_full_bar, turn_empty_bar, n_k_blocks, feature, token0);
      bool ok = true;
      if (lane == 0) ok = mbar_wait(accum_bar, 0);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) {
        if (lane == 0) atomicOr(args.status, HX_FLAG_WAIT_TIMEOUT);
      } else if (!IN_BLOCKS) {
        tc_fence_after();
        if (CLUSTERS && args.cluster > 1)
          leave_part<BN>(reinterpret_cast<float*>(smem), lane_address, quarter * 32 + lane,
                         min(BN, args.tokens - token0));
        else
          write_tile<BN, EPI>(args.out, args.ldo, args.tokens, args.features, lane_address, feature,
                              token0, args.activation, args.gate_limit, args.gate_bias, args.up_bias,
                              args.softcap);
      }
    }
  }
  if (CLUSTERS && args.cluster > 1) {      // (every CTA of a cluster comes here, whatever went wrong)
    __syncthreads();
    cluster_sync();
    if (warp >= 2)
      gather_parts<BN, EPI>(args, reinterpret_cast<const float*>(smem), static_cast<int>(cluster_rank()),
                            (warp & 3) * 32 + lane, feature0 + (warp & 3) * 32 + lane, token0);
    __syncthreads();
    cluster_sync();      // nobody's part is read any more
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLUMNS);
  }
}

// ------------------------------------------------- persistent kernel for prompt portions
//
// With hundreds of tokens the product is compute bound, and the tile's epilogue (reading a
// 128 x 256 accumulator back, converting, storing) takes a good part of the time of its main
// loop.  Here one CTA per SM walks a list of work units: all of shared memory is one ring of
// operand stages that runs on across units, tensor memory holds TWO accumulators of 256
// columns, and the epilogue warps drain one while the MMA warp fills the other.
//
// The tile is turned round with respect to the kernel above: 128 TOKENS are the MMA's M
// side and 256 weight rows its N side, so a thread of the epilogue owns one token and finds
// 256 consecutive features of it in its lane of tensor memory: it writes them 16 at a time
// with 16-byte stores (or 16-byte reductions into the float32 residual), which the memory
// system takes several times faster than the two-byte stores of a feature-per-thread layout.
// For SwiGLU the N side is 128 gate rows followed by the matching 128 up rows of the fused
// matrix: gate and up of a feature sit side by side in the thread's own lane.
//
// The add epilogue does not add at the memory side here (float32 reductions reach only about
// 1.8 TB/s in the L2, a quarter of what this product would need): it reads the output's old values, the
// first of them while the unit's products run, adds and stores.  One writer per element: the result is
// deterministic.  Old values loaded INTO the accumulator before the products took 65.6 us at 2,048 x 4,096 x 4,096,
// 137.2 at depth 11,008 and 201.5 at 1,900 x 5,120 x 13,824 (weights and inputs out of the L2); so it is 61.4,
// 131.0 and 194.6, and depths of 64 and 512 take 32.8 and 35.6 us after 33.6 and 35.6.
//
// Tiles are dealt round-robin with the token tile varying fastest, so the CTAs that run side
// by side read the same weight tiles at the same time, once from DRAM.

// Floats between rows, and bytes, of what the add epilogue's warps exchange (see add_tile).
constexpr int ADD_STRIDE = 36;
constexpr int ADD_BYTES = 4 * 32 * ADD_STRIDE * 4;      // of the four epilogue warps

struct PersistentConfig {
  static constexpr int kRowsA = BM;              // tokens
  static constexpr int kRowsB = 2 * BM;          // weight rows: the accumulator's columns
  static constexpr int kBytesA = kRowsA * BK * 2;
  static constexpr int kBytesB = kRowsB * BK * 2;
  static constexpr int kStageBytes = kBytesA + kBytesB;
  static constexpr int kStages = 200 * 1024 / kStageBytes;
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*alignment*/ + 256 /*barriers*/ + ADD_BYTES;
  static constexpr int kBufferColumns = 256;     // one accumulator per half of tensor memory
  static constexpr int kTmemColumns = 512;
};

// What the rotary/append epilogue needs beyond the product: the output row is
// [q heads | k heads | v heads], each head `head_dim` wide (a multiple of 16, so the 16
// features a thread handles at a time lie in one head).  Queries are rotated and stored to
// `out`; keys are rotated and, like the values, written into the token's slot of its page
// (k_cache == nullptr: the caller owns no cache, keys and values are dropped).  Pairs are
// adjacent coordinates (2p, 2p + 1); the first `rotary_dim` coordinates of a head rotate.
struct RopeArgs {
  const int* positions;
  const int* token_request;
  const int* request_table_row;
  const int* block_tables;
  int table_stride;
  __nv_bfloat16* k_cache;
  __nv_bfloat16* v_cache;
  const float* cos_table;      // [table_positions][rotary_dim / 2]
  const float* sin_table;
  int table_positions;
  int heads, kv_heads, head_dim, rotary_dim, page_size, num_pages;
  int shared_values;           // no v heads: the values are the keys before the rotation
};

#ifndef HX_GEMM_STREAM_K
#define HX_GEMM_STREAM_K 1      // 0: every unit of the persistent kernel is a whole tile
#endif

struct PersistentArgs {
  void* out;
  int ldo;
  int tokens;
  int features;
  int depth;
  int up_row_offset;
  int k_tiles;                // > 0: the weights are stored as tiles, this many along k
  int token_tiles;            // tiles along the tokens
  int units;                  // token_tiles * feature tiles
  int k_blocks;               // per tile
  int* status;
  RopeArgs rope;              // EPI_ROPE_APPEND only
  int whole_rounds;           // >= 0: the tiles behind this many whole rounds are shared out by
                              // k-blocks (add epilogue only); -1: every unit is a whole tile
  int activation;             // gated epilogue: what the gate passes through (HxGateActivation)
  // Grouped product (see GemmArgs): token tile t multiplies with group tile_group[t] of the
  // weight matrix; a unit of a tile with a negative group loads, multiplies and writes nothing.
  const int* tile_group;
  int group_rows;
  float gate_limit = 0.0f;    // gated epilogue: the limit of HX_GATE_CLAMPED_SIGMOID
  // gated epilogue: float32 biases of the gate and the up rows, [features] each (null: none)
  const float* gate_bias = nullptr;
  const float* up_bias = nullptr;
  float softcap = 0.0f;       // float32 store: see level_off
  int tail_ctas = 0;          // CTAs that share the tiles behind the whole rounds
  int tail_pieces = 1;        // pairs: the tiles behind the whole rounds are cut into so many pieces
  // One small product per head (heads > 1): the feature tiles come head by head, head_tiles of
  // them; head h multiplies the columns of x from h * head_x on with the rows of the weights from
  // h * features on and writes its `features` columns from h * head_out on.
  int heads = 1;
  int head_tiles = 0, head_x = 0, head_out = 0;
};

// What a CTA works on at a time: a tile, or (`partial`) a run of k-blocks of a tile that
// other CTAs hold the rest of.
struct Unit {
  int token_tile, feature_tile, kb_begin, kb_end;
  bool partial;
  int pieces, piece;      // pairs: which of so many pieces of the tile's columns
};

// The grid walks the tiles round by round.  The last round seldom fills the grid: 256 tiles
// on 148 CTAs are 1.73 rounds that cost 2.  Where the epilogue ADDS into a float32 output the
// order of the sum is free, so the tiles of that last round are laid end to end as one list
// of k-blocks and the first `tail_ctas` CTAs take an equal run of it each (one or two pieces of
// tiles), which they add to the output with atomic adds; whole tiles keep the plain
// read-add-store.
// `worker` of `grid`: a CTA of the grid, or a pair of them.
__device__ __forceinline__ bool unit_at(const PersistentArgs& a, int iteration, Unit& u, int worker,
                                        int grid) {
  int index;
  u.pieces = 1;
  u.piece = 0;
  if (a.tail_pieces > 1 && iteration == a.whole_rounds) {
    if (worker >= (a.units - a.whole_rounds * grid) * a.tail_pieces) return false;
    index = a.whole_rounds * grid + worker / a.tail_pieces;
    u.pieces = a.tail_pieces;
    u.piece = worker % a.tail_pieces;
    u.kb_begin = 0;
    u.kb_end = a.k_blocks;
    u.partial = false;
  } else if (a.tail_pieces > 1 && iteration > a.whole_rounds) {
    return false;
  } else if (a.whole_rounds < 0 || iteration < a.whole_rounds) {
    index = worker + iteration * grid;
    if (index >= a.units) return false;
    u.kb_begin = 0;
    u.kb_end = a.k_blocks;
    u.partial = false;
  } else {
    const int first = a.whole_rounds * grid;
    if (worker >= a.tail_ctas) return false;
    const long long blocks = static_cast<long long>(a.units - first) * a.k_blocks;
    const long long begin = blocks * worker / a.tail_ctas;
    const long long end = blocks * (worker + 1) / a.tail_ctas;
    const long long tile = begin / a.k_blocks + (iteration - a.whole_rounds);
    const long long from = max(begin, tile * a.k_blocks);
    const long long to = min(end, (tile + 1) * a.k_blocks);
    if (from >= to) return false;
    index = first + static_cast<int>(tile);
    u.kb_begin = static_cast<int>(from - tile * a.k_blocks);
    u.kb_end = static_cast<int>(to - tile * a.k_blocks);
    u.partial = u.kb_begin != 0 || u.kb_end != a.k_blocks;
  }
  u.token_tile = index % a.token_tiles;
  u.feature_tile = index / a.token_tiles;
  return true;
}

// The add epilogue of a warp's 32 tokens, 32 columns at a time, the next 32 on their way.  A thread finds a token's
// sums in its lane of tensor memory; in the output 32 columns of a token are a line of 128 bytes, which eight threads
// read and write with 16 bytes each.  So the sums change places in shared memory (rows ADD_STRIDE floats apart use
// different banks).  With a token a thread, every access 32 lines, 2,048 x 4,096 took 35.8 us at a depth of 64 and
// 39.7 at 512, so 32.8 and 35.6; at 4,096 64.5, so 61.4.

// Old values: four columns from `column` on of tokens first + 4 i + lane / 8 (zeros behind the output's edges).
__device__ __forceinline__ void load_old(const float* out, int ldo, int features, int first, int tokens, int column,
                                         bool wide, float4 (&v)[8]) {
  const int lane = threadIdx.x & 31, at = column + 4 * (lane & 7);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int token = first + 4 * i + (lane >> 3);
    v[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (token < tokens) {
      const float* from = out + static_cast<size_t>(token) * ldo + at;
      if (wide && at + 4 <= features) {
        v[i] = *reinterpret_cast<const float4*>(from);
      } else {
        if (at < features) v[i].x = from[0];
        if (at + 1 < features) v[i].y = from[1];
        if (at + 2 < features) v[i].z = from[2];
        if (at + 3 < features) v[i].w = from[3];
      }
    }
  }
}

// 256 columns from feature0 on; `old` holds the first 32.  All lanes of the warp, with the same arguments.
__device__ __forceinline__ void add_tile(float* out, int ldo, int features, uint32_t lane_address, int first,
                                         int tokens, int feature0, bool wide, float* exchange, float4 (&old)[8]) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int column = 0; column < 2 * BM; column += 32) {
    if (feature0 + column >= features) break;      // uniform over the warp
    float4 next[8];
    if (column + 32 < 2 * BM) load_old(out, ldo, features, first, tokens, feature0 + column + 32, wide, next);
    uint32_t acc[2][16];
    tmem_load16_issue(lane_address + column, acc[0]);
    tmem_load16_issue(lane_address + column + 16, acc[1]);
    tmem_load_wait();
    __syncwarp();      // (the last columns are read)
#pragma unroll
    for (int j = 0; j < 8; ++j)
      *reinterpret_cast<uint4*>(exchange + lane * ADD_STRIDE + 4 * j) =
          make_uint4(acc[j / 4][4 * j % 16], acc[j / 4][4 * j % 16 + 1], acc[j / 4][4 * j % 16 + 2],
                     acc[j / 4][4 * j % 16 + 3]);
    __syncwarp();
    const int at = feature0 + column + 4 * (lane & 7);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = 4 * i + (lane >> 3), token = first + row;
      const float4 sum = *reinterpret_cast<const float4*>(exchange + row * ADD_STRIDE + 4 * (lane & 7));
      const float4 v = make_float4(old[i].x + sum.x, old[i].y + sum.y, old[i].z + sum.z, old[i].w + sum.w);
      if (token < tokens) {
        float* to = out + static_cast<size_t>(token) * ldo + at;
        if (wide && at + 4 <= features) {
          *reinterpret_cast<float4*>(to) = v;
        } else {
          if (at < features) to[0] = v.x;
          if (at + 1 < features) to[1] = v.y;
          if (at + 2 < features) to[2] = v.z;
          if (at + 3 < features) to[3] = v.w;
        }
      }
      old[i] = next[i];
    }
  }
}

// This thread's token: `columns` features starting at feature0, 16 at a time, from its lane of
// the accumulator.  With SwiGLU the accumulator holds `columns` gate columns, then the up columns.
template <int EPI>
__device__ __forceinline__ void write_row(int columns, void* out, int ldo, int features, uint32_t lane_address,
                                          int token, int tokens, int feature0, int activation,
                                          float gate_limit, const float* gate_bias,
                                          const float* up_bias, float softcap) {
  using Element = typename std::conditional<EPI == EPI_STORE_BF16 || EPI == EPI_SWIGLU,
                                            __nv_bfloat16, float>::type;
  const bool wide = (ldo % (16 / static_cast<int>(sizeof(Element))) == 0) &&
                    ((reinterpret_cast<uintptr_t>(out) & 15) == 0);
#pragma unroll 1
  for (int column = 0; column < columns; column += 16) {
    if (feature0 + column >= features) break;      // uniform over the warp
    float acc[16];
    tmem_load16(lane_address + column, acc);
    if (EPI == EPI_SWIGLU) {
      float up[16];
      tmem_load16(lane_address + columns + column, up);
      if (gate_bias != nullptr || up_bias != nullptr) {
        // this thread's 16 features: their biases (the same for every token of the tile)
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int feature = feature0 + column + j;
          if (feature < features) {
            if (gate_bias != nullptr) acc[j] += gate_bias[feature];
            if (up_bias != nullptr) up[j] += up_bias[feature];
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) acc[j] = hx_gated_fast(acc[j], up[j], activation, gate_limit);
    }
    if (EPI == EPI_STORE_F32 && softcap > 0.0f) {
#pragma unroll
      for (int j = 0; j < 16; ++j) acc[j] = level_off(acc[j], softcap);
    }
    if (token >= tokens) continue;
    Element* row = static_cast<Element*>(out) + static_cast<size_t>(token) * ldo + feature0 + column;
    if (wide && feature0 + column + 16 <= features) {
      if constexpr (std::is_same<Element, __nv_bfloat16>::value) {
        uint4 packed[2];
        __nv_bfloat162* pairs = reinterpret_cast<__nv_bfloat162*>(packed);
#pragma unroll
        for (int j = 0; j < 8; ++j) pairs[j] = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
        reinterpret_cast<uint4*>(row)[0] = packed[0];
        reinterpret_cast<uint4*>(row)[1] = packed[1];
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          reinterpret_cast<float4*>(row)[j] =
              make_float4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (feature0 + column + j < features) {
          if constexpr (std::is_same<Element, __nv_bfloat16>::value) {
            row[j] = __float2bfloat16_rn(acc[j]);
          } else {
            row[j] = acc[j];
          }
        }
      }
    }
  }
}

// The rotary/append epilogue for this thread's token: the same arithmetic as the separate
// kernel (hx_rope_append) applied to the product rounded to bfloat16, as the plain store
// would have rounded it: rotation in float32 from the cos/sin table, one more rounding.
__device__ __forceinline__ void write_row_rope(int columns, const PersistentArgs& a,
                                               uint32_t lane_address, int token, int feature0) {
  const RopeArgs& r = a.rope;
  const bool live = token < a.tokens;
  const int half = r.rotary_dim / 2;
  const float* cos_row = r.cos_table;
  const float* sin_row = r.sin_table;
  int page = -1, slot = 0;
  if (live) {
    const int position = r.positions[token];
    const int table_position = min(max(position, 0), r.table_positions - 1);
    if (table_position != position && r.rotary_dim > 0 && feature0 == 0 && a.status != nullptr)
      atomicOr(a.status, HX_FLAG_BAD_POSITION);
    cos_row += static_cast<size_t>(table_position) * half;
    sin_row += static_cast<size_t>(table_position) * half;
    if (r.k_cache != nullptr) {
      const int table_row = r.request_table_row[r.token_request[token]];
      page = r.block_tables[static_cast<size_t>(table_row) * r.table_stride + position / r.page_size];
      slot = position % r.page_size;
      if (page < 0 || page >= r.num_pages) {
        atomicOr(a.status, HX_FLAG_BAD_PAGE);
        page = -1;
      }
    }
  }
  const int q_features = r.heads * r.head_dim;
  const int k_end = q_features + r.kv_heads * r.head_dim;
  const bool wide_table = half % 4 == 0 &&
                          ((reinterpret_cast<uintptr_t>(r.cos_table) |
                            reinterpret_cast<uintptr_t>(r.sin_table)) & 15) == 0;
#pragma unroll 1
  for (int column = 0; column < columns; column += 16) {
    const int feature = feature0 + column;
    if (feature >= a.features) break;      // uniform over the warp
    float x[16];
    tmem_load16(lane_address + column, x);
    if (!live) continue;
    const bool is_query = feature < q_features;
    const bool is_key = !is_query && feature < k_end;
    const int inside = feature - (is_query ? 0 : (is_key ? q_features : k_end));
    const int head = inside / r.head_dim;
    const int d0 = inside - head * r.head_dim;
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = __bfloat162float(__float2bfloat16_rn(x[j]));
    if (r.shared_values && is_key && page >= 0) {
      uint4 packed[2];
      __nv_bfloat162* pairs = reinterpret_cast<__nv_bfloat162*>(packed);
#pragma unroll
      for (int j = 0; j < 8; ++j) pairs[j] = __floats2bfloat162_rn(x[2 * j], x[2 * j + 1]);
      *reinterpret_cast<uint4*>(r.v_cache + hx_cache_offset(page, head, slot, d0, r.kv_heads,
                                                            r.page_size, r.head_dim, 8)) = packed[0];
      *reinterpret_cast<uint4*>(r.v_cache + hx_cache_offset(page, head, slot, d0 + 8, r.kv_heads,
                                                            r.page_size, r.head_dim, 8)) = packed[1];
    }
    if ((is_query || is_key) && d0 < r.rotary_dim) {
      // the eight angles of this piece: four 16-byte loads where the table's rows allow it
      // (every lane reads another row of the table, so the number of loads is what counts)
      float c[8], sn[8];
      if (wide_table && d0 + 16 <= r.rotary_dim) {
        const float4 c0 = __ldg(reinterpret_cast<const float4*>(cos_row + d0 / 2));
        const float4 c1 = __ldg(reinterpret_cast<const float4*>(cos_row + d0 / 2 + 4));
        const float4 s0 = __ldg(reinterpret_cast<const float4*>(sin_row + d0 / 2));
        const float4 s1 = __ldg(reinterpret_cast<const float4*>(sin_row + d0 / 2 + 4));
        c[0] = c0.x; c[1] = c0.y; c[2] = c0.z; c[3] = c0.w;
        c[4] = c1.x; c[5] = c1.y; c[6] = c1.z; c[7] = c1.w;
        sn[0] = s0.x; sn[1] = s0.y; sn[2] = s0.z; sn[3] = s0.w;
        sn[4] = s1.x; sn[5] = s1.y; sn[6] = s1.z; sn[7] = s1.w;
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const bool rotates = d0 + 2 * i + 1 < r.rotary_dim;
          c[i] = rotates ? __ldg(cos_row + d0 / 2 + i) : 1.0f;
          sn[i] = rotates ? __ldg(sin_row + d0 / 2 + i) : 0.0f;
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float u = x[2 * i], v = x[2 * i + 1];
        x[2 * i] = u * c[i] - v * sn[i];
        x[2 * i + 1] = u * sn[i] + v * c[i];
      }
    }
    uint4 packed[2];
    __nv_bfloat162* pairs = reinterpret_cast<__nv_bfloat162*>(packed);
#pragma unroll
    for (int j = 0; j < 8; ++j) pairs[j] = __floats2bfloat162_rn(x[2 * j], x[2 * j + 1]);
    if (is_query) {
      uint4* row = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(a.out) +
                                            static_cast<size_t>(token) * a.ldo + feature);
      row[0] = packed[0];
      row[1] = packed[1];
    } else if (page >= 0) {
      __nv_bfloat16* cache = is_key ? r.k_cache : r.v_cache;
      *reinterpret_cast<uint4*>(cache + hx_cache_offset(page, head, slot, d0, r.kv_heads,
                                                        r.page_size, r.head_dim, 8)) = packed[0];
      *reinterpret_cast<uint4*>(cache + hx_cache_offset(page, head, slot, d0 + 8, r.kv_heads,
                                                        r.page_size, r.head_dim, 8)) = packed[1];
    }
  }
}

// The piece of a tile that a partial unit computed: added to the float32 output with atomic
// adds (four values at a time where the row allows).
__device__ __forceinline__ void add_row_atomically(float* out, int ldo, int features,
                                                   uint32_t lane_address, int token, int tokens,
                                                   int feature0) {
  const bool wide = (ldo % 4 == 0) && ((reinterpret_cast<uintptr_t>(out) & 15) == 0);
#pragma unroll 1
  for (int column = 0; column < 2 * BM; column += 16) {
    if (feature0 + column >= features) break;      // uniform over the warp
    float acc[16];
    tmem_load16(lane_address + column, acc);
    if (token >= tokens) continue;
    float* row = out + static_cast<size_t>(token) * ldo + feature0 + column;
    if (wide && feature0 + column + 16 <= features) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(row + 4 * j),
                     "f"(acc[4 * j]), "f"(acc[4 * j + 1]), "f"(acc[4 * j + 2]),
                     "f"(acc[4 * j + 3]) : "memory");
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (feature0 + column + j < features) atomicAdd(row + j, acc[j]);
    }
  }
}

template <int EPI>
__global__ __launch_bounds__(THREADS) void gemm_tc_persistent_kernel(
    const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
    const PersistentArgs args) {
  using Config = PersistentConfig;
  constexpr int STAGES = Config::kStages;
  // features of the output per tile, and where the second half of the N operand comes from
  constexpr int FEATURES = EPI == EPI_SWIGLU ? BM : 2 * BM;

  hx_pdl_trigger();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * Config::kStageBytes);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tmem_full_bar = empty_bar + STAGES;      // [2]: the accumulator is complete
  uint64_t* tmem_empty_bar = tmem_full_bar + 2;      // [2]: the epilogue has read it
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(tmem_empty_bar + 2);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int worker = blockIdx.x, workers = gridDim.x;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full_bar[b], 1);
      mbar_init(&tmem_empty_bar[b], 4);      // one arrival per epilogue warp
    }
    *failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_holder, Config::kTmemColumns);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  hx_pdl_wait();

  if (warp == 0) {
    // -------------------------------------------------------------- TMA producer
    if (hx_elect_one()) {
      uint32_t fill = 0;      // stages filled so far, over all units
      Unit unit;
      for (int iteration = 0; unit_at(args, iteration, unit, worker, workers) && !*failed; ++iteration) {
        int group_row0 = 0, kb_end = unit.kb_end;
        if (args.tile_group != nullptr) {
          const int group = args.tile_group[unit.token_tile];
          if (group < 0) kb_end = unit.kb_begin;
          else group_row0 = group * args.group_rows;
        }
        int feature0 = group_row0 + unit.feature_tile * FEATURES, k_first = 0;
        if (EPI == EPI_STORE_BF16 && args.heads > 1) {
          const int head = unit.feature_tile / args.head_tiles;
          feature0 = head * args.features + (unit.feature_tile - head * args.head_tiles) * FEATURES;
          k_first = head * args.head_x;
        }
        const int second_half = EPI == EPI_SWIGLU ? args.up_row_offset + feature0 : feature0 + BM;
        const int token0 = unit.token_tile * BM;
        for (int kb = unit.kb_begin; kb < kb_end; ++kb, ++fill) {
          const int s = fill % STAGES;
          const uint32_t round = fill / STAGES;
          if (!mbar_wait(&empty_bar[s], (round & 1u) ^ 1u)) {
            atomicOr(args.status, HX_FLAG_WAIT_TIMEOUT);
            *failed = 1;
            break;
          }
          uint8_t* stage = smem + s * Config::kStageBytes;
          mbar_expect_tx(&full_bar[s], Config::kStageBytes);
          tma_load_2d(stage, &map_x, &full_bar[s], k_first + kb * BK, token0);
          load_weight_box(stage + Config::kBytesA, &map_w, &full_bar[s], feature0, kb, args.k_tiles);
          load_weight_box(stage + Config::kBytesA + BM * BK * 2, &map_w, &full_bar[s], second_half,
                          kb, args.k_tiles);
        }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    if (hx_elect_one()) {
      constexpr uint32_t idesc = make_idesc(BM, Config::kRowsB);
      uint32_t drained = 0;      // stages consumed so far, over all units
      Unit unit;
      for (int iteration = 0; unit_at(args, iteration, unit, worker, workers) && !*failed; ++iteration) {
        const int buffer = iteration & 1;
        const uint32_t use = static_cast<uint32_t>(iteration >> 1);
        // the epilogue must have read this accumulator's previous unit
        if (!mbar_wait(&tmem_empty_bar[buffer], (use & 1u) ^ 1u)) {
          atomicOr(args.status, HX_FLAG_WAIT_TIMEOUT);
          *failed = 1;
          break;
        }
        tc_fence_after();
        const uint32_t accumulator = tmem_base + buffer * Config::kBufferColumns;
        const bool skipped = args.tile_group != nullptr && args.tile_group[unit.token_tile] < 0;
        for (int kb = unit.kb_begin; kb < (skipped ? unit.kb_begin : unit.kb_end); ++kb, ++drained) {
          const int s = drained % STAGES;
          const uint32_t round = drained / STAGES;
          if (!mbar_wait(&full_bar[s], round & 1u)) {
            atomicOr(args.status, HX_FLAG_WAIT_TIMEOUT);
            *failed = 1;
            break;
          }
          tc_fence_after();
          const uint32_t stage = smem_u32(smem + s * Config::kStageBytes);
          const uint64_t desc_a = make_smem_desc(stage);
          const uint64_t desc_b = make_smem_desc(stage + Config::kBytesA);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t step = static_cast<uint64_t>(k * UMMA_K * 2 >> 4);
            const uint32_t accumulate = (kb > unit.kb_begin || k > 0) ? 1u : 0u;
            umma_bf16(accumulator, desc_a + step, desc_b + step, idesc, accumulate);
          }
          umma_commit(&empty_bar[s]);
        }
        if (*failed) break;
        umma_commit(&tmem_full_bar[buffer]);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int quarter = warp & 3;     // tensor-memory lanes [32 * quarter, 32 * quarter + 32)
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    Unit unit;
    // the add epilogue's: whether output rows take 16-byte accesses, and where sums change places
    const bool wide = args.ldo % 4 == 0 && (reinterpret_cast<uintptr_t>(args.out) & 15) == 0;
    float* exchange = reinterpret_cast<float*>(smem + STAGES * Config::kStageBytes + 256);
    for (int iteration = 0; unit_at(args, iteration, unit, worker, workers) && !*failed; ++iteration) {
      const int buffer = iteration & 1;
      const uint32_t use = static_cast<uint32_t>(iteration >> 1);
      bool ok = true;
      float4 old[8];
      if (EPI == EPI_ADD_F32 && !unit.partial)      // on their way while the unit's products run
        load_old(static_cast<const float*>(args.out), args.ldo, args.features, unit.token_tile * BM + quarter * 32,
                 args.tokens, unit.feature_tile * FEATURES, wide, old);
      if (lane == 0) ok = mbar_wait(&tmem_full_bar[buffer], use & 1u);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) {
        if (lane == 0) {
          atomicOr(args.status, HX_FLAG_WAIT_TIMEOUT);
          *failed = 1;
        }
        break;
      }
      tc_fence_after();
      if constexpr (EPI == EPI_ROPE_APPEND) {
        write_row_rope(FEATURES, args, lane_base + buffer * Config::kBufferColumns,
                       unit.token_tile * BM + quarter * 32 + lane, unit.feature_tile * FEATURES);
      } else if constexpr (EPI == EPI_ADD_F32) {
        if (!unit.partial)
          add_tile(static_cast<float*>(args.out), args.ldo, args.features,
                   lane_base + buffer * Config::kBufferColumns, unit.token_tile * BM + quarter * 32, args.tokens,
                   unit.feature_tile * FEATURES, wide, exchange + quarter * 32 * ADD_STRIDE, old);
        else
          add_row_atomically(static_cast<float*>(args.out), args.ldo, args.features,
                             lane_base + buffer * Config::kBufferColumns,
                             unit.token_tile * BM + quarter * 32 + lane, args.tokens,
                             unit.feature_tile * FEATURES);
      } else if (EPI == EPI_STORE_BF16 && args.heads > 1) {
        const int head = unit.feature_tile / args.head_tiles;
        write_row<EPI>(FEATURES, static_cast<__nv_bfloat16*>(args.out) + static_cast<size_t>(head) * args.head_out,
                       args.ldo, args.features, lane_base + buffer * Config::kBufferColumns,
                       unit.token_tile * BM + quarter * 32 + lane, args.tokens,
                       (unit.feature_tile - head * args.head_tiles) * FEATURES, args.activation,
                       args.gate_limit, args.gate_bias, args.up_bias, args.softcap);
      } else if (args.tile_group == nullptr || args.tile_group[unit.token_tile] >= 0) {
        write_row<EPI>(FEATURES, args.out, args.ldo, args.features,
                       lane_base + buffer * Config::kBufferColumns,
                       unit.token_tile * BM + quarter * 32 + lane, args.tokens,
                       unit.feature_tile * FEATURES, args.activation, args.gate_limit,
                       args.gate_bias, args.up_bias, args.softcap);
      }
      // every lane's tcgen05.ld has completed (the loads are waited for where they are
      // issued): hand the accumulator back
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty_bar[buffer]);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Config::kTmemColumns);
  }
}

// ------------------------------------------------------------- the same by pairs of CTAs
//
// A tile of 128 tokens by 256 weight rows reads 48 KB of operands per k-block, at the tensor cores'
// rate about what an SM gets from the L2, and every SM multiplies by weights that it has brought in
// for itself.  Here two CTAs share a tile of 256 tokens: each brings its own 128 tokens and HALF of
// the weight rows (for SwiGLU: the gate rows, and the up rows), and tcgen05.mma.cta_group::2 reads
// both halves: 32 KB a k-block and CTA, so six stages instead of four.  The leader (the even CTA)
// issues the products for both; either CTA's accumulators hold its own 128 tokens, so the epilogues
// are those of the kernel above.  Where the last round has few tiles and the epilogue does not add,
// they are cut into two or four pieces of columns, a pair each.
// Measured (2,048 tokens, alone, one CTA a tile and pairs): [12,288 x 4,096] 155.8 -> 139.6 us (1,476
// TFLOP/s), sums by [4,096 x 4,096] 71.3 -> 55.7, gate and up [22,016 x 4,096] 270.3 -> 256.5, sums by
// [4,096 x 11,008] 173.2 -> 167.9; 512 tokens 54.8 -> 48.2, 25.4 -> 24.6, 90.2 -> 79.9, 66.7 -> 54.5.
struct PairConfig {
  static constexpr int kBytesA = BM * BK * 2;    // this CTA's tokens
  static constexpr int kBytesB = BM * BK * 2;    // its half of the weight rows
  static constexpr int kStageBytes = kBytesA + kBytesB;
  static constexpr int kStages = 6;
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*alignment*/ + 256 /*barriers*/ + ADD_BYTES;
};

template <int EPI>
__global__ __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS) void gemm_tc_pair_kernel(
    const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_w_piece,
    const __grid_constant__ CUtensorMap map_x, const PersistentArgs args) {
  using Config = PairConfig;
  constexpr int STAGES = Config::kStages;
  constexpr int FEATURES = EPI == EPI_SWIGLU ? BM : 2 * BM;
  constexpr int kBufferColumns = PersistentConfig::kBufferColumns;

  hx_pdl_trigger();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * Config::kStageBytes);  // leader's count
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tmem_full_bar = empty_bar + STAGES;      // [2]
  uint64_t* tmem_empty_bar = tmem_full_bar + 2;      // [2]: leader's count, of both CTAs' epilogues
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(tmem_empty_bar + 2);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_holder + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_rank());
  const int worker = blockIdx.x >> 1, workers = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full_bar[b], 1);
      mbar_init(&tmem_empty_bar[b], 8);      // one arrival per epilogue warp of both CTAs
    }
    *failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) tmem_alloc_pair(tmem_holder, PersistentConfig::kTmemColumns);
  tc_fence_before();
  __syncthreads();
  cluster_sync();      // nothing arrives at the other CTA's barriers before they are there
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  hx_pdl_wait();

  if (warp == 0) {
    // -------------------------------------------------------------- TMA producer
    if (hx_elect_one()) {
      uint32_t fill = 0;      // stages filled so far, over all units
      Unit unit;
      for (int iteration = 0; unit_at(args, iteration, unit, worker, workers) && !*failed; ++iteration) {
        const int rows = BM / unit.pieces;      // this CTA's half of the tile's (or piece's) rows
        const int feature0 = unit.feature_tile * FEATURES + unit.piece * (FEATURES / unit.pieces);
        const int weight_row = rank == 0 ? feature0
                               : EPI == EPI_SWIGLU ? args.up_row_offset + feature0 : feature0 + rows;
        const CUtensorMap* map = unit.pieces > 1 ? &map_w_piece : &map_w;
        const uint32_t bytes = Config::kBytesA + static_cast<uint32_t>(rows) * BK * 2;
        // tiled weights: a piece lies inside one stored tile
        const int tile_row = args.k_tiles > 0 ? (weight_row / BM) * args.k_tiles * BM + weight_row % BM : 0;
        const int token0 = unit.token_tile * 2 * BM + rank * BM;
        for (int kb = unit.kb_begin; kb < unit.kb_end; ++kb, ++fill) {
          const int s = fill % STAGES;
          if (!mbar_wait(&empty_bar[s], ((fill / STAGES) & 1u) ^ 1u)) {
            atomicOr(args.status, HX_FLAG_WAIT_TIMEOUT);
            *failed = 1;
            break;
          }
          uint8_t* stage = smem + s * Config::kStageBytes;
          if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * bytes);
          const uint32_t bar = cluster_address(&full_bar[s], 0);
          tma_load_2d_pair(stage, &map_x, bar, kb * BK, token0);
          if (args.k_tiles > 0)
            tma_load_2d_pair(stage + Config::kBytesA, map, bar, 0, tile_row + kb * BM);
          else
            tma_load_2d_pair(stage + Config::kBytesA, map, bar, kb * BK, weight_row);
        }
      }
      // the leader's last arrivals at this CTA's barriers, before the CTA may end
      for (uint32_t last = fill > STAGES ? fill - STAGES : 0; last < fill && !*failed; ++last)
        if (!mbar_wait(&empty_bar[last % STAGES], (last / STAGES) & 1u)) {
          atomicOr(args.status, HX_FLAG_WAIT_TIMEOUT);
          *failed = 1;
        }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    if (rank == 0 && hx_elect_one()) {
      uint32_t drained = 0;
      Unit unit;
      for (int iteration = 0; unit_at(args, iteration, unit, worker, workers) && !*failed; ++iteration) {
        const int buffer = iteration & 1;
        const uint32_t use = static_cast<uint32_t>(iteration >> 1);
        if (!mbar_wait_cluster(&tmem_empty_bar[buffer], (use & 1u) ^ 1u)) {
          atomicOr(args.status, HX_FLAG_WAIT_TIMEOUT);
          *failed = 1;
          break;
        }
        tc_fence_after();
        const uint32_t accumulator = tmem_base + buffer * kBufferColumns;
        const uint32_t idesc = make_idesc(2 * BM, 2 * BM / unit.pieces);
        for (int kb = unit.kb_begin; kb < unit.kb_end; ++kb, ++drained) {
          const int s = drained % STAGES;
          if (!mbar_wait_cluster(&full_bar[s], (drained / STAGES) & 1u)) {
            atomicOr(args.status, HX_FLAG_WAIT_TIMEOUT);
            *failed = 1;
            break;
          }
          tc_fence_after();
          const uint32_t stage = smem_u32(smem + s * Config::kStageBytes);
          const uint64_t desc_a = make_smem_desc(stage);
          const uint64_t desc_b = make_smem_desc(stage + Config::kBytesA);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t step = static_cast<uint64_t>(k * UMMA_K * 2 >> 4);
            const uint32_t accumulate = (kb > unit.kb_begin || k > 0) ? 1u : 0u;
            umma_bf16_pair(accumulator, desc_a + step, desc_b + step, idesc, accumulate);
          }
          umma_commit_pair(&empty_bar[s]);
        }
        if (*failed) break;
        umma_commit_pair(&tmem_full_bar[buffer]);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int quarter = warp & 3;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    const int row = rank * BM + quarter * 32 + lane;      // of the tile's 256 tokens
    Unit unit;
    auto hand_over = [&](int buffer) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(cluster_address(&tmem_empty_bar[buffer], 0));
    };
    // the add epilogue's: whether output rows take 16-byte accesses, and where sums change places
    const bool wide = args.ldo % 4 == 0 && (reinterpret_cast<uintptr_t>(args.out) & 15) == 0;
    float* exchange = reinterpret_cast<float*>(smem + STAGES * Config::kStageBytes + 256);
    for (int iteration = 0; unit_at(args, iteration, unit, worker, workers) && !*failed; ++iteration) {
      const int buffer = iteration & 1;
      const uint32_t use = static_cast<uint32_t>(iteration >> 1);
      bool ok = true;
      float4 old[8];
      if (EPI == EPI_ADD_F32 && !unit.partial)      // on their way while the unit's products run
        load_old(static_cast<const float*>(args.out), args.ldo, args.features,
                 unit.token_tile * 2 * BM + row - lane, args.tokens, unit.feature_tile * FEATURES, wide, old);
      if (lane == 0) ok = mbar_wait_cluster(&tmem_full_bar[buffer], use & 1u);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) {
        if (lane == 0) {
          atomicOr(args.status, HX_FLAG_WAIT_TIMEOUT);
          *failed = 1;
        }
        break;
      }
      tc_fence_after();
      const uint32_t accumulator = lane_base + buffer * kBufferColumns;
      const int columns = FEATURES / unit.pieces;
      const int token = unit.token_tile * 2 * BM + row;
      const int feature0 = unit.feature_tile * FEATURES + unit.piece * columns;
      if constexpr (EPI == EPI_ROPE_APPEND) {
        write_row_rope(columns, args, accumulator, token, feature0);
      } else if constexpr (EPI == EPI_ADD_F32) {
        if (!unit.partial)
          add_tile(static_cast<float*>(args.out), args.ldo, args.features, accumulator, token - lane, args.tokens,
                   feature0, wide, exchange + quarter * 32 * ADD_STRIDE, old);
        else
          add_row_atomically(static_cast<float*>(args.out), args.ldo, args.features, accumulator, token,
                             args.tokens, feature0);
      } else {
        write_row<EPI>(columns, args.out, args.ldo, args.features, accumulator, token, args.tokens, feature0,
                       args.activation, args.gate_limit, args.gate_bias, args.up_bias, args.softcap);
      }
      hand_over(buffer);
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync();      // neither CTA's memory is read or arrived at any more
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, PersistentConfig::kTmemColumns);
  }
}

// ----------------------------------------------------------------- host side

// The map of a matrix of bfloat16 whose boxes are `box_rows` rows of one k-block.
int get_tensor_map(const void* base, uint64_t rows, uint64_t depth, uint64_t ld, uint32_t box_rows,
                   CUtensorMap* out) {
  return hx_tensor_map("hx_gemm_tc", base, rows, depth, ld, box_rows, BK, true, out);
}

template <int BN, int EPI, bool IN_BLOCKS = false>
int launch(const CUtensorMap& map_w, const CUtensorMap& map_x, const GemmArgs& args, dim3 grid,
           cudaStream_t stream) {
  using Config = TileConfig<BN, EPI == EPI_SWIGLU>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(gemm_tc_kernel<BN, EPI, IN_BLOCKS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             Config::kSmemBytes) != cudaSuccess) {
      hx_set_error("hx_gemm_tc: cannot reserve %d bytes of shared memory", Config::kSmemBytes);
      cudaGetLastError();
      return HX_ERR_LAUNCH;
    }
    configured = true;
  }
  if (args.cluster > 1) {
    cudaLaunchConfig_t config = {};
    config.gridDim = grid;
    config.blockDim = THREADS;
    config.dynamicSmemBytes = Config::kSmemBytes;
    config.stream = stream;
    cudaLaunchAttribute attributes[2];
    attributes[0].id = cudaLaunchAttributeClusterDimension;
    attributes[0].val.clusterDim.x = attributes[0].val.clusterDim.y = 1;
    attributes[0].val.clusterDim.z = args.cluster;
    attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attributes;
    config.numAttrs = hx_pdl_enabled() ? 2 : 1;
    cudaLaunchKernelEx(&config, gemm_tc_kernel<BN, EPI, IN_BLOCKS>, map_w, map_x, args);
    return HX_OK;
  }
  hx_launch(gemm_tc_kernel<BN, EPI, IN_BLOCKS>, grid, THREADS, Config::kSmemBytes, stream, map_w, map_x, args);
  return HX_OK;
}

template <int BN>
int launch_epilogue(int epilogue, const CUtensorMap& map_w, const CUtensorMap& map_x,
                    const GemmArgs& args, dim3 grid, cudaStream_t stream) {
  switch (epilogue) {
    case EPI_STORE_BF16: return launch<BN, EPI_STORE_BF16>(map_w, map_x, args, grid, stream);
    case EPI_STORE_F32: return launch<BN, EPI_STORE_F32>(map_w, map_x, args, grid, stream);
    case EPI_ADD_F32: return launch<BN, EPI_ADD_F32>(map_w, map_x, args, grid, stream);
    case EPI_SWIGLU: return launch<BN, EPI_SWIGLU>(map_w, map_x, args, grid, stream);
    default:
      hx_set_error("hx_gemm_tc: unknown epilogue %d", epilogue);
      return HX_ERR_ARGUMENT;
  }
}

// How `workers` (CTAs, or pairs of them) go through the tiles of a product: the time in k-blocks of
// a worker, and for the add epilogue how the last, partly filled round is shared out (see unit_at).
//
// Sharing a round out pays where little of it is there.  A piece costs its run of k-blocks and an
// epilogue of atomic adds, 128 KB of them, which measured about as much as 8 k-blocks of products
// alone and 15 more when all SMs add at the same time; so many workers share the tiles that the
// sum of both is least.  With 2,048 tokens by [4,096 x 4,096] (108 tiles left for 148 SMs) sharing
// out gains nothing, with 512 tokens (64 tiles, less than half the grid) it takes 20 % off.
// 1,900 tokens by [5,120 x 13,824] leave 4 of 300 tiles: 261 us as a whole round, 195 shared out
// among 80 CTAs.
//
// Otherwise (pairs only, `most_pieces` > 1) the tiles of a last round may be cut into pieces of
// columns: half a tile takes 0.55 of a tile's time, a quarter 0.35 (its tokens are loaded as for a
// whole one).  256 tokens by [22,016 x 4,096], 86 tiles on 74 pairs: 63.6 -> 47.9 us; 2,048 by
// [12,288 x 4,096], 384: 142 -> 132 us in place.
// `ordered`: every sum has one writer, so nothing is shared out.
double plan_rounds(long long units, int workers, int k_blocks, bool add, bool ordered, int most_pieces,
                   int& whole_rounds, int& tail_workers, int& pieces) {
  const int rest = static_cast<int>(units % workers);
  const long long rounds = units / workers;
  whole_rounds = -1;
  tail_workers = 0;
  pieces = 1;
  if (!add && rest > 0) {
    while (2 * pieces <= most_pieces && 2 * pieces * rest <= workers) pieces *= 2;
    if (pieces > 1) {
      whole_rounds = static_cast<int>(rounds);
      return k_blocks * (static_cast<double>(rounds) + (pieces == 2 ? 0.55 : 0.35));
    }
  }
  if (add && !ordered && HX_GEMM_STREAM_K && rest > 0 && rest * 2 <= workers) {
    const double blocks = static_cast<double>(rest) * k_blocks;
    int share = static_cast<int>(sqrt(blocks * workers / 15.0));
    share = share < rest ? rest : share > workers ? workers : share;
    const double tail = blocks / share + 8.0 + 15.0 * share / workers;
    if (k_blocks - tail >= 12.0) {
      whole_rounds = static_cast<int>(rounds);
      tail_workers = share;
      return static_cast<double>(rounds) * k_blocks + tail;
    }
  }
  return static_cast<double>(rounds + (rest > 0 ? 1 : 0)) * k_blocks;
}

template <typename Kernel>
bool reserve_shared(Kernel kernel, int bytes) {
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess)
    return true;
  hx_set_error("hx_gemm_tc: cannot reserve %d bytes of shared memory", bytes);
  cudaGetLastError();
  return false;
}

// What the tensor map of the weights is made from; tiled ones (k_tiles > 0) are rows of 64 elements,
// tile behind tile.
struct WeightBoxes {
  const void* base;
  uint64_t rows, depth, ld;
};
WeightBoxes weight_boxes(const void* w, int weight_rows, int depth, int ldw, int k_tiles) {
  if (k_tiles > 0)
    return {w, static_cast<uint64_t>((weight_rows + BM - 1) / BM) * k_tiles * BM, BK, BK};
  return {w, static_cast<uint64_t>(weight_rows), static_cast<uint64_t>(depth), static_cast<uint64_t>(ldw)};
}

constexpr int MOST_PIECES = 4;      // of a tile of the last round

template <int EPI>
int launch_persistent(const CUtensorMap& map_w, const CUtensorMap& map_x, PersistentArgs args,
                      const WeightBoxes& boxes, cudaStream_t stream, bool ordered = false) {
  static bool configured = false;
  const int sms = hx_device_sm_count();
  if (sms <= 0) return HX_ERR_LAUNCH;
  if (!configured) {
    if (!reserve_shared(gemm_tc_persistent_kernel<EPI>, PersistentConfig::kSmemBytes) ||
        !reserve_shared(gemm_tc_pair_kernel<EPI>, PairConfig::kSmemBytes))
      return HX_ERR_LAUNCH;
    configured = true;
  }
  constexpr int kFeatures = EPI == EPI_SWIGLU ? BM : 2 * BM;
  args.head_tiles = (args.features + kFeatures - 1) / kFeatures;
  const int feature_tiles = args.heads * args.head_tiles;
  args.token_tiles = (args.tokens + BM - 1) / BM;
  const long long tiles = static_cast<long long>(args.token_tiles) * feature_tiles;
  HX_REQUIRE(tiles < (1ll << 30), "hx_gemm_tc: too many tiles");
  args.units = static_cast<int>(tiles);
  int whole_rounds = -1, tail = 0, pieces = 1;
  const double alone = plan_rounds(tiles, sms, args.k_blocks, EPI == EPI_ADD_F32, ordered, 1,
                                   args.whole_rounds, args.tail_ctas, pieces);
  // Pairs, unless their tiles of 256 tokens make the rounds longer by more than the twentieth that a
  // round is shorter at least (1,900 tokens by [27,648 x 5,120]: 12 rounds against 11, 380 against 375
  // us); short sums that are all pieces have nothing to win (129 tokens by [4,096 x 4,096]: 18.8
  // against 17.0 us).
  const int pair_tiles = (args.tokens + 2 * BM - 1) / (2 * BM), pairs = sms / 2;
  const long long pair_units = static_cast<long long>(pair_tiles) * feature_tiles;
  if (args.heads == 1 && args.tile_group == nullptr && args.tokens > BM && pairs > 0) {
    const double paired = plan_rounds(pair_units, pairs, args.k_blocks, EPI == EPI_ADD_F32, ordered,
                                      MOST_PIECES, whole_rounds, tail, pieces);
    const double penalty = EPI == EPI_ADD_F32 && whole_rounds == 0 && args.k_blocks < 96 ? 4.0 : 0.0;
    if (0.95 * paired + penalty <= alone) {
      args.token_tiles = pair_tiles;
      args.units = static_cast<int>(pair_units);
      args.whole_rounds = whole_rounds;
      args.tail_ctas = tail;
      args.tail_pieces = pieces;
      CUtensorMap map_piece = map_w;
      if (pieces > 1) {
        const int rc = get_tensor_map(boxes.base, boxes.rows, boxes.depth, boxes.ld, BM / pieces, &map_piece);
        if (rc != HX_OK) return rc;
      }
      const long long work = pieces > 1 && whole_rounds == 0 ? pair_units * pieces
                             : whole_rounds == 0             ? tail
                                                             : pair_units;
      hx_launch(gemm_tc_pair_kernel<EPI>, 2 * static_cast<int>(work < pairs ? work : pairs), THREADS,
                PairConfig::kSmemBytes, stream, map_w, map_piece, map_x, args);
      return HX_OK;
    }
  }
  const int ctas = args.whole_rounds == 0 ? args.tail_ctas : args.units < sms ? args.units : sms;
  hx_launch(gemm_tc_persistent_kernel<EPI>, ctas, THREADS, PersistentConfig::kSmemBytes, stream, map_w,
            map_x, args);
  return HX_OK;
}

int launch_persistent_epilogue(int epilogue, const CUtensorMap& map_w, const CUtensorMap& map_x,
                               const PersistentArgs& args, const WeightBoxes& boxes,
                               cudaStream_t stream, bool ordered = false) {
  switch (epilogue) {
    case EPI_STORE_BF16: return launch_persistent<EPI_STORE_BF16>(map_w, map_x, args, boxes, stream);
    case EPI_STORE_F32: return launch_persistent<EPI_STORE_F32>(map_w, map_x, args, boxes, stream);
    case EPI_ADD_F32: return launch_persistent<EPI_ADD_F32>(map_w, map_x, args, boxes, stream, ordered);
    case EPI_SWIGLU: return launch_persistent<EPI_SWIGLU>(map_w, map_x, args, boxes, stream);
    case EPI_ROPE_APPEND: return launch_persistent<EPI_ROPE_APPEND>(map_w, map_x, args, boxes, stream);
    default:
      hx_set_error("hx_gemm_tc: unknown epilogue %d", epilogue);
      return HX_ERR_ARGUMENT;
  }
}

}  // namespace

// Token tile the kernel would use for this many tokens (for tests and the bench's records).
HX_API int hx_gemm_tc_token_tile(int tokens) {
  if (tokens <= 16) return 16;
  if (tokens <= 32) return 32;
  if (tokens <= 64) return 64;
  if (tokens <= 128) return 128;
  return 256;
}

// 1 when the tensor-core kernel takes this shape; 0 when the caller must use hx_gemm_simt.
HX_API int hx_gemm_tc_supports(int tokens, int features, int depth, int ldx, int ldw) {
  return tokens > 0 && features > 0 && depth > 0 && depth % 8 == 0 && ldx % 8 == 0 &&
         ldw % 8 == 0;
}

// x: [tokens, depth] bf16 (row stride ldx), w: [weight_rows, depth] bf16 (row stride ldw).
// epilogue 0/1/2: `features` = weight_rows outputs per token.  epilogue 3 (SwiGLU; 5: the same
// with gelu_tanh in place of silu): w is the
// fused [gate; up] matrix, `features` = intermediate size, gate rows [0, features), up rows
// [up_row_offset, up_row_offset + features).  k_splits > 1 only with epilogue 2.
// weight_tiles != 0: w holds the matrix as [ceil(weight_rows / 128)][ceil(depth / 64)] tiles of
// [128][64] elements, zero padded (ldw is ignored; up_row_offset is then a multiple of 128).
// x_capacity_rows: rows of the buffer behind x (the tensor map is made for the buffer, so it
// can be reused for every batch size).
static int gemm_tc(const void* x, int ldx, int x_capacity_rows, const void* w, int ldw,
                   int weight_rows, void* out, int ldo, int tokens, int features, int depth,
                   int epilogue, int activation, float gate_limit, const float* gate_bias,
                   const float* up_bias, int up_row_offset, int k_splits, int weight_tiles,
                   int* status, cudaStream_t stream, float softcap = 0.0f, bool ordered = false) {
  if (weight_tiles) ldw = 8;      // not a stride of anything here
  HX_REQUIRE(softcap >= 0.0f && (softcap == 0.0f || epilogue == EPI_STORE_F32),
             "hx_gemm_tc: a softcap belongs to a float32 store");
  HX_REQUIRE(!weight_tiles || epilogue != EPI_SWIGLU || up_row_offset % BM == 0,
             "hx_gemm_tc: with tiled weights the up rows must start on a multiple of %d", BM);
  HX_REQUIRE(hx_gemm_tc_supports(tokens, features, depth, ldx, ldw),
             "hx_gemm_tc: shape tokens=%d features=%d depth=%d ldx=%d ldw=%d is not supported "
             "(depth and strides must be multiples of 8)", tokens, features, depth, ldx, ldw);
  HX_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0,
             "hx_gemm_tc: operands must be 16-byte aligned");
  HX_REQUIRE(x_capacity_rows >= tokens, "hx_gemm_tc: buffer rows %d < tokens %d", x_capacity_rows,
             tokens);
  HX_REQUIRE(status != nullptr, "hx_gemm_tc: status word missing");
  HX_REQUIRE(epilogue >= EPI_STORE_BF16 && epilogue <= EPI_SWIGLU,
             "hx_gemm_tc: unknown epilogue %d", epilogue);
  HX_REQUIRE(k_splits >= 1 && (k_splits == 1 || epilogue == EPI_ADD_F32),
             "hx_gemm_tc: split-K needs the add epilogue");
  HX_REQUIRE(epilogue != EPI_SWIGLU || up_row_offset + features <= weight_rows,
             "hx_gemm_tc: up rows exceed the weight matrix");
  HX_REQUIRE(epilogue == EPI_SWIGLU || features <= weight_rows,
             "hx_gemm_tc: features exceed the weight matrix");
  HX_REQUIRE(ldo >= features, "hx_gemm_tc: output stride too small");

  int bn = hx_gemm_tc_token_tile(tokens);
  // prompt portions: the persistent kernel, whose tiles have 128 tokens on the M side.  A sum
  // into a float32 output over at most 128 tokens is a weight stream even when it is not cut
  // along the reduction (the fused gate/up matrix has tiles enough as it is) and stays with
  // the streaming kernel: 128 weight rows per CTA, two CTAs an SM (measured: steps of 65 to
  // 128 tokens take 6 to 8 % less time than with that one product on the persistent kernel).
  const int total_k_blocks = (depth + BK - 1) / BK;
  // Products that are stored, deep and of few tiles: as many CTAs a tile, each with a run of k-blocks of its own, as
  // fill a wave of two CTAs an SM to four fifths (see gather_parts).  A cluster costs about 4 us of its own, so it
  // needs a depth of 2,048 and four runs (two of 32 blocks for 97 tiles: 17 us without, 18 with).  More than 128
  // tokens have the persistent kernels, 0.17 us a block of 64 against 0.25, and the epilogues of several tiles of 128
  // tokens: from a depth of 3,072 on, and four runs up to 6,144 (us, without / four runs / eight: 300 tokens by [16 x
  // 2,048] 9.0 / 9.9 / 10.9, x 3,072 11.8 / 11.2 / 11.4, x 5,120 17.4 / 13.7 / 12.9; 1,500 by [16 x 3,072] 11.6 / 11.4 / 15.0, x 4,096
  // 14.5 / 12.9 / 15.8; 700 by [256 x 4,096] 15.3 / 13.0 / 15.8; eight runs, 1,500 by [16 x 6,144] 19.8 / 17.0).
  const bool stores = epilogue == EPI_STORE_BF16 || epilogue == EPI_STORE_F32;
  int cluster = 1;
  if (stores && !ordered && total_k_blocks >= (tokens <= 128 ? 32 : 48)) {
    const long long tiles = static_cast<long long>((tokens + 127) / 128) * ((features + BM - 1) / BM);
    const long long fit = static_cast<long long>(0.8 * 2 * hx_device_sm_count()) / tiles;
    if (fit >= 4 && (tokens <= 128 || tiles <= 16)) {
      cluster = fit < 8 ? static_cast<int>(fit) : 8;
      if (tokens > 128 && total_k_blocks < 96) cluster = 4;
      const int per = (total_k_blocks + cluster - 1) / cluster;
      cluster = (total_k_blocks + per - 1) / per;      // none without a block
      if (bn > 128) bn = 128;
    }
  }
  const bool persistent =
      cluster <= 1 && bn >= 128 && k_splits == 1 && !(epilogue == EPI_ADD_F32 && tokens <= 128);
  if (cluster > 1) k_splits = cluster;
  CUtensorMap map_w, map_x;
  const int k_tiles = weight_tiles ? total_k_blocks : 0;
  const WeightBoxes boxes = weight_boxes(w, weight_rows, depth, ldw, k_tiles);
  int rc = get_tensor_map(boxes.base, boxes.rows, boxes.depth, boxes.ld, BM, &map_w);
  if (rc != HX_OK) return rc;
  rc = get_tensor_map(x, x_capacity_rows, depth, ldx, persistent ? BM : bn, &map_x);
  if (rc != HX_OK) return rc;

  if (persistent) {
    PersistentArgs args{out, ldo, tokens, features, depth, up_row_offset, k_tiles, 0, 0,
                        total_k_blocks, status, RopeArgs{}, -1, activation, nullptr, 0,
                        gate_limit, gate_bias, up_bias, softcap};
    rc = launch_persistent_epilogue(epilogue, map_w, map_x, args, boxes, stream, ordered);
    if (rc != HX_OK) return rc;
    HX_CHECK_LAUNCH("hx_gemm_tc");
    return HX_OK;
  }
  if (k_splits > total_k_blocks) k_splits = total_k_blocks;
  const int per_split = (total_k_blocks + k_splits - 1) / k_splits;
  k_splits = (total_k_blocks + per_split - 1) / per_split;
  GemmArgs args{out, ldo, tokens, features, depth, up_row_offset, per_split, k_tiles, status,
                activation, nullptr, 0, gate_limit, gate_bias, up_bias, softcap, cluster > 1 ? k_splits : 1};
  const dim3 grid((tokens + bn - 1) / bn, (features + BM - 1) / BM, k_splits);
  HX_REQUIRE(grid.y <= 65535, "hx_gemm_tc: too many features (%d)", features);

  switch (bn) {
    case 16: rc = launch_epilogue<16>(epilogue, map_w, map_x, args, grid, stream); break;
    case 32: rc = launch_epilogue<32>(epilogue, map_w, map_x, args, grid, stream); break;
    case 64: rc = launch_epilogue<64>(epilogue, map_w, map_x, args, grid, stream); break;
    case 128: rc = launch_epilogue<128>(epilogue, map_w, map_x, args, grid, stream); break;
    default: rc = launch_epilogue<256>(epilogue, map_w, map_x, args, grid, stream); break;
  }
  if (rc != HX_OK) return rc;
  HX_CHECK_LAUNCH("hx_gemm_tc");
  return HX_OK;
}

HX_API int hx_gemm_tc(const void* x, int ldx, int x_capacity_rows, const void* w, int ldw,
                      int weight_rows, void* out, int ldo, int tokens, int features, int depth,
                      int epilogue, int up_row_offset, int k_splits, int weight_tiles, int* status,
                      cudaStream_t stream) {
  // the gated epilogue by the gate's activation: 3 is silu(gate) * up, 5 gelu_tanh(gate) * up
  int activation = HX_GATE_SILU;
  if (epilogue == 5) {
    epilogue = EPI_SWIGLU;
    activation = HX_GATE_GELU_TANH;
  }
  return gemm_tc(x, ldx, x_capacity_rows, w, ldw, weight_rows, out, ldo, tokens, features, depth,
                 epilogue, activation, 0.0f, nullptr, nullptr, up_row_offset, k_splits,
                 weight_tiles, status, stream);
}

// The product added to a float32 output by one writer per sum, for any number of tokens: the same call
// gives the same bits.  (hx_gemm_tc shares a short last round of sums out by atomic adds: 512 tokens by
// [4,096 x 4,096] 35.9 us from a cold L2, 39.9 here, by [4,096 x 11,008] 56.4 and 72.7.)
HX_API int hx_gemm_tc_ordered(const void* x, int ldx, int x_capacity_rows, const void* w, int ldw,
                              int weight_rows, float* out, int ldo, int tokens, int features,
                              int depth, int weight_tiles, int* status, cudaStream_t stream) {
  return gemm_tc(x, ldx, x_capacity_rows, w, ldw, weight_rows, out, ldo, tokens, features, depth,
                 EPI_ADD_F32, HX_GATE_SILU, 0.0f, nullptr, nullptr, 0, 1, weight_tiles, status, stream,
                 0.0f, true);
}

// The stored product as one chain over the depth, never by clusters: a token's sums do not depend on how many
// others the call has.  (As hx_gemm_tc does it where few tiles have a deep reduction: 64 tokens by [1,280 x 4,096]
// 9.9 us, 16.3 here.)
HX_API int hx_gemm_tc_stored_ordered(const void* x, int ldx, int x_capacity_rows, const void* w, int ldw,
                                     int weight_rows, void* out, int ldo, int tokens, int features,
                                     int depth, int epilogue, float softcap, int weight_tiles, int* status,
                                     cudaStream_t stream) {
  HX_REQUIRE(epilogue == EPI_STORE_BF16 || epilogue == EPI_STORE_F32,
             "hx_gemm_tc_stored_ordered: epilogue %d does not store", epilogue);
  return gemm_tc(x, ldx, x_capacity_rows, w, ldw, weight_rows, out, ldo, tokens, features, depth, epilogue,
                 HX_GATE_SILU, 0.0f, nullptr, nullptr, 0, 1, weight_tiles, status, stream, softcap, true);
}

// The product with a float32 store whose sums run into a level: out = cap * tanh(x w^T / cap).
HX_API int hx_gemm_tc_softcapped(const void* x, int ldx, int x_capacity_rows, const void* w,
                                 int ldw, int weight_rows, float* out, int ldo, int tokens,
                                 int features, int depth, float softcap, int weight_tiles,
                                 int* status, cudaStream_t stream) {
  return gemm_tc(x, ldx, x_capacity_rows, w, ldw, weight_rows, out, ldo, tokens, features, depth,
                 EPI_STORE_F32, HX_GATE_SILU, 0.0f, nullptr, nullptr, 0, 1, weight_tiles, status,
                 stream, softcap);
}

// The product with the gated epilogue for every HxGateActivation and with float32 biases on
// the gate and the up rows ([features] each, either may be null): out = f(gate + gate_bias,
// up + up_bias) in the compute type.
HX_API int hx_gemm_tc_gated(const void* x, int ldx, int x_capacity_rows, const void* w, int ldw,
                            int weight_rows, void* out, int ldo, int tokens, int features,
                            int depth, int activation, float gate_limit, const float* gate_bias,
                            const float* up_bias, int up_row_offset, int weight_tiles,
                            int* status, cudaStream_t stream) {
  HX_REQUIRE(activation >= HX_GATE_SILU && activation <= HX_GATE_CLAMPED_SIGMOID,
             "hx_gemm_tc_gated: unknown activation %d", activation);
  return gemm_tc(x, ldx, x_capacity_rows, w, ldw, weight_rows, out, ldo, tokens, features, depth,
                 EPI_SWIGLU, activation, gate_limit, gate_bias, up_bias, up_row_offset, 1,
                 weight_tiles, status, stream);
}

// The grouped product: rows of x come in tiles of `token_tile` (16, 32, 64, 128 or 256), and
// tile t multiplies with group tile_group[t] of w, which holds `groups` matrices of
// `group_rows` rows one below the other (row-major, row stride ldw); a negative entry skips the
// tile.  tile_group (device memory, ceil(tokens / token_tile) entries) may be written by the
// kernel before this one on the stream.  `tokens` is the host's bound on the rows in use; rows
// of tiles that are only partly in use are computed and stored like the others.  Epilogues 0,
// 1 and 3 (5); `features` and `up_row_offset` count inside a group.
static int gemm_tc_grouped(const void* x, int ldx, int x_capacity_rows, const void* w, int ldw,
                           int group_rows, int groups, void* out, int ldo, int tokens,
                           int features, int depth, int epilogue, int activation,
                           float gate_limit, int up_row_offset, int token_tile,
                           const int* tile_group, int* status, cudaStream_t stream) {
  HX_REQUIRE(groups > 0 && group_rows > 0 && tile_group != nullptr,
             "hx_gemm_tc_grouped: bad groups");
  HX_REQUIRE(static_cast<long long>(groups) * group_rows < (1ll << 31),
             "hx_gemm_tc_grouped: too many weight rows");
  HX_REQUIRE(hx_gemm_tc_supports(tokens, features, depth, ldx, ldw),
             "hx_gemm_tc_grouped: shape tokens=%d features=%d depth=%d ldx=%d ldw=%d is not "
             "supported (depth and strides must be multiples of 8)", tokens, features, depth, ldx,
             ldw);
  HX_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0,
             "hx_gemm_tc_grouped: operands must be 16-byte aligned");
  HX_REQUIRE(x_capacity_rows >= tokens, "hx_gemm_tc_grouped: buffer rows %d < tokens %d",
             x_capacity_rows, tokens);
  HX_REQUIRE(status != nullptr, "hx_gemm_tc_grouped: status word missing");
  HX_REQUIRE(epilogue == EPI_STORE_BF16 || epilogue == EPI_STORE_F32 || epilogue == EPI_SWIGLU,
             "hx_gemm_tc_grouped: epilogue %d is not one of store and gated", epilogue);
  HX_REQUIRE(epilogue == EPI_SWIGLU ? up_row_offset + features <= group_rows
                                    : features <= group_rows,
             "hx_gemm_tc_grouped: features exceed a group's rows");
  HX_REQUIRE(ldo >= features, "hx_gemm_tc_grouped: output stride too small");
  HX_REQUIRE(token_tile == 16 || token_tile == 32 || token_tile == 64 || token_tile == 128 ||
                 token_tile == 256,
             "hx_gemm_tc_grouped: token tile %d", token_tile);
  CUtensorMap map_w, map_x;
  int rc = get_tensor_map(w, static_cast<uint64_t>(groups) * group_rows, depth, ldw, BM, &map_w);
  if (rc != HX_OK) return rc;
  rc = get_tensor_map(x, x_capacity_rows, depth, ldx, token_tile, &map_x);
  if (rc != HX_OK) return rc;
  const int total_k_blocks = (depth + BK - 1) / BK;
  if (token_tile == BM) {
    // tiles of 128 tokens: the persistent kernel, as for prompt portions of a plain product
    PersistentArgs persistent{out, ldo, tokens, features, depth, up_row_offset, 0, 0, 0,
                              total_k_blocks, status, RopeArgs{}, -1, activation, tile_group,
                              group_rows, gate_limit};
    rc = launch_persistent_epilogue(epilogue, map_w, map_x, persistent, WeightBoxes{}, stream);
    if (rc != HX_OK) return rc;
    HX_CHECK_LAUNCH("hx_gemm_tc_grouped");
    return HX_OK;
  }
  GemmArgs args{out, ldo, tokens, features, depth, up_row_offset, total_k_blocks, 0, status,
                activation, tile_group, group_rows, gate_limit};
  const dim3 grid((tokens + token_tile - 1) / token_tile, (features + BM - 1) / BM, 1);
  HX_REQUIRE(grid.y <= 65535, "hx_gemm_tc_grouped: too many features (%d)", features);
  switch (token_tile) {
    case 16:
      // fewer than 16 tiles: experts of one to three tokens, whose float32 sums are those of products a pair
      if (epilogue == EPI_STORE_F32 && tokens < 16 * 16)
        rc = launch<16, EPI_STORE_F32, true>(map_w, map_x, args, grid, stream);
      else
        rc = launch_epilogue<16>(epilogue, map_w, map_x, args, grid, stream);
      break;
    case 32: rc = launch_epilogue<32>(epilogue, map_w, map_x, args, grid, stream); break;
    case 64: rc = launch_epilogue<64>(epilogue, map_w, map_x, args, grid, stream); break;
    default: rc = launch_epilogue<256>(epilogue, map_w, map_x, args, grid, stream); break;
  }
  if (rc != HX_OK) return rc;
  HX_CHECK_LAUNCH("hx_gemm_tc_grouped");
  return HX_OK;
}

HX_API int hx_gemm_tc_grouped(const void* x, int ldx, int x_capacity_rows, const void* w, int ldw,
                              int group_rows, int groups, void* out, int ldo, int tokens,
                              int features, int depth, int epilogue, int up_row_offset,
                              int token_tile, const int* tile_group, int* status,
                              cudaStream_t stream) {
  int activation = HX_GATE_SILU;
  if (epilogue == 5) {
    epilogue = EPI_SWIGLU;
    activation = HX_GATE_GELU_TANH;
  }
  return gemm_tc_grouped(x, ldx, x_capacity_rows, w, ldw, group_rows, groups, out, ldo, tokens,
                         features, depth, epilogue, activation, 0.0f, up_row_offset, token_tile,
                         tile_group, status, stream);
}

// The grouped product with the gated epilogue for any HxGateActivation: out = f(gate, up) with
// the gate rows at 0 and the up rows at up_row_offset inside a group; gate_limit is the limit of
// HX_GATE_CLAMPED_SIGMOID.
HX_API int hx_gemm_tc_grouped_gated(const void* x, int ldx, int x_capacity_rows, const void* w,
                                    int ldw, int group_rows, int groups, void* out, int ldo,
                                    int tokens, int features, int depth, int activation,
                                    float gate_limit, int up_row_offset, int token_tile,
                                    const int* tile_group, int* status, cudaStream_t stream) {
  HX_REQUIRE(activation >= HX_GATE_SILU && activation <= HX_GATE_CLAMPED_SIGMOID,
             "hx_gemm_tc_grouped_gated: unknown activation %d", activation);
  return gemm_tc_grouped(x, ldx, x_capacity_rows, w, ldw, group_rows, groups, out, ldo, tokens,
                         features, depth, EPI_SWIGLU, activation, gate_limit, up_row_offset,
                         token_tile, tile_group, status, stream);
}

// One product per head on the persistent kernel: out[t, h * out_stride + o] = sum_i w[h][o][i] *
// x[t, h * x_stride + i], x [tokens, ldx], w [heads][out_dim][in_dim], out [tokens, ldo], all bf16.
// Whole k-blocks only (in_dim a multiple of 64): a box must not reach into the next head's columns.
HX_API int hx_gemm_tc_heads_supports(int in_dim, int x_stride, int ldx) {
  return in_dim > 0 && in_dim % BK == 0 && x_stride % 8 == 0 && ldx % 8 == 0;
}

HX_API int hx_gemm_tc_heads(const void* x, int ldx, int x_capacity_rows, int x_stride, const void* w,
                            void* out, int ldo, int out_stride, int tokens, int heads, int out_dim,
                            int in_dim, int* status, cudaStream_t stream) {
  HX_REQUIRE(tokens >= 0 && heads > 0 && out_dim > 0 && hx_gemm_tc_heads_supports(in_dim, x_stride, ldx),
             "hx_gemm_tc_heads: heads of %d by %d, %d apart in rows of %d, are not supported", out_dim,
             in_dim, x_stride, ldx);
  HX_REQUIRE(static_cast<long long>(heads) * out_dim < (1ll << 31) && x_stride >= 0 &&
                 ldx >= (heads - 1) * x_stride + in_dim && ldo >= (heads - 1) * out_stride + out_dim,
             "hx_gemm_tc_heads: bad strides");
  HX_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0,
             "hx_gemm_tc_heads: operands must be 16-byte aligned");
  HX_REQUIRE(x_capacity_rows >= tokens, "hx_gemm_tc_heads: buffer rows %d < tokens %d", x_capacity_rows,
             tokens);
  HX_REQUIRE(status != nullptr, "hx_gemm_tc_heads: status word missing");
  if (tokens == 0) return HX_OK;
  CUtensorMap map_w, map_x;
  int rc = get_tensor_map(w, static_cast<uint64_t>(heads) * out_dim, in_dim, in_dim, BM, &map_w);
  if (rc != HX_OK) return rc;
  rc = get_tensor_map(x, x_capacity_rows, (heads - 1) * x_stride + in_dim, ldx, BM, &map_x);
  if (rc != HX_OK) return rc;
  PersistentArgs args{out, ldo, tokens, out_dim, in_dim, 0, 0, 0, 0, in_dim / BK, status, RopeArgs{}, -1,
                      HX_GATE_SILU, nullptr, 0};
  args.heads = heads;
  args.head_x = x_stride;
  args.head_out = out_stride;
  rc = launch_persistent<EPI_STORE_BF16>(
      map_w, map_x, args, weight_boxes(w, heads * out_dim, in_dim, in_dim, 0), stream);
  if (rc != HX_OK) return rc;
  HX_CHECK_LAUNCH("hx_gemm_tc_heads");
  return HX_OK;
}

// Fewest tokens hx_gemm_tc_rope_append takes: it exists for the persistent kernel only.
HX_API int hx_gemm_tc_rope_append_min_tokens() { return 65; }

// The fused QKV product of a prompt portion with the rotary encoding and the cache append as
// its epilogue: qkv[t] = x[t] @ w.T with w = [q heads | k heads | v heads] x head_dim rows;
// the queries are rotated and stored to `out` (row stride ldo; the key and value parts of an
// out row are NOT written), the keys are rotated and, like the values, written to the
// token's slot of its page in k_cache / v_cache (both nullptr: dropped).  The arguments from
// `positions` on mean what they mean to hx_rope_append, with adjacent pairs; x, w, ldx, ldw,
// x_capacity_rows, weight_rows and weight_tiles what they mean to hx_gemm_tc.  Needs more
// than 64 tokens, bfloat16, head_dim a multiple of 16 and 16-byte aligned out and caches.
// shared_values != 0: w = [q heads | k heads], and the keys before the rotation are the values.
HX_API int hx_gemm_tc_rope_append_shared(const void* x, int ldx, int x_capacity_rows, const void* w,
                                  int ldw, int weight_rows, void* out, int ldo, int tokens,
                                  int depth, int weight_tiles, const int* positions,
                                  const int* token_request, const int* request_table_row,
                                  const int* block_tables, int table_stride, void* k_cache,
                                  void* v_cache, const float* cos_table, const float* sin_table,
                                  int table_positions, int heads, int kv_heads, int head_dim,
                                  int rotary_dim, int page_size, int num_pages, int shared_values,
                                  int* status, cudaStream_t stream) {
  const int row_heads = heads + (shared_values ? 1 : 2) * kv_heads;
  if (weight_tiles) ldw = 8;      // not a stride of anything here
  HX_REQUIRE(heads > 0 && kv_heads > 0 && head_dim > 0 && head_dim % 16 == 0,
             "hx_gemm_tc_rope_append: head_dim %d must be a multiple of 16", head_dim);
  HX_REQUIRE(static_cast<long long>(row_heads) * head_dim <= weight_rows,
             "hx_gemm_tc_rope_append: %d heads of %d exceed the %d weight rows", row_heads, head_dim,
             weight_rows);
  const int features = row_heads * head_dim;
  HX_REQUIRE(tokens >= hx_gemm_tc_rope_append_min_tokens(),
             "hx_gemm_tc_rope_append: %d tokens; it takes prompt portions of at least %d", tokens,
             hx_gemm_tc_rope_append_min_tokens());
  HX_REQUIRE(hx_gemm_tc_supports(tokens, features, depth, ldx, ldw),
             "hx_gemm_tc_rope_append: shape tokens=%d features=%d depth=%d ldx=%d ldw=%d is not "
             "supported (depth and strides must be multiples of 8)", tokens, features, depth, ldx,
             ldw);
  HX_REQUIRE(rotary_dim >= 0 && rotary_dim <= head_dim && rotary_dim % 2 == 0,
             "hx_gemm_tc_rope_append: rotary_dim %d must be even and at most head_dim %d",
             rotary_dim, head_dim);
  HX_REQUIRE(rotary_dim == 0 || (table_positions > 0 && cos_table && sin_table),
             "hx_gemm_tc_rope_append: rotary table missing");
  HX_REQUIRE((k_cache == nullptr) == (v_cache == nullptr),
             "hx_gemm_tc_rope_append: key and value cache come together");
  HX_REQUIRE(k_cache == nullptr || (page_size > 0 && num_pages > 0 && table_stride > 0 &&
                                    token_request && request_table_row && block_tables),
             "hx_gemm_tc_rope_append: cache arguments missing");
  HX_REQUIRE(positions != nullptr && status != nullptr,
             "hx_gemm_tc_rope_append: positions or status word missing");
  HX_REQUIRE(ldo >= heads * head_dim && ldo % 8 == 0,
             "hx_gemm_tc_rope_append: output stride %d must hold the queries and be a multiple "
             "of 8", ldo);
  HX_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(out) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(k_cache) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(v_cache) & 15) == 0,
             "hx_gemm_tc_rope_append: operands must be 16-byte aligned");
  HX_REQUIRE(x_capacity_rows >= tokens, "hx_gemm_tc_rope_append: buffer rows %d < tokens %d",
             x_capacity_rows, tokens);

  CUtensorMap map_w, map_x;
  const int total_k_blocks = (depth + BK - 1) / BK;
  const int k_tiles = weight_tiles ? total_k_blocks : 0;
  const WeightBoxes boxes = weight_boxes(w, weight_rows, depth, ldw, k_tiles);
  int rc = get_tensor_map(boxes.base, boxes.rows, boxes.depth, boxes.ld, BM, &map_w);
  if (rc != HX_OK) return rc;
  rc = get_tensor_map(x, x_capacity_rows, depth, ldx, BM, &map_x);
  if (rc != HX_OK) return rc;
  PersistentArgs args{out, ldo, tokens, features, depth, 0, k_tiles, 0, 0, total_k_blocks, status,
                      RopeArgs{positions, token_request, request_table_row, block_tables,
                               table_stride, static_cast<__nv_bfloat16*>(k_cache),
                               static_cast<__nv_bfloat16*>(v_cache), cos_table, sin_table,
                               table_positions, heads, kv_heads, head_dim, rotary_dim, page_size,
                               num_pages, shared_values}};
  rc = launch_persistent_epilogue(EPI_ROPE_APPEND, map_w, map_x, args, boxes, stream);
  if (rc != HX_OK) return rc;
  HX_CHECK_LAUNCH("hx_gemm_tc_rope_append");
  return HX_OK;
}

HX_API int hx_gemm_tc_rope_append(const void* x, int ldx, int x_capacity_rows, const void* w,
                                  int ldw, int weight_rows, void* out, int ldo, int tokens,
                                  int depth, int weight_tiles, const int* positions,
                                  const int* token_request, const int* request_table_row,
                                  const int* block_tables, int table_stride, void* k_cache,
                                  void* v_cache, const float* cos_table, const float* sin_table,
                                  int table_positions, int heads, int kv_heads, int head_dim,
                                  int rotary_dim, int page_size, int num_pages, int* status,
                                  cudaStream_t stream) {
  return hx_gemm_tc_rope_append_shared(x, ldx, x_capacity_rows, w, ldw, weight_rows, out, ldo,
                                       tokens, depth, weight_tiles, positions, token_request,
                                       request_table_row, block_tables, table_stride, k_cache,
                                       v_cache, cos_table, sin_table, table_positions, heads,
                                       kv_heads, head_dim, rotary_dim, page_size, num_pages, 0,
                                       status, stream);
}

// ------------------------------------------------------------ the bounded wait, by itself
//
// What a kernel of this library does when an mbarrier it waits for never completes: the wait
// gives up after its limit, the thread sets HX_FLAG_WAIT_TIMEOUT in the status word and the
// kernel returns; the host then fails the step.  This entry point runs exactly that path on a
// barrier of its own, with a limit of `polls` polls instead of the kernels' forty million, so
// that the path can be exercised in a fraction of a millisecond: with `arrive` = 0 nobody
// ever arrives at the barrier and the wait must run out; with `arrive` = 1 the waiting
// thread's own arrival completes the phase first and the wait must succeed.  `succeeded`
// (device, one int, may be null) receives 1 when the wait succeeded and 0 when it ran out.
namespace {

__global__ void bounded_wait_kernel(uint32_t polls, int arrive, int* status, int* succeeded) {
  __shared__ __align__(8) uint64_t barrier;
  hx_pdl_prologue();
  if (threadIdx.x == 0) {
    mbar_init(&barrier, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (arrive) mbar_arrive(&barrier);
    const bool ok = mbar_wait(&barrier, 0, polls);
    if (!ok && status != nullptr) atomicOr(status, HX_FLAG_WAIT_TIMEOUT);
    if (succeeded != nullptr) *succeeded = ok ? 1 : 0;
  }
}

}  // namespace

HX_API int hx_bounded_wait_check(int polls, int arrive, int* status, int* succeeded,
                                 cudaStream_t stream) {
  HX_REQUIRE(polls > 0 && polls <= 1000000, "hx_bounded_wait_check: 1 to 1,000,000 polls");
  HX_REQUIRE(status != nullptr, "hx_bounded_wait_check: status word missing");
  hx_launch(bounded_wait_kernel, 1, 32, 0, stream, static_cast<uint32_t>(polls), arrive, status,
            succeeded);
  HX_CHECK_LAUNCH("hx_bounded_wait_check");
  return HX_OK;
}
