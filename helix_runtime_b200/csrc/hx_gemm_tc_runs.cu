// Grouped products of many tokens (the experts of a prompt): the rows of the tokens lie group by
// group, every group's rows padded to a multiple of 32, and a group's rows are multiplied with that
// group's matrix.
//
// What bounds it: with more than some hundred tokens a group the tensor cores, as long as tiles are
// full and every SM has as many of them.  The groups' sizes are the router's choice and known on the
// device only.  With tiles of 256 tokens as the M side a group of 270 tokens pays two whole tiles, and
// a static share of a list whose end is empty leaves some CTAs a tile more than others.  So here
//
// * the WEIGHTS are the M side (256 rows over a pair of CTAs, tcgen05.mma.cta_group::2) and the tokens
//   the N side, in any multiple of 32 up to 256;
// * each group's run of rows is cut into as few tiles as hold it, all as large (up to 32 rows);
// * every CTA makes the list of tiles for itself from the groups' list, sorted by size, and the units
//   (a tile by 256 weight rows) are dealt round by round over the pairs, so that the last round is made
//   of the smallest ones.  A group's tiles stay neighbours: its weights come from DRAM once.
//
// For the gated epilogue the 128 weight rows of a CTA are 64 gate rows and the 64 up rows that belong
// to them in turns of 16 (one copy with a tensor map of four dimensions), so that a gate and its up
// value are 16 lanes apart in one warp and the two halves of the warp exchange half of their tokens.
//
// Measured (us, gate and up [16 x 5,632 x 4,096] + down [16 x 4,096 x 2,816], L2 flushed; tiles of 64 or 128
// tokens by one CTA before): 64 tokens a group on average 160 + 94 -> 150 + 87, 100: 190 + 112 -> 157 + 91,
// 256: 263 + 153 -> 185 + 104 (tiles of 256 tokens by pairs: 258 + 120), 1,000: 738 + 417 -> 646 + 323; up to
// about 200 tokens the stream of the weights (738 + 369 MB) is the bound, from there the products.
//
// Every wait on an mbarrier is bounded; a wait that runs out sets a status bit, the CTAs skip their
// remaining work, free their tensor memory and return.
#include "hx_tcgen05.cuh"
#include "hx_tensor_map.cuh"

namespace {

constexpr int ROWS = 128;           // weight rows a CTA
constexpr int BK = 64;              // k elements per stage: 128 bytes, one swizzle span
constexpr int UMMA_K = 16;
constexpr int THREADS = 192;
constexpr int STEP = 32;            // rows of the tokens: what a group's rows are padded to
constexpr int TILE_STEPS = 8;       // steps of the largest tile
constexpr int MAX_STEPS = 4096;     // of the whole list
constexpr int STAGES = 6;
constexpr int WEIGHT_BYTES = ROWS * BK * 2;
constexpr int STAGE_BYTES = 2 * WEIGHT_BYTES;      // a CTA brings at most 128 of the tokens
constexpr int BUFFER_COLUMNS = STEP * TILE_STEPS;
constexpr int TMEM_COLUMNS = 2 * BUFFER_COLUMNS;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*alignment*/ + 256 /*barriers*/ + 4 * MAX_STEPS;

struct RunsArgs {
  void* out;
  int ldo;
  int steps;               // entries of tile_group: a group each, or -1 (no rows)
  int features;
  int feature_tiles;
  int k_blocks;
  int group_rows;
  int activation;
  float gate_limit;
  const int* tile_group;
  int* status;
};

// Boxes of 16, 32, 64 and 128 rows of the tokens.
struct TokenMaps {
  CUtensorMap boxes[4];
};

// A tile in 32 bits: its first step, its steps, its group.
__device__ __forceinline__ uint32_t pack_tile(int first, int steps, int group) {
  return static_cast<uint32_t>(first) | static_cast<uint32_t>(steps - 1) << 12 |
         static_cast<uint32_t>(group) << 16;
}

// How many tiles of every size the list makes, and which come first: the largest.
struct TileList {
  int count[TILE_STEPS + 1];      // [size of a run's largest tile]
};

// The tiles of the runs of equal groups in tile_group, sorted by the size of their run's largest, into
// `tiles`.  All threads of the CTA; `scratch`: 7 bytes an entry and a few more.  The order depends on
// the list alone: every CTA finds the same.
__device__ __forceinline__ void make_tiles(const int* __restrict__ tile_group, int steps, uint8_t* scratch,
                                           uint32_t* tiles, TileList& list) {
  uint32_t* packed = reinterpret_cast<uint32_t*>(scratch);
  int16_t* groups = reinterpret_cast<int16_t*>(packed + MAX_STEPS);
  uint8_t* sizes = reinterpret_cast<uint8_t*>(groups + MAX_STEPS);
  uint32_t* starts = reinterpret_cast<uint32_t*>(sizes + MAX_STEPS);      // a bit for every run's first entry
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int t = threadIdx.x; t < steps; t += THREADS) groups[t] = static_cast<int16_t>(max(tile_group[t], -1));
  __syncthreads();
  for (int word = warp; word <= steps / 32; word += THREADS / 32) {
    const int t = 32 * word + lane;
    const uint32_t bits = __ballot_sync(0xffffffffu, t == 0 || t >= steps || groups[t] != groups[t - 1]);
    if (lane == 0) starts[word] = bits;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < steps; t += THREADS) {
    uint8_t size = 0;
    if (groups[t] >= 0) {
      int word = t >> 5;
      uint32_t bits = starts[word] & (0xffffffffu >> (31 - (t & 31)));
      while (bits == 0) bits = starts[--word];      // entry 0 starts a run
      const int first = 32 * word + 31 - __clz(bits);
      word = t >> 5;
      bits = starts[word] & ~(0xffffffffu >> (31 - (t & 31)));
      while (bits == 0) bits = starts[++word];      // entry `steps` does
      const int length = 32 * word + __ffs(bits) - 1 - first;
      const int count = (length + TILE_STEPS - 1) / TILE_STEPS;
      const int k = ((t - first) * count + length - 1) / length;      // the first tile not in front of t
      if (k * length / count == t - first) {
        size = static_cast<uint8_t>((length + count - 1) / count);
        packed[t] = pack_tile(t, (k + 1) * length / count - k * length / count, groups[t]);
      }
    }
    sizes[t] = size;
  }
  __syncthreads();
  // a warp counts a size
  for (int size = 1 + warp; size <= TILE_STEPS; size += THREADS / 32) {
    int count = 0;
    for (int base = 0; base < steps; base += 32)
      count += __popc(__ballot_sync(0xffffffffu, base + lane < steps && sizes[base + lane] == size));
    if (lane == 0) list.count[size] = count;
  }
  __syncthreads();
  for (int size = 1 + warp; size <= TILE_STEPS; size += THREADS / 32) {
    int at = 0;
    for (int larger = size + 1; larger <= TILE_STEPS; ++larger) at += list.count[larger];
    for (int base = 0; base < steps; base += 32) {
      const bool mine = base + lane < steps && sizes[base + lane] == size;
      const uint32_t bits = __ballot_sync(0xffffffffu, mine);
      if (mine) tiles[at + __popc(bits & ((1u << lane) - 1))] = packed[base + lane];
      at += __popc(bits);
    }
  }
  // the ring of operands takes the scratch's place: copies come after these accesses
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
}

struct RunUnit {
  int token0, steps, group, feature_tile;
};

// Unit `index`: the largest tiles by all weight rows first, the tile varying fastest.
__device__ __forceinline__ bool run_unit(const RunsArgs& a, const TileList& list, const uint32_t* tiles,
                                         int index, RunUnit& u) {
  int first = 0;
#pragma unroll 1
  for (int size = TILE_STEPS; size > 0; --size) {
    const int count = list.count[size];
    const int units = count * a.feature_tiles;
    if (index < units) {
      const uint32_t tile = tiles[first + index % count];
      u.token0 = static_cast<int>(tile & 0xfffu) * STEP;
      u.steps = static_cast<int>(tile >> 12 & 0xfu) + 1;
      u.group = static_cast<int>(tile >> 16);
      u.feature_tile = index / count;
      return true;
    }
    index -= units;
    first += count;
  }
  return false;
}

__device__ __forceinline__ void tma_load_4d_pair(void* dst, const CUtensorMap* map, uint32_t bar, int x, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(0), "r"(w)
      : "memory");
}

// grid: pairs of CTAs.  GATED: bfloat16 activations of gate and up rows; else float32 sums.
template <bool GATED>
__global__ __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS) void gemm_tc_runs_kernel(
    const __grid_constant__ CUtensorMap map_w, const __grid_constant__ TokenMaps map_x, const RunsArgs args) {
  constexpr int FEATURES = GATED ? ROWS : 2 * ROWS;      // of a unit

  hx_pdl_trigger();
  extern __shared__ uint8_t smem_raw[];
  __shared__ TileList list;
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);      // leader's count
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tmem_full_bar = empty_bar + STAGES;      // [2]
  uint64_t* tmem_empty_bar = tmem_full_bar + 2;      // [2]: leader's count, of both CTAs' epilogues
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(tmem_empty_bar + 2);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_holder + 1);
  uint32_t* tiles = reinterpret_cast<uint32_t*>(smem + STAGES * STAGE_BYTES + 256);

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
  if (warp == 1) tmem_alloc_pair(tmem_holder, TMEM_COLUMNS);
  hx_pdl_wait();
  make_tiles(args.tile_group, args.steps, smem, tiles, list);
  tc_fence_before();
  __syncthreads();
  cluster_sync();      // nothing arrives at the other CTA's barriers before they are there
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  if (warp == 0) {
    // -------------------------------------------------------------- TMA producer
    if (hx_elect_one()) {
      uint32_t fill = 0;      // stages filled so far, over all units
      RunUnit unit;
      for (int index = worker; run_unit(args, list, tiles, index, unit) && !*failed; index += workers) {
        const int my_tokens = unit.steps * (STEP / 2);
        const int token0 = unit.token0 + rank * my_tokens;
        const int weight_row = unit.group * args.group_rows + unit.feature_tile * FEATURES + rank * (FEATURES / 2);
        const uint32_t bytes = WEIGHT_BYTES + static_cast<uint32_t>(my_tokens) * BK * 2;
        for (int kb = 0; kb < args.k_blocks; ++kb, ++fill) {
          const int s = fill % STAGES;
          if (!mbar_wait(&empty_bar[s], ((fill / STAGES) & 1u) ^ 1u)) {
            atomicOr(args.status, HX_FLAG_WAIT_TIMEOUT);
            *failed = 1;
            break;
          }
          uint8_t* stage = smem + s * STAGE_BYTES;
          if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * bytes);
          const uint32_t bar = cluster_address(&full_bar[s], 0);
          if (GATED) tma_load_4d_pair(stage, &map_w, bar, kb * BK, weight_row / 16);
          else tma_load_2d_pair(stage, &map_w, bar, kb * BK, weight_row);
          int row = 0;
#pragma unroll
          for (int box = 3; box >= 0; --box) {
            if (unit.steps >> box & 1) {
              tma_load_2d_pair(stage + WEIGHT_BYTES + row * BK * 2, &map_x.boxes[box], bar, kb * BK, token0 + row);
              row += 16 << box;
            }
          }
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
      RunUnit unit;
      int iteration = 0;
      for (int index = worker; run_unit(args, list, tiles, index, unit) && !*failed; index += workers, ++iteration) {
        const int buffer = iteration & 1;
        if (!mbar_wait_cluster(&tmem_empty_bar[buffer], (static_cast<uint32_t>(iteration >> 1) & 1u) ^ 1u)) {
          atomicOr(args.status, HX_FLAG_WAIT_TIMEOUT);
          *failed = 1;
          break;
        }
        tc_fence_after();
        const uint32_t accumulator = tmem_base + buffer * BUFFER_COLUMNS;
        const uint32_t idesc = make_idesc(2 * ROWS, unit.steps * STEP);
        for (int kb = 0; kb < args.k_blocks; ++kb, ++drained) {
          const int s = drained % STAGES;
          if (!mbar_wait_cluster(&full_bar[s], (drained / STAGES) & 1u)) {
            atomicOr(args.status, HX_FLAG_WAIT_TIMEOUT);
            *failed = 1;
            break;
          }
          tc_fence_after();
          const uint32_t stage = smem_u32(smem + s * STAGE_BYTES);
          const uint64_t desc_w = make_smem_desc(stage);
          const uint64_t desc_x = make_smem_desc(stage + WEIGHT_BYTES);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t step = static_cast<uint64_t>(k * UMMA_K * 2 >> 4);
            umma_bf16_pair(accumulator, desc_w + step, desc_x + step, idesc, kb > 0 || k > 0 ? 1u : 0u);
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
    RunUnit unit;
    int iteration = 0;
    for (int index = worker; run_unit(args, list, tiles, index, unit) && !*failed; index += workers, ++iteration) {
      const int buffer = iteration & 1;
      bool ok = true;
      if (lane == 0) ok = mbar_wait_cluster(&tmem_full_bar[buffer], static_cast<uint32_t>(iteration >> 1) & 1u);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) {
        if (lane == 0) {
          atomicOr(args.status, HX_FLAG_WAIT_TIMEOUT);
          *failed = 1;
        }
        break;
      }
      tc_fence_after();
      const uint32_t accumulator = lane_base + buffer * BUFFER_COLUMNS;
      const int columns = unit.steps * STEP;
      if constexpr (GATED) {
        // lanes 0-15 hold gates and finish tokens 0-7 of 16, lanes 16-31 the up rows and tokens 8-15
        const bool upper = lane >= 16;
        const int feature = unit.feature_tile * FEATURES + rank * (FEATURES / 2) + quarter * 16 + (lane & 15);
        __nv_bfloat16* out = static_cast<__nv_bfloat16*>(args.out) +
                             static_cast<size_t>(unit.token0 + (upper ? 8 : 0)) * args.ldo + feature;
#pragma unroll 1
        for (int column = 0; column < columns; column += 16) {
          float v[16];
          tmem_load16(accumulator + column, v);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float other = __shfl_xor_sync(0xffffffffu, upper ? v[j] : v[8 + j], 16);
            const float gated = hx_gated_fast(upper ? other : v[j], upper ? v[8 + j] : other, args.activation,
                                              args.gate_limit);
            if (feature < args.features) out[static_cast<size_t>(column + j) * args.ldo] = __float2bfloat16_rn(gated);
          }
        }
      } else {
        const int feature = unit.feature_tile * FEATURES + rank * (FEATURES / 2) + quarter * 32 + lane;
        float* out = static_cast<float*>(args.out) + static_cast<size_t>(unit.token0) * args.ldo + feature;
#pragma unroll 1
        for (int column = 0; column < columns; column += 16) {
          float v[16];
          tmem_load16(accumulator + column, v);
          if (feature < args.features) {
#pragma unroll
            for (int j = 0; j < 16; ++j) out[static_cast<size_t>(column + j) * args.ldo] = v[j];
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(cluster_address(&tmem_empty_bar[buffer], 0));
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync();      // neither CTA's memory is read or arrived at any more
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLUMNS);
  }
}

template <bool GATED>
int launch_runs(const CUtensorMap& map_w, const TokenMaps& map_x, const RunsArgs& args, cudaStream_t stream) {
  static std::once_flag once;
  static bool configured = false;
  const int sms = hx_device_sm_count();
  if (sms <= 0) return HX_ERR_LAUNCH;
  std::call_once(once, [] {
    configured = cudaFuncSetAttribute(gemm_tc_runs_kernel<GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      SMEM_BYTES) == cudaSuccess;
    if (!configured) cudaGetLastError();
  });
  if (!configured) {
    hx_set_error("hx_gemm_tc_runs: cannot reserve %d bytes of shared memory", SMEM_BYTES);
    return HX_ERR_LAUNCH;
  }
  hx_launch(gemm_tc_runs_kernel<GATED>, 2 * (sms / 2), THREADS, SMEM_BYTES, stream, map_w, map_x, args);
  return HX_OK;
}

}  // namespace

// Whether hx_gemm_tc_runs takes `rows` rows of tokens in up to `groups` groups.  up_row_offset 0: plain sums.
HX_API int hx_gemm_tc_runs_supports(int rows, int groups, int group_rows, int up_row_offset, int depth, int ldx) {
  return rows > 0 && rows % STEP == 0 && rows / STEP <= MAX_STEPS && groups > 0 && groups <= 32767 &&
         depth > 0 && depth % 8 == 0 && ldx % 8 == 0 && hx_device_sm_count() > 1 &&
         (up_row_offset == 0 || (up_row_offset % 16 == 0 && group_rows % 16 == 0));
}

// x [rows, ldx] bf16, w [groups][group_rows][depth] bf16; tile_group int32 [rows / 32]: the group that 32
// rows belong to, -1 for none (their output is not written).  up_row_offset > 0: out [rows, ldo] bf16 is
// the gated activation of rows f (gate) and up_row_offset + f (up) of the group; 0: out float32 sums.
HX_API int hx_gemm_tc_runs(const void* x, int ldx, int x_capacity_rows, const void* w, int group_rows, int groups,
                           void* out, int ldo, int rows, int features, int depth, int activation, float gate_limit,
                           int up_row_offset, const int* tile_group, int* status, cudaStream_t stream) {
  HX_REQUIRE(hx_gemm_tc_runs_supports(rows, groups, group_rows, up_row_offset, depth, ldx),
             "hx_gemm_tc_runs: rows=%d groups=%d of %d (up rows %d behind) depth=%d ldx=%d are not supported", rows,
             groups, group_rows, up_row_offset, depth, ldx);
  HX_REQUIRE(group_rows > 0 && static_cast<long long>(groups) * group_rows < (1ll << 31),
             "hx_gemm_tc_runs: too many weight rows");
  HX_REQUIRE((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0,
             "hx_gemm_tc_runs: operands must be 16-byte aligned");
  HX_REQUIRE(x_capacity_rows >= rows && ldx >= depth, "hx_gemm_tc_runs: buffer of %d rows of %d for %d of %d",
             x_capacity_rows, ldx, rows, depth);
  HX_REQUIRE(tile_group != nullptr && status != nullptr, "hx_gemm_tc_runs: list of groups or status word missing");
  HX_REQUIRE(up_row_offset >= 0 && features > 0 && up_row_offset + features <= group_rows,
             "hx_gemm_tc_runs: features exceed a group's rows");
  HX_REQUIRE(up_row_offset == 0 || features <= up_row_offset, "hx_gemm_tc_runs: gate rows reach into the up rows");
  HX_REQUIRE(ldo >= features, "hx_gemm_tc_runs: output stride too small");
  const bool gated = up_row_offset > 0;
  const uint64_t weight_rows = static_cast<uint64_t>(groups) * group_rows;
  CUtensorMap map_w;
  TokenMaps map_x;
  int rc = gated ? hx_tensor_map_interleaved("hx_gemm_tc_runs", w, weight_rows, depth, up_row_offset, ROWS, BK, &map_w)
                 : hx_tensor_map("hx_gemm_tc_runs", w, weight_rows, depth, depth, ROWS, BK, true, &map_w);
  for (int box = 0; box < 4 && rc == HX_OK; ++box)
    rc = hx_tensor_map("hx_gemm_tc_runs", x, x_capacity_rows, depth, ldx, 16 << box, BK, true, &map_x.boxes[box]);
  if (rc != HX_OK) return rc;
  const int unit_features = gated ? ROWS : 2 * ROWS;
  const RunsArgs args{out, ldo, rows / STEP, features, (features + unit_features - 1) / unit_features,
                      (depth + BK - 1) / BK, group_rows, activation, gate_limit, tile_group, status};
  HX_REQUIRE(static_cast<long long>(args.steps) * args.feature_tiles < (1ll << 30), "hx_gemm_tc_runs: too many tiles");
  rc = gated ? launch_runs<true>(map_w, map_x, args, stream) : launch_runs<false>(map_w, map_x, args, stream);
  if (rc != HX_OK) return rc;
  HX_CHECK_LAUNCH("hx_gemm_tc_runs");
  return HX_OK;
}
