// Paged causal attention for prompt portions on the 5th-generation tensor cores (tcgen05),
// bfloat16 storage.  The same computation as hx_attention_mma.cu (the reference materialises
// a [heads, T, T] score tensor for it, src/attention/cuda.cu:31-77), with both products as
// tcgen05.mma and the scores, the probabilities and the output in tensor memory.
//
// One CTA takes 128 consecutive query tokens of one request and one head (the M of a product), and
// walks the request's keys in tiles of 64, anchored at key 0.  Warp roles:
//   warp 0      one lane asks for the pages of each tile, its values behind the keys of the next
//               one: the keys of a (page, head) are one contiguous block of the cache and so are
//               its values, so a tile is a handful of bulk copies (cp.async.bulk counted on an
//               mbarrier) into a ring of stages;
//   warp 1      one lane issues S = Q K^T into one of two (four) score buffers in tensor memory;
//   warp 2      one lane issues O += P V;
//   warp 3      (pages of 32 and 64 keys) rewrites the keys of a landed tile piece-major over all 64
//               keys (see below); (pages of 16, heads wider than 128) one lane asks for the values;
//   warps 4-7   softmax: thread r owns query row r.  It reads its row of S from tensor memory,
//               keeps the running maximum and sum in float32 registers and writes the
//               probabilities back over the scores it has read, as TWO bfloat16 terms (P = hi + lo,
//               so the softmax stays a float32 quantity as far as the result can tell).  P is the
//               A operand of O += P V straight from tensor memory, and O stays in tensor memory
//               over all tiles.  The maximum a row's exponentials are taken against is only raised
//               when a tile exceeds it by more than 2^8 (any fixed reference gives the same
//               quotient; float32 has the range), so the pass over O that a new maximum costs is
//               rare;
//   warps 8-11  (heads wider than 128) three more to rewrite keys, or a second group of softmax warps.
//
// Heads of up to 128: two CTAs share an SM.  A tile's way through a CTA is a chain (products,
// softmax, products), and what a CTA spends before its first and after its last tile is several
// microseconds more; two CTAs fill each other's gaps, in the middle and at their ends.  The issuing
// threads are picked by elect.sync (behind `lane == 0` a thread needs 55 ns to issue a product of any
// size).
// Measured (2,048 tokens, 32 heads of 128, in place): 129 us a layer with two lanes of 128 rows in one
// CTA and four issuing threads, 108 with elect.sync, 87 with the softmax's arithmetic in pairs, 91
// with two CTAs and 66 with their keys gathered.
//
// Wider heads leave one CTA an SM (64 KB of queries, a page's values 8 KB).  There a tile of an even turn and
// one of an odd turn go through two groups of softmax warps, with four score buffers, so that scores are
// multiplied while the output products of earlier tiles still run; the reference of a row is told from
// group to group.  Measured (2,048 tokens, 32 heads of 256 over one cached row, window 1,024): 610 us on
// mma.sync, 126 with one group and two buffers (2,850 cycles a tile), 128 with two groups, 112 with four
// buffers (2,330), 104 with queries loaded four pieces a row and values asked for by a thread of their own, 96
// with the 192 coordinates of the values that are wanted (and queries asked for before the second tile).
// Of a CTA's 43,000 cycles 13,000 bring queries and first tiles in and the output out, which a second CTA
// would hide.
//
// Operand layouts.  Nothing is swizzled: every operand is made of "core matrices" of 8 rows
// x 16 bytes (128 contiguous bytes), which is exactly what a page block of the cache is made
// of ([head_dim / 8][slot][8 elements]: eight consecutive slots of one 16-byte piece).  For
// O = P V a page block is used as it lies: 16 keys are the K dimension of an MN-major operand
// (a row of a core matrix is 8 consecutive coordinates of one key, its 8 rows are 8 keys).
// For S = Q K^T the keys are the N operand (K-major), and one product should cover all 64
// keys of the tile, which needs one stride from 8 keys to the next across pages: with pages of 16
// keys a gathering copy (tile::gather4) brings one piece of the four pages at a time, otherwise a warp
// rewrites the tile as [piece][64 keys][16 bytes] (products of one page each are four times
// as many).  Q is written to shared memory by the CTA itself in the same core-matrix form.
//
// A query row's result depends on its own position only (tiles are anchored at key 0, rows do
// not interact).  Requests with fewer than `min_query_len` tokens are left to
// hx_paged_attention.  Every wait is bounded; a wait that runs out sets a status bit, and
// the CTA frees its tensor memory and returns.
#include "hx_tcgen05.cuh"
#include "hx_tensor_map.cuh"

namespace {

constexpr int BLOCK_M = 128;   // query rows per CTA (the MMA's M)
constexpr int BLOCK_N = 64;    // keys per tile
constexpr int WARP_PAGES = 0, WARP_SCORES = 1, WARP_OUTPUT = 2, WARP_REWRITE = 3, WARP_SOFTMAX = 4,
              WARP_MORE = 8;
constexpr int GROUP_STRIDE = 128;             // bytes from one 8-row core matrix to the next row group
constexpr int CHUNK_STRIDE = BLOCK_M * 16;    // bytes from one 16-byte column of Q to the next
constexpr float RAISE_MAXIMUM_BY = 8.0f;      // log2 units a tile must exceed a row's reference by

struct TcPrefillArgs {
  const __nv_bfloat16* q;
  int ldq;
  const __nv_bfloat16* k_cache;
  const __nv_bfloat16* v_cache;
  const int* request_start;     // [requests + 1] first token of each request in the batch
  const int* request_context;   // [requests] tokens cached before this step
  const int* request_table_row;
  const int* block_tables;
  int table_stride;
  __nv_bfloat16* out;
  int ldo;
  int requests;
  int heads;
  int kv_heads;
  int page_size;
  int num_pages;
  float scale;
  int min_query_len;
  int* status;
  int window;       // 0: every earlier key; else the query at p sees key j <= p with p - j < window
  int keep_first;   // ... or j < keep_first (with a window only)
  // Optional, per query head (null: absent).  sinks: the softmax's denominator also holds
  // exp(sinks[h]), a term without key or value.  slopes: the score of key j for the query at
  // position i is lowered by slopes[h] * (i - j).
  const float* sinks = nullptr;
  const float* slopes = nullptr;
  int chunk = 0;          // > 0: positions see each other only inside chunks of this many
  float softcap = 0.0f;   // > 0: the scaled score s becomes softcap * tanh(s / softcap)
  int pack = 1;           // packed kernels: the query heads of a key/value head, side by side in
                          // a tile's rows, token by token; the grid's x counts key/value heads
  int value_dim = 0;      // packed kernels: so many leading coordinates of the values are wanted (a multiple
                          // of 16); the others of `out` are not written
};

// Shared memory holds the queries, key tiles as they land (where they are rewritten), key tiles as
// they are used and value tiles (held until multiplied): 112 KB for a head of 128, so that two CTAs
// fit.
//
// GATHER (pages of 16 keys): a gathering TMA copy brings one 16-byte piece of all 64 keys of a tile
// from its four pages, which is the order the score product wants; the keys land where they are
// used.  Other pages land as they are and are rewritten.
template <int D, bool GATHER>
struct TcConfig {
  static constexpr int kCtas = D <= 128 ? 2 : 1;
  static constexpr int kKeyStages = GATHER ? 0 : 2, kValueStages = 2, kKeyBuffers = GATHER ? 3 : 1;
  static constexpr int kRewriters = GATHER ? 0 : D <= 128 ? 1 : 4;
  // Softmax warps: four, a row a thread; where the CTA has an SM to itself and no warp rewrites keys a second
  // four take every other tile.
  static constexpr int kSoftmaxGroups = D > 128 && GATHER ? 2 : 1;
  static constexpr int kScoreBuffers = 2 * kSoftmaxGroups;      // score tiles in tensor memory
  static constexpr int kThreads = kRewriters <= 1 && kSoftmaxGroups == 1 ? 256 : 384;
  static constexpr int kBarrierBytes = 256;
  static constexpr int kQBytes = BLOCK_M * D * 2;
  static constexpr int kHalfBytes = BLOCK_N * D * 2;          // keys (or values) of a tile
  static constexpr int kSmemBytes = kQBytes + (kKeyStages + kValueStages + kKeyBuffers) * kHalfBytes +
                                    128 /*alignment*/ + kBarrierBytes +
                                    (kSoftmaxGroups > 1 ? 2 * kSoftmaxGroups * BLOCK_M * 4 : 0);
  static constexpr int kScoreColumns = BLOCK_N;               // per score buffer
  static constexpr int kLowTermColumn = BLOCK_N / 2;          // P: hi in columns [0, 32), lo after
  static constexpr int kOutputColumn = kScoreBuffers * BLOCK_N;
  static constexpr int kTmemColumns = D <= 128 ? 256 : 512;
  static_assert(kScoreBuffers * BLOCK_N + D <= kTmemColumns, "tensor memory of a CTA");
  static_assert(kCtas * (kSmemBytes + 1024) <= 228 * 1024, "an SM has 228 KB of shared memory");
};

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Two float32 operations in one instruction, each rounded as its scalar form; and the largest of
// three.  The softmax is bound by the instructions it issues: these take half of them off.
__device__ __forceinline__ uint64_t pair_of(float low, float high) {
  uint64_t pair;
  asm("mov.b64 %0, {%1, %2};" : "=l"(pair) : "f"(low), "f"(high));
  return pair;
}
__device__ __forceinline__ void halves_of(uint64_t pair, float& low, float& high) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(low), "=f"(high) : "l"(pair));
}
__device__ __forceinline__ uint64_t pair_fma(uint64_t x, uint64_t y, uint64_t z) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z));
  return r;
}
__device__ __forceinline__ uint64_t pair_add(uint64_t x, uint64_t y) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
  return r;
}
__device__ __forceinline__ float max_of_3(float x, float y, float z) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(x), "f"(y), "f"(z));
  return r;
}

__device__ __forceinline__ uint32_t pack_bf16(float low, float high) {
  const __nv_bfloat162 pair = __floats2bfloat162_rn(low, high);
  return *reinterpret_cast<const uint32_t*>(&pair);
}

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes,
                                          uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      ::"r"(dst), "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// Four rows of a matrix, the same columns of each, one behind the other into shared memory.
__device__ __forceinline__ void tma_gather_rows(uint32_t dst, const CUtensorMap* map, uint64_t* bar,
                                                int column, const int (&rows)[4]) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5, %6, %7}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(column), "r"(rows[0]), "r"(rows[1]),
      "r"(rows[2]), "r"(rows[3])
      : "memory");
}

template <int D, bool PACKED, bool GATHER>
__global__ __launch_bounds__(TcConfig<D, GATHER>::kThreads, TcConfig<D, GATHER>::kCtas) void
prefill_attention_tc_kernel(const __grid_constant__ CUtensorMap key_pages, const TcPrefillArgs a) {
  using Config = TcConfig<D, GATHER>;
  constexpr int THREADS = Config::kThreads;
  constexpr int K_STAGES = Config::kKeyStages, V_STAGES = Config::kValueStages;
  constexpr int KEY_BUFFERS = Config::kKeyBuffers, REWRITERS = Config::kRewriters;
  constexpr int kDSteps = D / 16;      // k-steps of Q K^T
  constexpr int GROUPS = Config::kSoftmaxGroups, S_BUFFERS = Config::kScoreBuffers;
  // (with two CTAs an SM a second thread that asks costs more than it gives: 68 -> 74 us)
  constexpr bool SPLIT_REQUESTS = GATHER && GROUPS > 1;
  hx_pdl_trigger();

  // which request and which 128-row tile of it is this CTA?  The last rows of a request see
  // the most keys: their CTAs are started first (the grid is walked heads first, then tiles),
  // so the short ones fill the gaps at the end.
  // A row is a token of one head, or with PACKED one of the `pack` heads of a token.
  const int pack = PACKED ? a.pack : 1;
  auto token_of = [&](int row) { return PACKED ? row / pack : row; };
  const int tile_tokens = token_of(BLOCK_M);
  int tile_in_request = 0, tiles_of_request = 0;
  const int request = hx_find_query_tile(a.request_start, a.requests, a.min_query_len,
                                         tile_tokens, blockIdx.z * gridDim.y + blockIdx.y,
                                         tile_in_request, tiles_of_request);
  tile_in_request = tiles_of_request - 1 - tile_in_request;
  if (request < 0) return;      // before any barrier or allocation: the whole CTA leaves

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~static_cast<uintptr_t>(127));
  uint8_t* q_tile = smem;
  uint8_t* k_stages = q_tile + Config::kQBytes;
  uint8_t* v_stages = k_stages + K_STAGES * Config::kHalfBytes;
  uint8_t* keys_by_piece = v_stages + V_STAGES * Config::kHalfBytes;      // [KEY_BUFFERS]
  uint64_t* k_full = reinterpret_cast<uint64_t*>(keys_by_piece + KEY_BUFFERS * Config::kHalfBytes);
  uint64_t* k_empty = k_full + K_STAGES;
  uint64_t* v_full = k_empty + K_STAGES;
  uint64_t* v_empty = v_full + V_STAGES;       // the product has read it
  uint64_t* s_full = v_empty + V_STAGES;       // [S_BUFFERS] scores of tile t in buffer t % S_BUFFERS
  uint64_t* p_full = s_full + S_BUFFERS;       // [S_BUFFERS] its probabilities are in place
  uint64_t* o_full = p_full + S_BUFFERS;       // [S_BUFFERS] its output product is done
  uint64_t* k_ready = o_full + S_BUFFERS;      // [KEY_BUFFERS] the tile's keys are rewritten
  uint64_t* k_done = k_ready + KEY_BUFFERS;    // [KEY_BUFFERS] its scores have read them
  uint64_t* q_ready = k_done + KEY_BUFFERS;    // the query tile is in shared memory
  uint64_t* told_bar = q_ready + 1;            // [GROUPS][4] a group's warp has told its reference
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(told_bar + (GROUPS > 1 ? 4 * GROUPS : 0));
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_holder + 1);
  constexpr int kBarriers = 2 * K_STAGES + 2 * V_STAGES + 3 * S_BUFFERS + 2 * KEY_BUFFERS + 1 +
                            (GROUPS > 1 ? 4 * GROUPS : 0);
  static_assert(kBarriers * 8 + 8 <= Config::kBarrierBytes, "the place of barriers, tensor memory's address and flag");
  // two groups of softmax warps: [GROUPS][BLOCK_M] references they tell each other, then their sums
  float* told = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(k_full) + Config::kBarrierBytes);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int head0 = PACKED ? blockIdx.x * pack : blockIdx.x;      // of a token's first row
  const int kv_head = PACKED ? blockIdx.x : blockIdx.x / (a.heads / a.kv_heads);
  auto head_of = [&](int row, int token) { return PACKED ? head0 + row - token * pack : head0; };
  const int q_begin = a.request_start[request];
  const int q_len = a.request_start[request + 1] - q_begin;
  const int context = a.request_context[request];
  const int token0 = tile_in_request * tile_tokens;           // first token of the CTA's rows
  const int tokens_here = min(tile_tokens, q_len - token0);
  const int rows_here = PACKED ? tokens_here * pack : tokens_here;
  const int last_key = context + token0 + tokens_here - 1;    // last key any row here sees
  // With a window or chunks the CTA walks the key tiles that hold kept first keys and then the
  // tiles from the one with the first key its FIRST row sees; `skipped` tiles lie
  // between the two runs.  Every loop below counts TURNS: turn t works on key tile
  // tile_at(t); rings and barriers go by turns, positions and pages by key tiles.  Keys from
  // keep_first up to first_needed are seen by no row of the CTA: their pages may have been
  // given back and are not read.
  const int first_needed = hx_first_seen(context + token0, a.window, a.chunk);
  const int kept_tiles =
      a.window > 0 ? min((a.keep_first + BLOCK_N - 1) / BLOCK_N, first_needed / BLOCK_N) : 0;
  const int skipped = first_needed / BLOCK_N - kept_tiles;
  auto tile_at = [&](int turn) { return turn < kept_tiles ? turn : turn + skipped; };
  const int n_tiles = last_key / BLOCK_N + 1 - skipped;
  const int page_size = GATHER ? BLOCK_N / 4 : a.page_size;
  const int pages_per_tile = BLOCK_N / page_size;
  const uint32_t page_bytes = static_cast<uint32_t>(page_size) * D * 2;
  const uint32_t piece_stride = static_cast<uint32_t>(page_size) * 16;   // next 16-byte piece of a key

  if (threadIdx.x == 0) {
    for (int s = 0; s < K_STAGES; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], REWRITERS);
    }
    for (int s = 0; s < V_STAGES; ++s) {
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    for (int b = 0; b < S_BUFFERS; ++b) {
      mbar_init(&s_full[b], 1);
      mbar_init(&p_full[b], 4);   // one arrival per softmax warp
      mbar_init(&o_full[b], 1);
    }
    for (int b = 0; b < KEY_BUFFERS; ++b) {
      mbar_init(&k_ready[b], GATHER ? 1 : REWRITERS);      // the copies, or the warps that rewrite
      mbar_init(&k_done[b], 1);
    }
    if (GROUPS > 1) {
      for (int i = 0; i < 4 * GROUPS; ++i) mbar_init(&told_bar[i], 1);
    }
    mbar_init(q_ready, THREADS / 32 - WARP_SCORES);      // one arrival per warp that loads queries
    *failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == WARP_SCORES) tmem_alloc(tmem_holder, Config::kTmemColumns);
  hx_pdl_wait();

  tc_fence_before();
  __syncthreads();      // barriers and tensor memory are there; nothing else is waited for here
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;

  // ---- the query tile: [D / 8 pieces][16 row groups][8 rows][16 bytes], written by the warps from
  // WARP_SCORES on while the first pages are on their way.  All of a thread's loads are in flight
  // together (one after the other they cost the CTA 6 us); a warp takes four neighbouring pieces of eight
  // rows, which it stores to different banks (32 pieces of a row, 2 KB apart, cost 4 us more).
  if (warp >= WARP_SCORES) {
    constexpr int kLoaders = THREADS / 32 - WARP_SCORES;      // warps
    constexpr int kPieces = D / 8, kItems = BLOCK_M / 8 * kPieces;
    constexpr int kTurns = (kItems + 4 * kLoaders - 1) / (4 * kLoaders);
    uint4 values[kTurns];
    auto place = [&](int turn, int& row, int& piece) {
      const int item = (turn * kLoaders + warp - WARP_SCORES) * 4 + (lane >> 3);
      const int row_group = item / kPieces;
      piece = item - row_group * kPieces;
      row = 8 * row_group + (lane & 7);
      return item < kItems;
    };
#pragma unroll
    for (int i = 0; i < kTurns; ++i) {
      int row, piece;
      values[i] = make_uint4(0u, 0u, 0u, 0u);
      if (place(i, row, piece) && row < rows_here) {
        const int token = token_of(row);
        values[i] = *reinterpret_cast<const uint4*>(
            a.q + static_cast<size_t>(q_begin + token0 + token) * a.ldq +
            static_cast<size_t>(head_of(row, token)) * D + piece * 8);
      }
    }
#pragma unroll
    for (int i = 0; i < kTurns; ++i) {
      int row, piece;
      if (place(i, row, piece))
        *reinterpret_cast<uint4*>(q_tile + piece * CHUNK_STRIDE + (row >> 3) * GROUP_STRIDE +
                                  (row & 7) * 16) = values[i];
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(q_ready);
  }

  if (warp == WARP_PAGES || (SPLIT_REQUESTS && warp == WARP_REWRITE)) {
    // ------------------------------------------------------------ page requests
    if (hx_elect_one()) {
      const int* table = a.block_tables +
                         static_cast<size_t>(a.request_table_row[request]) * a.table_stride;
      const int last_page = last_key / page_size;
      auto pages_of = [&](int turn, int (&pages)[4]) {
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const int index = tile_at(turn) * pages_per_tile + p;
          // a page that holds no kept key and ends before the first key needed is not read
          const bool wanted = index * page_size < a.keep_first ||
                              (index + 1) * page_size > first_needed;
          int page = -2;                                             // -2: none
          if (p < pages_per_tile && index <= last_page && wanted) {
            page = table[index];
            if (page < 0 || page >= a.num_pages) page = -1;          // reported where it is asked for
          }
          pages[p] = page;
        }
      };
      // the copies of a tile's page blocks into a stage that is free
      auto request_tile = [&](const __nv_bfloat16* cache, uint8_t* stage, uint64_t* full,
                              const int (&pages)[4], uint32_t bytes) {
        uint32_t expected = 0;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          if (pages[p] == -1) atomicOr(a.status, HX_FLAG_BAD_PAGE);
          if (pages[p] >= 0) expected += page_bytes;
        }
        if (PACKED) expected = expected / page_bytes * bytes;
        mbar_expect_tx(full, expected);
        const uint32_t base = smem_u32(stage);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          if (pages[p] >= 0) {
            const size_t block = (static_cast<size_t>(pages[p]) * a.kv_heads + kv_head) * page_bytes;
            bulk_copy(base + p * page_bytes, reinterpret_cast<const uint8_t*>(cache) + block,
                      PACKED ? bytes : page_bytes, full);
          }
        }
      };
      auto request_keys = [&](int tile, const int (&pages)[4]) {
        if constexpr (GATHER) {
          const int buffer = tile % KEY_BUFFERS;
          if (!mbar_wait(&k_done[buffer], (static_cast<uint32_t>(tile / KEY_BUFFERS) & 1u) ^ 1u)) return false;
          // no page: any row will do, no key of it is seen
          int rows[4];
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            if (pages[p] == -1) atomicOr(a.status, HX_FLAG_BAD_PAGE);
            rows[p] = max(pages[p], 0) * a.kv_heads + kv_head;
          }
          mbar_expect_tx(&k_ready[buffer], Config::kHalfBytes);
          const uint32_t target = smem_u32(keys_by_piece + buffer * Config::kHalfBytes);
#pragma unroll 4
          for (int piece = 0; piece < D / 8; ++piece)
            tma_gather_rows(target + piece * (BLOCK_N * 16), &key_pages, &k_ready[buffer],
                            piece * (BLOCK_N / 4) * 8, rows);
        } else {
          const int stage = tile % K_STAGES;
          if (!mbar_wait(&k_empty[stage], (static_cast<uint32_t>(tile / K_STAGES) & 1u) ^ 1u)) return false;
          request_tile(a.k_cache, k_stages + stage * Config::kHalfBytes, &k_full[stage], pages, page_bytes);
        }
        return true;
      };
      auto request_values = [&](int tile, const int (&pages)[4]) {
        const int stage = tile % V_STAGES;
        if (!mbar_wait(&v_empty[stage], (static_cast<uint32_t>(tile / V_STAGES) & 1u) ^ 1u)) return false;
        request_tile(a.v_cache, v_stages + stage * Config::kHalfBytes, &v_full[stage], pages,
                     static_cast<uint32_t>(page_size) * a.value_dim * 2);
        return true;
      };
      // Turn t asks for the keys of tile t and for the values of tile t - 1, which are wanted
      // later: their keys are (rewritten and) multiplied, and the softmax runs, in between.  With two threads
      // that ask, one asks for values alone, as soon as there is room.
      const bool asks_keys = !SPLIT_REQUESTS || warp == WARP_PAGES;
      const bool asks_values = !SPLIT_REQUESTS || warp != WARP_PAGES;
      // (behind the first tile's keys and the queries, which the first products wait for)
      bool waited = !SPLIT_REQUESTS;
      int pages[4], value_pages[4];
      pages_of(0, pages);
      for (int tile = 0; tile <= n_tiles && !*failed; ++tile) {
        int next_pages[4];
        if (tile + 1 < n_tiles) pages_of(tile + 1, next_pages);      // in flight during the waits
        bool free = true;
        if (!waited && (tile > 0 || !asks_keys)) {
          free = mbar_wait(q_ready, 0);
          waited = true;
        }
        if (free && asks_keys && tile < n_tiles) free = request_keys(tile, pages);
        if (free && asks_values && tile > 0) free = request_values(tile - 1, value_pages);
        if (!free) {
          atomicOr(a.status, HX_FLAG_WAIT_TIMEOUT);
          *failed = 1;
          break;
        }
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          value_pages[p] = pages[p];
          pages[p] = next_pages[p];
        }
      }
    }
  } else if (!GATHER && (warp == WARP_REWRITE || (warp >= WARP_MORE && warp < WARP_MORE + REWRITERS - 1))) {
    if constexpr (!GATHER) {
    // ------------------------------------------------------ keys, piece by piece
    // The score product wants all 64 keys of the tile at one stride, but every page block
    // holds its own keys piece-major: this warp rewrites a landed tile as
    // [piece][64 keys][16 bytes] into buffer tile % KEY_BUFFERS.
    bool ok = true;
    // this warp's share of the pieces
    constexpr int kShare = D / 8 / REWRITERS;
    const int first_piece = warp == WARP_REWRITE ? 0 : (warp - WARP_MORE + 1) * kShare;
    // where keys `lane` and `lane + 32` of a tile sit inside the landed page blocks
    const uint32_t source_low = (lane / page_size) * page_bytes + (lane % page_size) * 16;
    const uint32_t source_high =
        ((lane + 32) / page_size) * page_bytes + ((lane + 32) % page_size) * 16;
    for (int tile = 0; tile < n_tiles && ok && !*failed; ++tile) {
      if (lane == 0) {
        ok = mbar_wait(&k_full[tile % K_STAGES], static_cast<uint32_t>(tile / K_STAGES) & 1u);
        // the score products that read this buffer KEY_BUFFERS tiles ago are done (the barrier's
        // next phase needs this very rewrite, so no phase can be mistaken for another)
        if (ok && tile >= KEY_BUFFERS)
          ok = mbar_wait(&k_done[tile % KEY_BUFFERS],
                         static_cast<uint32_t>((tile - KEY_BUFFERS) / KEY_BUFFERS) & 1u);
        if (!ok) {
          atomicOr(a.status, HX_FLAG_WAIT_TIMEOUT);
          *failed = 1;
        }
      }
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) break;
      const uint32_t source = smem_u32(k_stages + (tile % K_STAGES) * Config::kHalfBytes) +
                              first_piece * piece_stride;
      const uint32_t target =
          smem_u32(keys_by_piece + (tile % KEY_BUFFERS) * Config::kHalfBytes) + lane * 16 +
          first_piece * (BLOCK_N * 16);
      // eight pieces at a time: all their loads are in flight before the first store
#pragma unroll
      for (int piece0 = 0; piece0 < kShare; piece0 += 8) {
        uint4 low[8], high[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (piece0 + i >= kShare) continue;      // (a head of 112: fourteen pieces)
          asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(low[i].x), "=r"(low[i].y), "=r"(low[i].z), "=r"(low[i].w)
                       : "r"(source + source_low + (piece0 + i) * piece_stride));
          asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                       : "=r"(high[i].x), "=r"(high[i].y), "=r"(high[i].z), "=r"(high[i].w)
                       : "r"(source + source_high + (piece0 + i) * piece_stride));
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (piece0 + i >= kShare) continue;
          asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(
                           target + (piece0 + i) * (BLOCK_N * 16)),
                       "r"(low[i].x), "r"(low[i].y), "r"(low[i].z), "r"(low[i].w) : "memory");
          asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(
                           target + (piece0 + i) * (BLOCK_N * 16) + 512),
                       "r"(high[i].x), "r"(high[i].y), "r"(high[i].z), "r"(high[i].w) : "memory");
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&k_ready[tile % KEY_BUFFERS]);
        mbar_arrive(&k_empty[tile % K_STAGES]);      // the landed copy may be overwritten
      }
    }
    }
  } else if (warp == WARP_SCORES) {
    // ------------------------------------------------------------ score products
    if (hx_elect_one()) {
      constexpr uint32_t idesc_scores = make_idesc(BLOCK_M, BLOCK_N);
      // Descriptors differ from product to product only in their start address (the low 14
      // bits, in units of 16 bytes): build one of each kind and add offsets.
      const uint64_t desc_q = make_smem_desc_plain(smem_u32(q_tile), CHUNK_STRIDE, GROUP_STRIDE);
      const uint64_t desc_k0 =
          make_smem_desc_plain(smem_u32(keys_by_piece), BLOCK_N * 16, GROUP_STRIDE);
      constexpr uint32_t kKeyBufferStep = Config::kHalfBytes >> 4;
      constexpr uint32_t kChunkPairStep = (2 * CHUNK_STRIDE) >> 4;      // 16 coordinates of Q on
      constexpr uint32_t kKeyPiecePairStep = (2 * BLOCK_N * 16) >> 4;   // 16 coordinates of the keys on
      if (!mbar_wait(q_ready, 0)) {
        atomicOr(a.status, HX_FLAG_WAIT_TIMEOUT);
        *failed = 1;
      }
      // S[tile % S_BUFFERS] = Q K_tile^T: one product of 64 keys per 16 coordinates.  The buffer held the
      // probabilities of tile - S_BUFFERS, which the output product must have read.
      for (int tile = 0; tile < n_tiles && !*failed; ++tile) {
        const int b = tile % S_BUFFERS;
        if (!mbar_wait(&k_ready[tile % KEY_BUFFERS], static_cast<uint32_t>(tile / KEY_BUFFERS) & 1u) ||
            (tile >= S_BUFFERS &&
             !mbar_wait(&o_full[b], static_cast<uint32_t>((tile - S_BUFFERS) / S_BUFFERS) & 1u))) {
          atomicOr(a.status, HX_FLAG_WAIT_TIMEOUT);
          *failed = 1;
          break;
        }
        tc_fence_after();
        const uint64_t desc_k = desc_k0 + (tile % KEY_BUFFERS) * kKeyBufferStep;
        const uint32_t target = tmem_base + b * Config::kScoreColumns;
#pragma unroll
        for (int k = 0; k < kDSteps; ++k)
          umma_bf16(target, desc_q + k * kChunkPairStep, desc_k + k * kKeyPiecePairStep,
                    idesc_scores, k > 0 ? 1u : 0u);
        umma_commit(&s_full[b]);
        umma_commit(&k_done[tile % KEY_BUFFERS]);
      }
    }
  } else if (warp == WARP_OUTPUT) {
    // ----------------------------------------------------------- output products
    if (hx_elect_one()) {
      const uint32_t idesc_output = make_idesc_b_mn_major(BLOCK_M, PACKED ? a.value_dim : D);
      // values: MN-major, the next 8 keys are 128 bytes on, the next 8 coordinates one piece on
      const uint64_t desc_v0 = make_smem_desc_plain(smem_u32(v_stages), GROUP_STRIDE, piece_stride);
      constexpr uint32_t kStageStep = Config::kHalfBytes >> 4;
      // where the 16 keys of each product of P V start inside a stage's value half
      uint32_t value_step[BLOCK_N / 16];
#pragma unroll
      for (int g = 0; g < BLOCK_N / 16; ++g) {
        const int key = g * 16;
        value_step[g] = ((key / page_size) * page_bytes + (key % page_size) * 16) >> 4;
      }
      const uint32_t target = tmem_base + Config::kOutputColumn;
      for (int tile = 0; tile < n_tiles && !*failed; ++tile) {
        // the probabilities of this tile lie where its scores were
        const int b = tile % S_BUFFERS, s = tile % V_STAGES;
        if (!mbar_wait(&p_full[b], static_cast<uint32_t>(tile / S_BUFFERS) & 1u) ||
            !mbar_wait(&v_full[s], static_cast<uint32_t>(tile / V_STAGES) & 1u)) {
          atomicOr(a.status, HX_FLAG_WAIT_TIMEOUT);
          *failed = 1;
          break;
        }
        tc_fence_after();
        const uint64_t desc_v = desc_v0 + s * kStageStep;
        const uint32_t p_hi = tmem_base + b * Config::kScoreColumns;
        const uint32_t p_lo = p_hi + Config::kLowTermColumn;
        // O += P V_tile: 16 keys (8 columns of P) per product, the hi and the lo term of P
#pragma unroll
        for (int g = 0; g < BLOCK_N / 16; ++g) {
          umma_bf16_a_tmem(target, p_hi + g * 8, desc_v + value_step[g], idesc_output,
                           (tile > 0 || g > 0) ? 1u : 0u);
          umma_bf16_a_tmem(target, p_lo + g * 8, desc_v + value_step[g], idesc_output, 1u);
        }
        umma_commit(&v_empty[s]);
        umma_commit(&o_full[b]);                     // O holds this tile; its P has been read
      }
    }
  } else if (warp >= WARP_SOFTMAX && warp < WARP_SOFTMAX + 4 * GROUPS) {
    // ------------------------------------------------------------------ softmax
    // With two groups a row has a thread in each: one takes the even tiles, the other the odd ones.  The
    // reference goes from tile to tile through shared memory, told before the exponentials are taken; each
    // keeps the sum of its own tiles.
    const int softmax_group = GROUPS > 1 ? (warp - WARP_SOFTMAX) >> 2 : 0;
    const int quarter = warp & 3;      // tensor-memory lanes [32 * quarter, 32 * quarter + 32)
    const int row = quarter * 32 + lane;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t output_base = lane_base + Config::kOutputColumn;
    const int my_token = token_of(row);
    const int head = min(head_of(row, my_token), a.heads - 1);
    const int q_position = context + token0 + my_token;             // the last key this row sees
    float row_max = -INFINITY;      // the reference of this row's exponentials, in log2 units
    float row_sum = 0.0f;
    const float scale_log2 = a.scale * 1.4426950408889634f;
    const int row_first = hx_first_seen(q_position, a.window, a.chunk);     // first key this row sees
    // a slope per position of distance, in the same log2 units (0: none)
    const float slope_log2 = a.slopes != nullptr ? a.slopes[head] * 1.4426950408889634f : 0.0f;
    const bool plain_scores = a.softcap <= 0.0f && a.slopes == nullptr && a.scale > 0.0f;
    const float factor = plain_scores ? scale_log2 : 1.0f;
    const uint64_t factor_pair = pair_of(factor, factor), minus_one = pair_of(-1.0f, -1.0f);
    bool ok = true;

    // One lane waits and looks at the failure flag, all lanes get the same answer (what
    // follows a wait is warp-wide: tensor-memory loads and stores need the warp together).
    auto wait_for = [&](uint64_t* bar, uint32_t parity_bit) {
      int state = 0;      // 0: go on, 1: this wait ran out, 2: somebody else failed
      if (lane == 0) state = *failed ? 2 : (mbar_wait(bar, parity_bit) ? 0 : 1);
      state = __shfl_sync(0xffffffffu, state, 0);
      if (state == 1 && lane == 0) {
        atomicOr(a.status, HX_FLAG_WAIT_TIMEOUT);
        *failed = 1;
      }
      return state == 0;
    };

    for (int tile = softmax_group; tile < n_tiles && ok; tile += GROUPS) {
      const int b = tile % S_BUFFERS;
      ok = wait_for(&s_full[b], static_cast<uint32_t>(tile / S_BUFFERS) & 1u);
      if (!ok) break;
      tc_fence_after();
      const uint32_t score_base = lane_base + b * Config::kScoreColumns;
      // ---- this row's scores of the tile, in units of log2(e) so that exp is one ex2
      float p[BLOCK_N];
      {
        uint32_t r[4][16];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_load16_issue(score_base + c * 16, r[c]);
        tmem_load_wait();
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 16; ++i) p[c * 16 + i] = __uint_as_float(r[c][i]);
      }
      // plain scores stay as they are until the exponential, whose argument is one multiply-add
      // (a positive factor does not change which is the largest); the others are scaled here
      if (a.softcap > 0.0f) {
        hx_level_off_fast(p, a.scale / a.softcap, a.softcap * 1.4426950408889634f);
      } else if (!plain_scores) {
#pragma unroll
        for (int i = 0; i < BLOCK_N; ++i) p[i] *= scale_log2;
      }
      const int key0 = tile_at(tile) * BLOCK_N;
      if (a.slopes != nullptr) {
        const float distance0 = static_cast<float>(q_position - key0);
#pragma unroll
        for (int i = 0; i < BLOCK_N; ++i)
          p[i] = fmaf(-slope_log2, distance0 - static_cast<float>(i), p[i]);
      }
      if (key0 + BLOCK_N - 1 > q_position) {
#pragma unroll
        for (int i = 0; i < BLOCK_N; ++i)
          if (key0 + i > q_position) p[i] = -INFINITY;
      }
      if (key0 < row_first) {
        // keys of the tile lie in front of what this row sees: they count only when kept
#pragma unroll
        for (int i = 0; i < BLOCK_N; ++i)
          if (key0 + i < row_first && key0 + i >= a.keep_first) p[i] = -INFINITY;
      }
      float part_max[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) part_max[u] = max_of_3(p[u], p[u + 4], p[u + 8]);
#pragma unroll
      for (int i = 12; i + 8 <= BLOCK_N; i += 8)
#pragma unroll
        for (int u = 0; u < 4; ++u) part_max[u] = max_of_3(part_max[u], p[i + u], p[i + 4 + u]);
#pragma unroll
      for (int u = 0; u < 4; ++u) part_max[u] = fmaxf(part_max[u], p[BLOCK_N - 4 + u]);
      const float tile_max = factor * fmaxf(max_of_3(part_max[0], part_max[1], part_max[2]), part_max[3]);
      // without a window key 0 is visible to every row and the reference is finite from the
      // first tile on; with one a row may see nothing of the CTA's first tiles and keeps
      // -inf as its reference (and zeros as its probabilities) until it does
      const float own_max = row_max;      // what the sum is taken against
      if (GROUPS > 1 && tile > 0) {
        const int other = softmax_group ^ 1;
        ok = wait_for(&told_bar[4 * other + quarter], static_cast<uint32_t>((tile - 1) / GROUPS) & 1u);
        if (!ok) break;
        row_max = told[other * BLOCK_M + row];
      }
      const float old_max = row_max;
      const bool raised = tile > 0 && __any_sync(0xffffffffu, tile_max > old_max + RAISE_MAXIMUM_BY);
      if (tile == 0) row_max = tile_max;
      else if (raised) row_max = fmaxf(old_max, tile_max);
      if (GROUPS > 1) {
        told[softmax_group * BLOCK_M + row] = row_max;
        __syncwarp();
        if (lane == 0) mbar_arrive(&told_bar[4 * softmax_group + quarter]);
      }
      if (GROUPS > 1 && row_max != own_max) row_sum *= own_max == -INFINITY ? 0.0f : fast_exp2(own_max - row_max);
      if (raised) {
        // ---- a new reference: what O holds was taken against the old one.  The
        // product of the previous tile must have landed; the product of this tile waits for
        // this warp's arrival below.  (o_full[b] completes a phase for every S_BUFFERS-th tile;
        // its previous phase was complete before the scores of the previous tile were.)
        const float correction = old_max == -INFINITY ? 0.0f : fast_exp2(old_max - row_max);
        if (GROUPS == 1) row_sum *= correction;
        ok = wait_for(&o_full[(tile - 1) % S_BUFFERS],
                      static_cast<uint32_t>((tile - 1) / S_BUFFERS) & 1u);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int d0 = 0; d0 < D; d0 += 32) {
          if (PACKED && d0 >= a.value_dim) break;
          const bool both = d0 + 16 < D;      // (compile time: D is a multiple of 16)
          uint32_t r0[16], r1[16];
          tmem_load16_issue(output_base + d0, r0);
          if (both) tmem_load16_issue(output_base + d0 + 16, r1);
          tmem_load_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            r0[i] = __float_as_uint(__uint_as_float(r0[i]) * correction);
            if (both) r1[i] = __float_as_uint(__uint_as_float(r1[i]) * correction);
          }
          tmem_store16_raw(output_base + d0, r0);
          if (both) tmem_store16_raw(output_base + d0 + 16, r1);
        }
      }
      uint64_t part_sum[4] = {0, 0, 0, 0};
      const float reference = row_max == -INFINITY ? 0.0f : row_max;
      const uint64_t reference_pair = pair_of(-reference, -reference);
#pragma unroll
      for (int i = 0; i < BLOCK_N; i += 2) {
        float x0, x1;
        halves_of(pair_fma(pair_of(p[i], p[i + 1]), factor_pair, reference_pair), x0, x1);
        p[i] = fast_exp2(x0);
        p[i + 1] = fast_exp2(x1);
        part_sum[(i / 2) % 4] = pair_add(part_sum[(i / 2) % 4], pair_of(p[i], p[i + 1]));
      }
      {
        float low, high;
        halves_of(pair_add(pair_add(part_sum[0], part_sum[1]), pair_add(part_sum[2], part_sum[3])), low,
                  high);
        row_sum += low + high;
      }

      // ---- P = hi + lo over the scores just read: hi is p rounded to bfloat16, lo is p - hi
      // (exact in float32) rounded the same way: together 16 bits of p.  Two keys per column,
      // the earlier key in the lower half.
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float p0 = p[c * 32 + 2 * i], p1 = p[c * 32 + 2 * i + 1];
          hi[i] = pack_bf16(p0, p1);
          float rest0, rest1;
          halves_of(pair_fma(pair_of(__uint_as_float(hi[i] << 16), __uint_as_float(hi[i] & 0xffff0000u)),
                             minus_one, pair_of(p0, p1)), rest0, rest1);
          lo[i] = pack_bf16(rest0, rest1);
        }
        tmem_store16_raw(score_base + c * 16, hi);
        tmem_store16_raw(score_base + Config::kLowTermColumn + c * 16, lo);
      }
      tmem_store_wait();

      // ---- value rows behind the last key hold whatever the pages (or an earlier tile)
      // left there; a NaN would survive a zero probability, so they are cleared.
      // The same goes for the keys between the kept ones and the first key needed, whose pages
      // were not read.
      const int first_stale = last_key + 1 - key0;
      const int unseen_from = a.keep_first - key0;      // tile-relative; may be negative
      const int unseen_to = first_needed - key0;        // exclusive
      const bool has_unseen = unseen_to > 0 && unseen_from < BLOCK_N &&
                              unseen_from < unseen_to;
      if (first_stale < BLOCK_N || has_unseen) {
        ok = wait_for(&v_full[tile % V_STAGES], static_cast<uint32_t>(tile / V_STAGES) & 1u);
        if (!ok) break;
        uint8_t* v_half = v_stages + (tile % V_STAGES) * Config::kHalfBytes;
        for (int index = row; index < BLOCK_N * (D / 8); index += 128) {
          const int key = index / (D / 8);
          const int piece = index - key * (D / 8);
          if (key >= first_stale || (has_unseen && key >= unseen_from && key < unseen_to))
            *reinterpret_cast<uint4*>(v_half + (key / page_size) * page_bytes +
                                      (piece * page_size + key % page_size) * 16) =
                make_uint4(0u, 0u, 0u, 0u);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[b]);
    }

    // ---- both groups' sums against the last reference, which is the largest (the barrier is met whatever went
    // wrong: every wait in front of it ends)
    if constexpr (GROUPS > 1) {
      // (a reference that was told is read before the next is: no place is written too early)
      float* sums = told + GROUPS * BLOCK_M;
      asm volatile("bar.sync 1, %0;" ::"n"(128 * GROUPS) : "memory");
      told[softmax_group * BLOCK_M + row] = row_max;
      sums[softmax_group * BLOCK_M + row] = row_sum;
      asm volatile("bar.sync 1, %0;" ::"n"(128 * GROUPS) : "memory");
      const float max0 = told[row], max1 = told[BLOCK_M + row];
      row_max = fmaxf(max0, max1);
      row_sum = (max0 == -INFINITY ? 0.0f : sums[row] * fast_exp2(max0 - row_max)) +
                (max1 == -INFINITY ? 0.0f : sums[BLOCK_M + row] * fast_exp2(max1 - row_max));
    }
    // ---- a commit covers every product its thread issued before it: the last tile says all of
    // them are done
    if (ok) {
      ok = wait_for(&o_full[(n_tiles - 1) % S_BUFFERS],
                    static_cast<uint32_t>((n_tiles - 1) / S_BUFFERS) & 1u);
      if (ok) {
        tc_fence_after();
        float inverse = 1.0f / row_sum;
        if (a.sinks != nullptr) {
          // the sink joins the finished row: with M = max(m, s) the result is
          // o 2^(m - M) / (l 2^(m - M) + 2^(s - M)), everything in log2 units
          const float sink_log2 = a.sinks[head] * 1.4426950408889634f;
          const float top = fmaxf(row_max, sink_log2);
          const float keep = row_max == -INFINITY ? 0.0f : fast_exp2(row_max - top);
          inverse = keep / (row_sum * keep + fast_exp2(sink_log2 - top));
        }
        // A group takes its share of the coordinates.  The rows gather in shared memory, where the queries and
        // values were (every product is done), 16 bytes apart more than they are long, so that a warp's rows
        // use different banks (a thread's own row, 16 bytes at a time, is half a sector a store).  With two CTAs
        // an SM they leave with whole rows side by side, with one by a bulk copy each (the other way round: heads
        // of 128 67 -> 70 us, heads of 256 over pages of 16 96 -> 101; pages of 32, 32 heads of 224 over one cached row,
        // 2,048 tokens 127 -> 137, eight decoded tokens behind 500 19.5 -> 21.9).  Heads of 64 over pages of 16, a line of
        // 128 bytes each, go straight from the registers (2,048 tokens of 32 heads 57.0 -> 55.6; over pages of 32 72 -> 76).
        constexpr bool LINE_ROWS = D == 64 && GATHER;
        constexpr int SHARE = D / GROUPS, ROW_BYTES = SHARE * 2 + 16;
        static_assert(4 * GROUPS * 32 * ROW_BYTES <= Config::kQBytes + (K_STAGES + V_STAGES) * Config::kHalfBytes,
                      "the rows' place");
        uint8_t* gathered = q_tile + ((4 * softmax_group + quarter) * 32 + lane) * ROW_BYTES;
        __nv_bfloat16* own_row = a.out + static_cast<size_t>(q_begin + token0 + my_token) * a.ldo +
                                 static_cast<size_t>(head) * D;
        const int share = min(SHARE, a.value_dim - softmax_group * SHARE);      // coordinates that are wanted
#pragma unroll
        for (int d0 = 0; d0 < SHARE; d0 += 32) {
          if (d0 >= share) break;
          const bool both = d0 + 16 < SHARE;
          uint32_t r[2][16];
          tmem_load16_issue(output_base + softmax_group * SHARE + d0, r[0]);
          if (both) tmem_load16_issue(output_base + softmax_group * SHARE + d0 + 16, r[1]);
          tmem_load_wait();
#pragma unroll
          for (int h = 0; h < (both ? 2 : 1); ++h)
#pragma unroll
            for (int d = 0; d < 16; d += 8) {
              uint4 packed;
              __nv_bfloat162* pairs = reinterpret_cast<__nv_bfloat162*>(&packed);
#pragma unroll
              for (int i = 0; i < 4; ++i)
                pairs[i] = __floats2bfloat162_rn(__uint_as_float(r[h][d + 2 * i]) * inverse,
                                                 __uint_as_float(r[h][d + 2 * i + 1]) * inverse);
              if constexpr (LINE_ROWS) {
                if (row < rows_here) *reinterpret_cast<uint4*>(own_row + d0 + h * 16 + d) = packed;
              } else {
                *reinterpret_cast<uint4*>(gathered + (d0 + h * 16 + d) * 2) = packed;
              }
            }
        }
        if constexpr (Config::kCtas == 1) {
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          if (row < rows_here && share > 0) {
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(
                             own_row + softmax_group * SHARE),
                         "r"(smem_u32(gathered)), "r"(2 * share)
                         : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
          }
        } else if constexpr (!LINE_ROWS) {
          __syncwarp();
          constexpr int PIECES = SHARE / 8;
          const uint8_t* of_warp = q_tile + quarter * 32 * ROW_BYTES;
#pragma unroll 4
          for (int item = lane; item < 32 * PIECES; item += 32) {
            const int r = item / PIECES, piece = item - r * PIECES, out_row = quarter * 32 + r;
            if (out_row < rows_here && 8 * piece < share) {
              const int token = token_of(out_row);
              *reinterpret_cast<uint4*>(a.out + static_cast<size_t>(q_begin + token0 + token) * a.ldo +
                                        static_cast<size_t>(head_of(out_row, token)) * D + piece * 8) =
                  *reinterpret_cast<const uint4*>(of_warp + r * ROW_BYTES + piece * 16);
            }
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == WARP_SCORES) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Config::kTmemColumns);
  }
}

template <int D, bool PACKED, bool GATHER>
int launch_with(const CUtensorMap& key_pages, const TcPrefillArgs& a, int tiles, cudaStream_t stream) {
  using Config = TcConfig<D, GATHER>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(prefill_attention_tc_kernel<D, PACKED, GATHER>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             Config::kSmemBytes) != cudaSuccess) {
      cudaGetLastError();
      hx_set_error("hx_prefill_attention_tc: cannot reserve %d bytes of shared memory",
                   Config::kSmemBytes);
      return HX_ERR_LAUNCH;
    }
    configured = true;
  }
  // `tiles` bounds tiles of 256 tokens, or exactly the packed ones
  const dim3 grid(PACKED ? a.heads / a.pack : a.heads, tiles, PACKED ? 1 : 256 / BLOCK_M);
  hx_launch(prefill_attention_tc_kernel<D, PACKED, GATHER>, grid, Config::kThreads, Config::kSmemBytes,
            stream, key_pages, a);
  return HX_OK;
}

template <int D, bool PACKED = false>
int launch(const TcPrefillArgs& a, int tiles, cudaStream_t stream) {
  CUtensorMap key_pages{};
  if (a.page_size != BLOCK_N / 4) return launch_with<D, PACKED, false>(key_pages, a, tiles, stream);
  // a row of the map is the block of a page and key/value head
  const uint64_t row = static_cast<uint64_t>(a.page_size) * D;
  const int rc = hx_tensor_map("hx_prefill_attention_tc", a.k_cache,
                               static_cast<uint64_t>(a.num_pages) * a.kv_heads, row, row, 1,
                               8 * a.page_size, false, &key_pages);
  if (rc != HX_OK) return rc;
  return launch_with<D, PACKED, true>(key_pages, a, tiles, stream);
}

}  // namespace

// 1 when the tcgen05 kernel takes this head size and page size: a page is the N operand of a
// product, so it has at least 16 keys.
HX_API int hx_prefill_attention_tc_supports(int head_dim, int page_size) {
  return head_dim >= 64 && head_dim <= 128 && head_dim % 16 == 0 &&
         (page_size == 16 || page_size == 32 || page_size == 64);
}

// The arguments of hx_prefill_attention; tile_bound bounds the number of 256-token query tiles
// (a larger bound only launches CTAs that leave at once).
// ... and with the optional per-head sinks and distance slopes (null: none), chunks (0: none)
// and a level the scores run into (0: none); see TcPrefillArgs.
HX_API int hx_prefill_attention_tc_biased(const void* q, int ldq, const void* k_cache,
                                          const void* v_cache, const int* request_start,
                                          const int* request_context,
                                          const int* request_table_row, const int* block_tables,
                                          int table_stride, void* out, int ldo, int requests,
                                          int tile_bound, int heads, int kv_heads, int head_dim,
                                          int page_size, int num_pages, float scale,
                                          int min_query_len, int window, int keep_first,
                                          const float* sinks, const float* slopes, int chunk,
                                          float softcap, int* status, cudaStream_t stream) {
  HX_REQUIRE(chunk >= 0 && softcap >= 0.0f, "hx_prefill_attention_tc: bad chunk or softcap");
  HX_REQUIRE(window >= 0 && keep_first >= 0, "hx_prefill_attention_tc: bad window");
  if (window == 0) keep_first = 0;
  HX_REQUIRE(hx_prefill_attention_tc_supports(head_dim, page_size),
             "hx_prefill_attention_tc: head_dim %d with pages of %d is not supported (head sizes "
             "64 to 128 in steps of 16, pages of 16, 32 or 64)", head_dim, page_size);
  HX_REQUIRE(requests >= 0 && tile_bound >= 0 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0,
             "hx_prefill_attention_tc: bad sizes");
  HX_REQUIRE(tile_bound <= 65535, "hx_prefill_attention_tc: too many query tiles");
  HX_REQUIRE(num_pages > 0 && table_stride > 0 &&
                 static_cast<long long>(num_pages) * kv_heads < (1ll << 31),
             "hx_prefill_attention_tc: bad cache geometry");
  HX_REQUIRE(status != nullptr, "hx_prefill_attention_tc: status word missing");
  HX_REQUIRE(ldq % 8 == 0 && ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(q) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(k_cache) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(v_cache) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(out) & 15) == 0,
             "hx_prefill_attention_tc: operands must be 16-byte aligned, row strides multiples of 8");
  if (requests == 0 || tile_bound == 0) return HX_OK;
  TcPrefillArgs a{static_cast<const __nv_bfloat16*>(q), ldq,
                  static_cast<const __nv_bfloat16*>(k_cache),
                  static_cast<const __nv_bfloat16*>(v_cache), request_start, request_context,
                  request_table_row, block_tables, table_stride, static_cast<__nv_bfloat16*>(out),
                  ldo, requests, heads, kv_heads, page_size, num_pages, scale, min_query_len, status,
                  window, keep_first, sinks, slopes, chunk, softcap, 1, head_dim};
  int rc;
  switch (head_dim) {
    case 64: rc = launch<64>(a, tile_bound, stream); break;
    case 80: rc = launch<80>(a, tile_bound, stream); break;
    case 96: rc = launch<96>(a, tile_bound, stream); break;
    case 112: rc = launch<112>(a, tile_bound, stream); break;
    default: rc = launch<128>(a, tile_bound, stream); break;
  }
  if (rc != HX_OK) return rc;
  HX_CHECK_LAUNCH("hx_prefill_attention_tc");
  return HX_OK;
}

HX_API int hx_prefill_attention_tc_windowed(const void* q, int ldq, const void* k_cache,
                                            const void* v_cache, const int* request_start,
                                            const int* request_context,
                                            const int* request_table_row, const int* block_tables,
                                            int table_stride, void* out, int ldo, int requests,
                                            int tile_bound, int heads, int kv_heads, int head_dim,
                                            int page_size, int num_pages, float scale,
                                            int min_query_len, int window, int keep_first,
                                            int* status, cudaStream_t stream) {
  return hx_prefill_attention_tc_biased(q, ldq, k_cache, v_cache, request_start, request_context,
                                        request_table_row, block_tables, table_stride, out, ldo,
                                        requests, tile_bound, heads, kv_heads, head_dim, page_size,
                                        num_pages, scale, min_query_len, window, keep_first,
                                        nullptr, nullptr, 0, 0.0f, status, stream);
}

// Every earlier key (no window).
HX_API int hx_prefill_attention_tc(const void* q, int ldq, const void* k_cache,
                                   const void* v_cache, const int* request_start,
                                   const int* request_context, const int* request_table_row,
                                   const int* block_tables, int table_stride, void* out, int ldo,
                                   int requests, int tile_bound, int heads, int kv_heads,
                                   int head_dim, int page_size, int num_pages, float scale,
                                   int min_query_len, int* status, cudaStream_t stream) {
  return hx_prefill_attention_tc_windowed(q, ldq, k_cache, v_cache, request_start,
                                          request_context, request_table_row, block_tables,
                                          table_stride, out, ldo, requests, tile_bound, heads,
                                          kv_heads, head_dim, page_size, num_pages, scale,
                                          min_query_len, 0, 0, status, stream);
}

// Tokens of a query tile of hx_prefill_attention_tc_packed; 0 where it does not apply.  It is for
// the heads that hx_prefill_attention_tc_supports leaves out (160 to 256 in steps of 32).
HX_API int hx_prefill_attention_tc_packed_tokens(int heads, int kv_heads, int head_dim, int page_size) {
  if (heads <= 0 || kv_heads <= 0 || heads % kv_heads != 0) return 0;
  // as many heads side by side as the mma.sync kernel takes
  if (heads / kv_heads < 2 || heads / kv_heads > BLOCK_M / 2) return 0;
  if (head_dim < 160 || head_dim > 256 || head_dim % 32 != 0) return 0;
  if (page_size != 16 && page_size != 32 && page_size != 64) return 0;
  return BLOCK_M / (heads / kv_heads);
}

// The arguments of hx_prefill_attention_tc_biased, for heads of 160 to 256 in steps of 32: a tile's
// 128 rows are the query heads of a key/value head, side by side, of
// hx_prefill_attention_tc_packed_tokens tokens; tile_bound bounds the number of such tiles.
// value_dim: the leading coordinates of the values that are wanted, a multiple of 32; the others of a row of
// `out` are not written.
HX_API int hx_prefill_attention_tc_packed_values(const void* q, int ldq, const void* k_cache,
                                          const void* v_cache, const int* request_start,
                                          const int* request_context,
                                          const int* request_table_row, const int* block_tables,
                                          int table_stride, void* out, int ldo, int requests,
                                          int tile_bound, int heads, int kv_heads, int head_dim,
                                          int page_size, int num_pages, float scale,
                                          int min_query_len, int window, int keep_first,
                                          const float* sinks, const float* slopes, int chunk,
                                          float softcap, int value_dim, int* status,
                                          cudaStream_t stream) {
  HX_REQUIRE(chunk >= 0 && softcap >= 0.0f, "hx_prefill_attention_tc_packed: bad chunk or softcap");
  HX_REQUIRE(window >= 0 && keep_first >= 0, "hx_prefill_attention_tc_packed: bad window");
  if (window == 0) keep_first = 0;
  HX_REQUIRE(hx_prefill_attention_tc_packed_tokens(heads, kv_heads, head_dim, page_size) > 0,
             "hx_prefill_attention_tc_packed: %d heads of %d on %d with pages of %d are not supported",
             heads, head_dim, kv_heads, page_size);
  HX_REQUIRE(requests >= 0 && tile_bound >= 0, "hx_prefill_attention_tc_packed: bad sizes");
  HX_REQUIRE(value_dim > 0 && value_dim <= head_dim && value_dim % 32 == 0,
             "hx_prefill_attention_tc_packed: %d of %d coordinates of the values", value_dim, head_dim);
  HX_REQUIRE(tile_bound <= 65535, "hx_prefill_attention_tc_packed: too many query tiles");
  HX_REQUIRE(num_pages > 0 && table_stride > 0 &&
                 static_cast<long long>(num_pages) * kv_heads < (1ll << 31),
             "hx_prefill_attention_tc_packed: bad cache geometry");
  HX_REQUIRE(status != nullptr, "hx_prefill_attention_tc_packed: status word missing");
  HX_REQUIRE(ldq % 8 == 0 && ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(q) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(k_cache) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(v_cache) & 15) == 0 &&
                 (reinterpret_cast<uintptr_t>(out) & 15) == 0,
             "hx_prefill_attention_tc_packed: operands must be 16-byte aligned, row strides multiples "
             "of 8");
  if (requests == 0 || tile_bound == 0) return HX_OK;
  TcPrefillArgs a{static_cast<const __nv_bfloat16*>(q), ldq,
                  static_cast<const __nv_bfloat16*>(k_cache),
                  static_cast<const __nv_bfloat16*>(v_cache), request_start, request_context,
                  request_table_row, block_tables, table_stride, static_cast<__nv_bfloat16*>(out),
                  ldo, requests, heads, kv_heads, page_size, num_pages, scale, min_query_len, status,
                  window, keep_first, sinks, slopes, chunk, softcap, heads / kv_heads, value_dim};
  int rc;
  switch (head_dim) {
    case 160: rc = launch<160, true>(a, tile_bound, stream); break;
    case 192: rc = launch<192, true>(a, tile_bound, stream); break;
    case 224: rc = launch<224, true>(a, tile_bound, stream); break;
    default: rc = launch<256, true>(a, tile_bound, stream); break;
  }
  if (rc != HX_OK) return rc;
  HX_CHECK_LAUNCH("hx_prefill_attention_tc_packed");
  return HX_OK;
}

// All of them.
HX_API int hx_prefill_attention_tc_packed(const void* q, int ldq, const void* k_cache,
                                          const void* v_cache, const int* request_start,
                                          const int* request_context,
                                          const int* request_table_row, const int* block_tables,
                                          int table_stride, void* out, int ldo, int requests,
                                          int tile_bound, int heads, int kv_heads, int head_dim,
                                          int page_size, int num_pages, float scale,
                                          int min_query_len, int window, int keep_first,
                                          const float* sinks, const float* slopes, int chunk,
                                          float softcap, int* status, cudaStream_t stream) {
  return hx_prefill_attention_tc_packed_values(q, ldq, k_cache, v_cache, request_start, request_context,
                                               request_table_row, block_tables, table_stride, out, ldo, requests,
                                               tile_bound, heads, kv_heads, head_dim, page_size, num_pages, scale,
                                               min_query_len, window, keep_first, sinks, slopes, chunk, softcap,
                                               head_dim, status, stream);
}
