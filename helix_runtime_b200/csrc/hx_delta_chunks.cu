// The gated delta rule in prompts, 64 tokens at a time on the tensor cores (bfloat16 rows):
//
//     S_t = e^(d_t) S_(t-1) + k_t u_t',   u_t = beta_t (v_t - e^(d_t) S_(t-1)' k_t),   o_t = S_t' q_t
//
// with queries and keys divided by their lengths (or scaled by constants).  Inside a chunk that
// starts from S_0, with L_t the sum of d up to t, the u_t solve a triangular system:
//
//     (1 + A) U = R,    A_ts = beta_t (k_t . k_s) e^(L_t - L_s)  (s < t),
//                       R_t  = beta_t v_t - beta_t e^(L_t) S_0' k_t
//     o_t  = e^(L_t) S_0' q_t + sum_(s <= t) P_ts u_s,   P_ts = (q_t . k_s) e^(L_t - L_s)
//     S_64 = e^(L_64) S_0 + sum_s e^(L_64 - L_s) k_s u_s'
//
// Every exponent is a difference of decays between two tokens of the chunk, never positive (decays
// of at most one).  A decay so small that float32 has only zero for it counts as e^-256, zero too,
// whose logarithm can be summed; a negative one has no logarithm and takes the road of numbers that
// are not finite (below).
//
//   * delta_weights_kernel, all chunks at once: T = (1 + A)^-1 by forward substitution in float32,
//     P, and the factors of a token.
//   * delta_states_kernel, one CTA per (request, head, 64 columns), chunk after chunk: two warps keep
//     S' for 16 columns in registers, half of the key coordinates each, as accumulators of mma.sync,
//     whose layout is also that of an A operand, so S' goes into S' K' and S' Q', R' into R' T', U'
//     into U' P' and U' K from registers.  A warpgroup copies the next chunk's rows meanwhile.
//
// Queries, keys and values go in as they are stored; what the scan holds in float32 (S, R, U, T,
// P) goes into the products as three bfloat16 terms, 24 bits; lengths and decays multiply the
// float32 sums.  The products of the small terms are summed before those of the large ones,
// which are then the only ones whose rounding counts.
//
// The weights of tokens that come later are zeros, and zero times a number that is not finite is
// none: such a number, wherever it comes in, shows in the chunk's outputs.  Warps that find one
// there take the chunk again token by token, from the state that they still hold.
//
// The scan walks a token in 0.6 us whatever the chip could do beside it (a chain of two dot
// products over the state); a chunk is a chain of about 800 products for 16 columns, in which the
// instructions between the products count as much.  Measured (one B200, 32 heads of 128 by 128, against the
// scan): a portion of 1,000 tokens 980 -> 142 us, eight of 256 1,064 -> 184, one of 128 134 -> 39; errors
// against 64 bits, 1,024 tokens, 1.8e-7 (outputs) and 1.3e-7 (state) where the scan has 2.3e-7 and 2.2e-7
// (2.6e-7 and 2.5e-7 with a chunk's products added onto the state itself).
#include "hx_mma.cuh"
#include "hx_scan.cuh"
#include "hx_tcgen05.cuh"

#include <mutex>

namespace {

constexpr int CHUNK = 64;
constexpr int ROW_PAD = 8;             // elements behind a staged row: rows start on different banks
constexpr int TERMS = 3;
constexpr int WEIGHT_COLUMNS = 2 * TERMS * CHUNK;      // a token's row of T, then of P, three terms each
constexpr int WEIGHT_STRIDE = WEIGHT_COLUMNS + ROW_PAD;
constexpr float NO_DECAY_LEFT = -256.0f;      // e^this is zero in float32 (from -104 on)

struct DeltaArgs {
  const __nv_bfloat16* q;    // [tokens, ld_q], already offset; qk_heads * dim columns
  const __nv_bfloat16* k;
  const __nv_bfloat16* v;    // heads * vdim columns
  int ld_q, ld_k, ld_v;
  const __nv_bfloat16* decay_in;      // as in LinearStateArgs
  const __nv_bfloat16* beta_in;
  int ld_gates;
  const float* a_log;
  const float* dt_bias;
  const float* fixed_decay_m1;
  int unit_norm;
  float unit_eps, q_scale, k_scale;
  __nv_bfloat16* weights;    // [heads, rows, WEIGHT_COLUMNS]
  float4* factors;           // [heads, rows]: of S' q, of S' k, of v, of u k'
  float* total;              // [heads, rows]: e^(L_64) at a chunk's first token
  int rows;
  float* state;
  long long state_stride;
  int head_stride;
  float* o;                  // [tokens, heads * vdim]
  const int* request_start;
  const int* request_slot;
  int requests, heads, qk_heads, dim, vdim, parts;
  int min_query_len;         // requests with fewer tokens are left alone;
  int portions;              // so many have as many
  int* status;               // may be null
  uint32_t polls;            // of a wait for copies, before it gives up
};

// two neighbouring values in three bfloat16 terms, a word each
__device__ __forceinline__ void split_terms(float x0, float x1, uint32_t& t0, uint32_t& t1,
                                            uint32_t& t2) {
  const __nv_bfloat162 high = __floats2bfloat162_rn(x0, x1);
  const float2 h = __bfloat1622float2(high);
  x0 -= h.x;
  x1 -= h.y;
  const __nv_bfloat162 middle = __floats2bfloat162_rn(x0, x1);
  const float2 m = __bfloat1622float2(middle);
  t0 = *reinterpret_cast<const uint32_t*>(&high);
  t1 = *reinterpret_cast<const uint32_t*>(&middle);
  t2 = hx_pack_bf16(x0 - m.x, x1 - m.y);
}

// The A operand of products over step `step`'s sixteen coordinates from two neighbouring
// accumulator tiles: all three terms, or the first one only (made anew, in volatile assembly:
// otherwise the compiler keeps the first terms of a whole pass over the state in registers that
// it does not have).
template <int TILES>
__device__ __forceinline__ void operand_terms(const float (&x)[TILES][4], int step, uint32_t (&t0)[4],
                                              uint32_t (&t1)[4], uint32_t (&t2)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int tile = 2 * step + (i >> 1), j = 2 * (i & 1);
    split_terms(x[tile][j], x[tile][j + 1], t0[i], t1[i], t2[i]);
  }
}
template <int TILES>
__device__ __forceinline__ void operand_high(const float (&x)[TILES][4], int step, uint32_t (&t0)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int tile = 2 * step + (i >> 1), j = 2 * (i & 1);
    asm volatile("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(t0[i]) : "f"(x[tile][j + 1]), "f"(x[tile][j]));
  }
}

// PIECES 16-byte pieces of each of 64 rows into shared memory (those in front of `columns`); rows
// from `live` on are zeros
template <int PIECES>
__device__ __forceinline__ void copy_rows(__nv_bfloat16* dst, int stride, const __nv_bfloat16* src,
                                          size_t ld, int columns, int live) {
  for (int i = threadIdx.x; i < CHUNK * PIECES; i += blockDim.x) {
    const int row = i / PIECES, piece = i - row * PIECES;
    const bool there = row < live;
    if (8 * piece < columns)
      hx_cp_async_16(hx_shared_address(dst + row * stride + 8 * piece),
                     there ? src + row * ld + 8 * piece : src, there ? 16 : 0);
  }
}

// zeros behind the copied columns, once: the copies never touch them
__device__ __forceinline__ void clear_columns(__nv_bfloat16* dst, int stride, int from, int to) {
  const int width = to - from;
  for (int i = threadIdx.x; i < CHUNK * width; i += blockDim.x) {
    const int row = i / width;
    dst[row * stride + from + i - row * width] = __float2bfloat16_rn(0.0f);
  }
}

constexpr int SOLVE_STRIDE = CHUNK + 4;

constexpr int TERMS_STRIDE = TERMS * CHUNK + ROW_PAD;      // of a token's row of T or P

// Shared memory of delta_weights_kernel: queries and keys (later the terms of P, then of T), A
// transposed, T.
__host__ __device__ constexpr int weights_rows(int padded) {
  return 2 * (padded + ROW_PAD) > TERMS_STRIDE ? 2 * (padded + ROW_PAD) : TERMS_STRIDE;
}
int weights_shared(int padded) {
  return 2 * CHUNK * weights_rows(padded) + 2 * 4 * CHUNK * SOLVE_STRIDE;
}

// grid (chunks of the step, heads), 128 threads: a warp takes 16 of the chunk's tokens
//
// Bound by chains of latency, three CTAs an SM to fill them.  Measured, 27 chunks of 32 heads: 44 -> 34 us with
// lengths a row a thread and P stored 16 bytes a thread beside the solution (of a CTA's 30,000 cycles 10,500
// solve, 4,200 find the chunk, 3,600 make the gates).
template <int STEPS>
__global__ __launch_bounds__(128) void delta_weights_kernel(const DeltaArgs a) {
  constexpr int PADDED = 16 * STEPS, STRIDE = PADDED + ROW_PAD;
  extern __shared__ uint4 shared_pieces[];
  __shared__ float level_hi[CHUNK], level_lo[CHUNK], q_length[CHUNK], k_length[CHUNK], write[CHUNK];
  hx_pdl_prologue();
  int chunk, chunks;
  const int request = hx_find_query_tile(a.request_start, a.requests, a.min_query_len, CHUNK, blockIdx.x, chunk, chunks);
  if (request < 0) return;
  const int head = blockIdx.y, qk_head = head / (a.heads / a.qk_heads);
  const int first = a.request_start[request] + chunk * CHUNK;
  const int live = min(CHUNK, a.request_start[request + 1] - first);
  __nv_bfloat16* queries = reinterpret_cast<__nv_bfloat16*>(shared_pieces);
  __nv_bfloat16* keys = queries + CHUNK * STRIDE;
  float* system = reinterpret_cast<float*>(queries + CHUNK * weights_rows(PADDED));      // [s][t]: A
  float* solution = system + CHUNK * SOLVE_STRIDE;                      // [t][s]: T
  copy_rows<2 * STEPS>(queries, STRIDE, a.q + static_cast<size_t>(first) * a.ld_q + qk_head * a.dim, a.ld_q, a.dim, live);
  copy_rows<2 * STEPS>(keys, STRIDE, a.k + static_cast<size_t>(first) * a.ld_k + qk_head * a.dim, a.ld_k, a.dim, live);
  hx_cp_async_commit();
  if (PADDED > a.dim) {
    clear_columns(queries, STRIDE, a.dim, PADDED);
    clear_columns(keys, STRIDE, a.dim, PADDED);
  }
  const size_t rows = static_cast<size_t>(head) * a.rows + first;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // One warp makes what the gates make of the tokens while the others take the lengths and go on to their
  // products (that warp's are the fewest).
  hx_cp_async_wait<0>();
  if (warp == 0) {
    asm volatile("bar.arrive 1, 128;" ::: "memory");
    // sums of the decays' logarithms, two neighbouring tokens a lane, in double: their
    // differences are what counts
    float d[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = 2 * lane + i;
      d[i] = 0.0f;
      float beta = 0.0f;
      if (t < live) {
        const size_t gate = static_cast<size_t>(first + t) * a.ld_gates + head;
        d[i] = a.decay_in != nullptr
                   ? -expf(a.a_log[head]) * softplus(__bfloat162float(a.decay_in[gate]) + a.dt_bias[head])
                   : log1pf(a.fixed_decay_m1[head]);
        if (d[i] < NO_DECAY_LEFT) d[i] = NO_DECAY_LEFT;      // (a NaN stays one)
        beta = hx_sigmoid(__bfloat162float(a.beta_in[gate]));
      }
      write[t] = beta;
    }
    double sum = static_cast<double>(d[0]) + static_cast<double>(d[1]);
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1) {
      const double other = __shfl_up_sync(0xffffffffu, sum, offset);
      if (lane >= offset) sum += other;
    }
    const double before = sum - static_cast<double>(d[1]);
    level_hi[2 * lane] = static_cast<float>(before);
    level_lo[2 * lane] = static_cast<float>(before - static_cast<double>(static_cast<float>(before)));
    level_hi[2 * lane + 1] = static_cast<float>(sum);
    level_lo[2 * lane + 1] = static_cast<float>(sum - static_cast<double>(static_cast<float>(sum)));
    asm volatile("bar.sync 2, 128;" ::: "memory");
  } else {
    asm volatile("bar.sync 1, 128;" ::: "memory");
    // what lengths and scales make of a query and a key, a row a thread (neighbours' 16-byte pieces lie on
    // different banks); one warp for 16 rows took 12,000 cycles of the kernel's 40,000
    for (int i = threadIdx.x - 32; i < 2 * CHUNK; i += 96) {
      const bool key = i >= CHUNK;
      const int t = i & (CHUNK - 1);
      float length = key ? a.k_scale : a.q_scale;
      if (a.unit_norm) {
        const __nv_bfloat16* x = (key ? keys : queries) + t * STRIDE;
        float squares[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) squares[j] = 0.0f;
#pragma unroll
        for (int e = 0; e < PADDED; e += 8) {
          const uint4 piece = *reinterpret_cast<const uint4*>(x + e);
          const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&piece);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 v = __bfloat1622float2(pairs[j]);
            float* sum = squares + (e & 8) + 2 * j;
            sum[0] = fmaf(v.x, v.x, sum[0]);
            sum[1] = fmaf(v.y, v.y, sum[1]);
          }
        }
#pragma unroll
        for (int offset = 8; offset > 0; offset >>= 1)
#pragma unroll
          for (int j = 0; j < offset; ++j) squares[j] += squares[j + offset];
        length /= sqrtf(squares[0] + a.unit_eps);
      }
      (key ? k_length : q_length)[t] = length;
    }
    asm volatile("bar.arrive 2, 128;" ::: "memory");
  }
  // sums of tokens 16 warp .. + 15 against the tiles of 8 tokens that do not lie behind them
  float qk[8][4], kk[8][4];
#pragma unroll
  for (int n = 0; n < 8; ++n)
#pragma unroll
    for (int j = 0; j < 4; ++j) qk[n][j] = kk[n][j] = 0.0f;
  const int tiles = 2 * warp + 2;
  const int matrix = lane >> 3, in_matrix = lane & 7;
  const uint32_t a_row = 2 * ((16 * warp + (matrix & 1) * 8 + in_matrix) * STRIDE + (matrix >> 1) * 8);
  const uint32_t q_at = hx_shared_address(queries) + a_row, k_at = hx_shared_address(keys) + a_row;
  const uint32_t b_at = hx_shared_address(keys + ((matrix >> 1) * 8 + in_matrix) * STRIDE + (matrix & 1) * 8);
#pragma unroll
  for (int step = 0; step < STEPS; ++step) {
    uint32_t qf[4], kf[4];
    hx_ldmatrix_x4(qf, q_at + 32 * step);
    hx_ldmatrix_x4(kf, k_at + 32 * step);
#pragma unroll
    for (int n = 0; n < 8; n += 2) {
      if (n < tiles) {
        uint32_t b[4];
        hx_ldmatrix_x4(b, b_at + 2 * (8 * n * STRIDE + 16 * step));
        hx_mma_bf16(qk[n], qf, b[0], b[1]);
        hx_mma_bf16(qk[n + 1], qf, b[2], b[3]);
        hx_mma_bf16(kk[n], kf, b[0], b[1]);
        hx_mma_bf16(kk[n + 1], kf, b[2], b[3]);
      }
    }
  }
  __syncthreads();      // (queries and keys are read, too: the terms of T and P gather in their place)
  // e^(L_t - L_s)
  auto faded = [&](int t, int s) {
    return expf((level_hi[t] - level_hi[s]) + (level_lo[t] - level_lo[s]));
  };
  if (threadIdx.x < live) {
    const int t = threadIdx.x;
    const float level = expf(level_hi[t] + level_lo[t]);
    a.factors[rows + t] = make_float4(q_length[t] * level, write[t] * k_length[t] * level, write[t],
                                      k_length[t] * faded(CHUNK - 1, t));
    if (t == 0) a.total[rows] = expf(level_hi[CHUNK - 1] + level_lo[CHUNK - 1]);
  }
  const int row = lane >> 2, column = 2 * (lane & 3);
  __nv_bfloat16* terms = queries;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const int t = 16 * warp + row + 8 * half;
    __nv_bfloat16* out = terms + t * TERMS_STRIDE;
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int s = 8 * n + column;
      float p[2] = {0.0f, 0.0f};
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float held = 0.0f;
        if (s + i <= t) {
          const float fade = faded(t, s + i) * k_length[s + i];
          p[i] = qk[n][2 * half + i] * (q_length[t] * fade);
          if (s + i < t) held = kk[n][2 * half + i] * (write[t] * k_length[t] * fade);
        }
        system[(s + i) * SOLVE_STRIDE + t] = held;
      }
      uint32_t t0, t1, t2;
      split_terms(p[0], p[1], t0, t1, t2);
      *reinterpret_cast<uint32_t*>(out + s) = t0;
      *reinterpret_cast<uint32_t*>(out + CHUNK + s) = t1;
      *reinterpret_cast<uint32_t*>(out + 2 * CHUNK + s) = t2;
    }
  }
  __syncthreads();
  if (threadIdx.x < CHUNK) {
    // a column of T a thread, sixteen rows at a time: what the rows in front of them leave, then
    // the rows among themselves
    const int j = threadIdx.x;
#pragma unroll 1
    for (int block = 0; block < CHUNK / 16; ++block) {
      float x[16];
#pragma unroll
      for (int r = 0; r < 16; ++r) x[r] = 16 * block + r == j ? 1.0f : 0.0f;
      if (16 * (block + 1) > (warp << 5)) {      // else all the warp's columns are zero here
#pragma unroll 4
        for (int s = warp << 5; s < 16 * block; ++s) {
          const float known = solution[s * SOLVE_STRIDE + j];
          const float4* held = reinterpret_cast<const float4*>(system + s * SOLVE_STRIDE + 16 * block);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const float4 h = held[r];
            x[4 * r] = fmaf(-h.x, known, x[4 * r]);
            x[4 * r + 1] = fmaf(-h.y, known, x[4 * r + 1]);
            x[4 * r + 2] = fmaf(-h.z, known, x[4 * r + 2]);
            x[4 * r + 3] = fmaf(-h.w, known, x[4 * r + 3]);
          }
        }
#pragma unroll
        for (int s = 0; s < 15; ++s) {
          const float4* held = reinterpret_cast<const float4*>(system + (16 * block + s) * SOLVE_STRIDE + 16 * block);
#pragma unroll
          for (int r = (s + 1) / 4; r < 4; ++r) {
            const float4 h = held[r];
            if (4 * r > s) x[4 * r] = fmaf(-h.x, x[s], x[4 * r]);
            if (4 * r + 1 > s) x[4 * r + 1] = fmaf(-h.y, x[s], x[4 * r + 1]);
            if (4 * r + 2 > s) x[4 * r + 2] = fmaf(-h.z, x[s], x[4 * r + 2]);
            if (4 * r + 3 > s) x[4 * r + 3] = fmaf(-h.w, x[s], x[4 * r + 3]);
          }
        }
      }
#pragma unroll
      for (int r = 0; r < 16; ++r) solution[(16 * block + r) * SOLVE_STRIDE + j] = x[r];
    }
  }
  // The warps that do not solve store P meanwhile: whole 16-byte pieces, a row's one behind the other.
  auto store = [&](int thread, int threads, int column) {
    constexpr int PIECES = TERMS * CHUNK / 8;
    for (int i = thread; i < live * PIECES; i += threads) {
      const int t = i / PIECES, piece = i - t * PIECES;
      *reinterpret_cast<uint4*>(a.weights + (rows + t) * WEIGHT_COLUMNS + column + 8 * piece) =
          *reinterpret_cast<const uint4*>(terms + t * TERMS_STRIDE + 8 * piece);
    }
  };
  if (threadIdx.x >= CHUNK) store(threadIdx.x - CHUNK, CHUNK, TERMS * CHUNK);
  __syncthreads();
  for (int i = threadIdx.x; i < CHUNK * (CHUNK / 2); i += 128) {
    const int t = i / (CHUNK / 2), s = 2 * (i - t * (CHUNK / 2));
    const float2 x = *reinterpret_cast<const float2*>(solution + t * SOLVE_STRIDE + s);
    __nv_bfloat16* out = terms + t * TERMS_STRIDE + s;
    uint32_t t0, t1, t2;
    split_terms(x.x, x.y, t0, t1, t2);
    *reinterpret_cast<uint32_t*>(out) = t0;
    *reinterpret_cast<uint32_t*>(out + CHUNK) = t1;
    *reinterpret_cast<uint32_t*>(out + 2 * CHUNK) = t2;
  }
  __syncthreads();
  store(threadIdx.x, 128, 0);
}

// Shared memory of delta_states_kernel: two stages of [queries | keys | weights | values | factors], then
// what the two warps of a block of 16 columns tell each other: two buffers of 32 numbers a lane, and a
// word; then a barrier for each stage.
constexpr int EXCHANGED = 32;
constexpr int BLOCKS = 4, BLOCK_COLUMNS = 16 * BLOCKS;      // of a CTA: a block of 16 columns for each quarter of an SM
constexpr int STATES_THREADS = 3 * 32 * BLOCKS;             // two warps a block, and a warpgroup that copies
// At launch 168 a thread; the warps that copy need few, the others take what they leave.
constexpr int WORK_REGISTERS = 224, COPY_REGISTERS = 56;
static_assert(2 * WORK_REGISTERS + COPY_REGISTERS <= 3 * 168, "what one side takes the other has given back");
template <int PADDED>
struct DeltaLayout {
  static constexpr int kValueStride = BLOCK_COLUMNS + ROW_PAD;
  static constexpr int kRowsBytes = 2 * CHUNK * (2 * (PADDED + ROW_PAD) + WEIGHT_STRIDE + kValueStride);
  static constexpr int kStageBytes = kRowsBytes + 16 * CHUNK;
  static constexpr int kExchange = 2 * kStageBytes;
  static constexpr int kOdd = kExchange + BLOCKS * 2 * EXCHANGED * 32 * 4;
  static constexpr int kBars = kOdd + BLOCKS * 16;
  static constexpr int kBytes = kBars + 16;
};

// A row into shared memory, counted on a barrier; both ends and the size are multiples of 16 bytes.
__device__ __forceinline__ void copy_row(void* dst, const void* src, int bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   hx_shared_address(dst)),
               "l"(src), "r"(bytes), "r"(hx_shared_address(bar))
               : "memory");
}

// sums = x' w', with x' [16 columns x 64 tokens s] in accumulators and w [t][s] of three terms in
// rows of the staged weights; w_ts is zero for t < s.  Six products carry 24 bits.
__device__ __forceinline__ void triangular_product(float (&sums)[8][4], const float (&x)[8][4],
                                                   uint32_t weights_at) {
#pragma unroll
  for (int n = 0; n < 8; ++n)
#pragma unroll
    for (int j = 0; j < 4; ++j) sums[n][j] = 0.0f;
#pragma unroll
  for (int step = 0; step < CHUNK / 16; ++step) {
    uint32_t x0[4], x1[4], x2[4];
    operand_terms(x, step, x0, x1, x2);
    // up to four tiles of tokens side by side: a sum's products follow one another
#pragma unroll
    for (int n0 = 2 * step; n0 < 8; n0 += 4) {
      uint32_t w0[2][4], w1[2][4], w2[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (n0 + 2 * i >= 8) continue;
        const uint32_t at = weights_at + 2 * (8 * (n0 + 2 * i) * WEIGHT_STRIDE + 16 * step);
        hx_ldmatrix_x4(w0[i], at);
        hx_ldmatrix_x4(w2[i], at + 4 * CHUNK);
        hx_ldmatrix_x4(w1[i], at + 2 * CHUNK);
      }
      auto products = [&](const uint32_t (&xt)[4], const uint32_t (&wt)[2][4]) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int n = n0 + 2 * i;
          if (n >= 8) continue;
          hx_mma_bf16(sums[n], xt, wt[i][0], wt[i][1]);
          hx_mma_bf16(sums[n + 1], xt, wt[i][2], wt[i][3]);
        }
      };
      products(x2, w0);
      products(x0, w2);
      products(x1, w1);
      products(x1, w0);
      products(x0, w1);
    }
  }
#pragma unroll
  for (int step = 0; step < CHUNK / 16; ++step) {
    uint32_t x0[4], w0[4][4];
#pragma unroll
    for (int i = step; i < 4; ++i) hx_ldmatrix_x4(w0[i], weights_at + 2 * (16 * i * WEIGHT_STRIDE + 16 * step));
    operand_high(x, step, x0);
#pragma unroll
    for (int i = step; i < 4; ++i) {
      hx_mma_bf16(sums[2 * i], x0, w0[i][0], w0[i][1]);
      hx_mma_bf16(sums[2 * i + 1], x0, w0[i][2], w0[i][3]);
    }
  }
}

// The chunk's tokens one after the other, as the recurrence is written, for chunks with numbers that
// are not finite.  S, queries, keys, values: as delta_states_kernel holds them; `first`: the chunk's
// first token, `column`: the first of the lane's two columns (8 apart).  (Not inlined: its caller
// has no register to spare.)
template <int TILES>
__device__ __noinline__ void tokens_in_turn(const DeltaArgs& a, float (*S)[4], const __nv_bfloat16* queries,
                                            const __nv_bfloat16* keys, int stride,
                                            const __nv_bfloat16* values, int value_stride, int first,
                                            int live, int head, int column) {
  const int pair = 2 * (threadIdx.x & 3);
  const float rate = a.decay_in != nullptr ? expf(a.a_log[head]) : 0.0f;
  // over the four lanes that share the columns
  auto summed = [](float x) {
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    return x + __shfl_xor_sync(0xffffffffu, x, 2);
  };
#pragma unroll 1
  for (int t = 0; t < live; ++t) {
    const size_t gate = static_cast<size_t>(first + t) * a.ld_gates + head;
    const float decay = a.decay_in != nullptr
                            ? expf(-rate * softplus(__bfloat162float(a.decay_in[gate]) + a.dt_bias[head]))
                            : 1.0f + a.fixed_decay_m1[head];
    const float beta = hx_sigmoid(__bfloat162float(a.beta_in[gate]));
    const __nv_bfloat16* q = queries + t * stride + pair;
    const __nv_bfloat16* k = keys + t * stride + pair;
    float fq = a.q_scale, fk = a.k_scale;
    if (a.unit_norm) {
      float sq = 0.0f, sk = 0.0f;
#pragma unroll
      for (int n = 0; n < TILES; ++n) {
        const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(q + 8 * n));
        const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(k + 8 * n));
        sq = fmaf(x.x, x.x, fmaf(x.y, x.y, sq));
        sk = fmaf(y.x, y.x, fmaf(y.y, y.y, sk));
      }
      fq /= sqrtf(summed(sq) + a.unit_eps);
      fk /= sqrtf(summed(sk) + a.unit_eps);
    }
    float u[2], o[2] = {0.0f, 0.0f};
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      float held = 0.0f;
#pragma unroll
      for (int n = 0; n < TILES; ++n) {
        const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(k + 8 * n));
        held = fmaf(S[n][2 * c], fk * y.x, fmaf(S[n][2 * c + 1], fk * y.y, held));
      }
      u[c] = beta * (__bfloat162float(values[t * value_stride + 8 * c]) - decay * summed(held));
    }
#pragma unroll
    for (int n = 0; n < TILES; ++n) {
      if (8 * n < a.dim) {      // (the dimension is a multiple of 8; what lies behind it stays zero)
        const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(q + 8 * n));
        const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(k + 8 * n));
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          S[n][2 * c] = fmaf(decay, S[n][2 * c], fk * y.x * u[c]);
          S[n][2 * c + 1] = fmaf(decay, S[n][2 * c + 1], fk * y.y * u[c]);
          o[c] = fmaf(S[n][2 * c], fq * x.x, fmaf(S[n][2 * c + 1], fq * x.y, o[c]));
        }
      }
    }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const float sum = summed(o[c]);
      if (pair == 0 && column + 8 * c < a.vdim)
        a.o[static_cast<size_t>(first + t) * (a.heads * a.vdim) + head * a.vdim + column + 8 * c] = sum;
    }
  }
}

// sums = S' x' over HALF steps of 16 key coordinates for all tokens of the chunk, [16 columns x 64
// tokens]; x: staged rows of keys or queries.  The rows that half a step takes are asked for while the
// products of the half before run.
template <int HALF>
__device__ __forceinline__ void state_product(float (&sums)[8][4], const float (&S)[2 * HALF][4], uint32_t rows_at,
                                              int stride) {
#pragma unroll
  for (int n = 0; n < 8; ++n)
#pragma unroll
    for (int j = 0; j < 4; ++j) sums[n][j] = 0.0f;
  uint32_t x[2][2][4];
  auto fetch = [&](int half) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
      hx_ldmatrix_x4(x[half & 1][i], rows_at + 2 * (8 * (4 * (half & 1) + 2 * i) * stride + 16 * (half >> 1)));
  };
  auto products = [&](int half, const uint32_t (&st)[4]) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int n = 4 * (half & 1) + 2 * i;
      hx_mma_bf16(sums[n], st, x[half & 1][i][0], x[half & 1][i][1]);
      hx_mma_bf16(sums[n + 1], st, x[half & 1][i][2], x[half & 1][i][3]);
    }
  };
  fetch(0);
#pragma unroll
  for (int step = 0; step < HALF; ++step) {
    uint32_t s0[4], s1[4], s2[4];
    operand_terms(S, step, s0, s1, s2);
#pragma unroll
    for (int half = 2 * step; half < 2 * step + 2; ++half) {
      fetch((half + 1) % (2 * HALF));
      products(half, s2);
      products(half, s1);
    }
  }
#pragma unroll
  for (int step = 0; step < HALF; ++step) {
    uint32_t s0[4];
    operand_high(S, step, s0);
#pragma unroll
    for (int half = 2 * step; half < 2 * step + 2; ++half) {
      if (half + 1 < 2 * HALF) fetch(half + 1);
      products(half, s0);
    }
  }
}

// grid (portions, heads, blocks of columns); two warps keep 16 columns, each one half of the key
// coordinates.  STEPS: steps of 16 key coordinates
//
// What bounds a chunk is a chain of warp-wide products and of the instructions between them, so the work of
// 16 columns is dealt to two warps of the same quarter of an SM, which fill each other's gaps: either
// multiplies its half of S' and carries it on; the first makes R and U, the second the outputs meanwhile:
//
//     first:   S' k | + the other's | R, U = T R | S' q (its half)  | state
//     second:  S' k |  S' q (its half)           | P U, + the first's S' q, outputs | state
//
// A third warpgroup copies (a row a bulk copy), because issuing them takes as long as a third of the chunk's
// products.  Cycles a chunk of 11,800: S' k 2,600, R 750, U 1,900, S' q beside P U 2,300, terms 1,100, outputs and
// state 2,600; the tensor pipe has 6,500 of work.  Measured, portions of 763 and 957 tokens, 32 heads of 128 by
// 128: 156 -> 101 us.  (One warp for 16 columns, 19,000 cycles a chunk; its products in another order, four to
// eight sums side by side, 156; two warps and their copies as cp.async 130, as bulk copies of the same warps 119.)
template <int STEPS>
__global__ __launch_bounds__(STATES_THREADS, 1) void delta_states_kernel(const __grid_constant__ DeltaArgs a) {
  constexpr int PADDED = 16 * STEPS, STRIDE = PADDED + ROW_PAD, HALF = STEPS / 2;
  static_assert(8 * HALF <= EXCHANGED, "a half of the state passes through a buffer");
  extern __shared__ uint4 shared_pieces[];
  hx_pdl_prologue();
  const int head = blockIdx.y, qk_head = head / (a.heads / a.qk_heads);
  int request = blockIdx.x;
  if (a.portions < a.requests) {
    int only, of_one;      // a portion is one tile of as many tokens as there can be
    request = hx_find_query_tile(a.request_start, a.requests, a.min_query_len, 1 << 30, blockIdx.x, only, of_one);
    if (request < 0) return;
  }
  const int start = a.request_start[request];
  const int count = a.request_start[request + 1] - start;
  if (count < a.min_query_len) return;
  const int lane = threadIdx.x & 31;
  const int block = (threadIdx.x >> 5) % BLOCKS;      // of 16 columns
  const bool second = (threadIdx.x >> 5) >= BLOCKS;
  const int row = lane >> 2, pair = 2 * (lane & 3);
  const int matrix = lane >> 3, in_matrix = lane & 7;
  const int column0 = blockIdx.z * BLOCK_COLUMNS;
  const int copied = min(a.vdim - column0, BLOCK_COLUMNS);
  using Layout = DeltaLayout<PADDED>;
  constexpr int value_stride = Layout::kValueStride;
  char* base = reinterpret_cast<char*>(shared_pieces);
  auto queries_of = [&](int stage) { return reinterpret_cast<__nv_bfloat16*>(base + stage * Layout::kStageBytes); };
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + Layout::kBars);
  // A chunk's rows, a copy each (of queries, keys, weights, values); rows behind the portion are zeros.
  auto fetch = [&](int chunk, int stage) {
    const size_t first = start + chunk * CHUNK;
    const int live = min(CHUNK, count - chunk * CHUNK);
    const size_t rows = static_cast<size_t>(head) * a.rows + first;
    __nv_bfloat16* queries = queries_of(stage);
    __nv_bfloat16* keys = queries + CHUNK * STRIDE;
    __nv_bfloat16* weights = keys + CHUNK * STRIDE;
    __nv_bfloat16* values = weights + CHUNK * WEIGHT_STRIDE;
    char* factors = base + stage * Layout::kStageBytes + Layout::kRowsBytes;
    uint64_t* bar = bars + stage;
    const int thread = threadIdx.x - 2 * 32 * BLOCKS;
    if (thread == 0) {
      mbar_expect_tx(bar, 2 * live * (2 * a.dim + WEIGHT_COLUMNS + copied) + 16 * live);
      copy_row(factors, a.factors + rows, 16 * live, bar);
    }
    for (int i = thread; i < 4 * CHUNK; i += 32 * BLOCKS) {
      const int what = i / CHUNK, t = i % CHUNK;
      __nv_bfloat16* to;
      const __nv_bfloat16* from;
      int size;
      if (what == 0) {
        to = queries + t * STRIDE, from = a.q + (first + t) * a.ld_q + qk_head * a.dim, size = a.dim;
      } else if (what == 1) {
        to = keys + t * STRIDE, from = a.k + (first + t) * a.ld_k + qk_head * a.dim, size = a.dim;
      } else if (what == 2) {
        to = weights + t * WEIGHT_STRIDE, from = a.weights + (rows + t) * WEIGHT_COLUMNS, size = WEIGHT_COLUMNS;
      } else {
        to = values + t * value_stride, from = a.v + (first + t) * a.ld_v + head * a.vdim + column0, size = copied;
      }
      if (t < live) {
        copy_row(to, from, 2 * size, bar);
      } else {
        for (int e = 0; e < size; e += 8) *reinterpret_cast<uint4*>(to + e) = make_uint4(0u, 0u, 0u, 0u);
        if (what == 3) *reinterpret_cast<float4*>(factors + 16 * t) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
    }
  };
  if (threadIdx.x == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  // what the copies leave alone
  for (int stage = 0; stage < 2; ++stage) {
    __nv_bfloat16* queries = queries_of(stage);
    if (PADDED > a.dim) {
      clear_columns(queries, STRIDE, a.dim, PADDED);
      clear_columns(queries + CHUNK * STRIDE, STRIDE, a.dim, PADDED);
    }
    if (copied < BLOCK_COLUMNS)
      clear_columns(queries + CHUNK * (2 * STRIDE + WEIGHT_STRIDE), value_stride, copied, BLOCK_COLUMNS);
  }
  const int chunks = (count + CHUNK - 1) / CHUNK;
  // Whether the chunk's rows are there; behind it nobody reads the other stage any more.
  auto arrived = [&](int chunk) {
    const bool there = mbar_wait(&bars[chunk & 1], (chunk >> 1) & 1u, a.polls);
    return __syncthreads_or(!there) == 0;
  };
  if (threadIdx.x >= 2 * 32 * BLOCKS) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(COPY_REGISTERS));
    fetch(0, 0);
    for (int chunk = 0; chunk < chunks; ++chunk) {
      if (!arrived(chunk)) {
        // what was asked for lands in memory that the CTA is about to give back
        mbar_wait(&bars[chunk & 1], (chunk >> 1) & 1u);
        return;
      }
      if (chunk + 1 < chunks) fetch(chunk + 1, (chunk + 1) & 1);
    }
    return;
  }
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(WORK_REGISTERS));

  // what the two warps tell each other, a lane's numbers 32 floats apart
  float* told = reinterpret_cast<float*>(base + Layout::kExchange) + block * (2 * EXCHANGED * 32) + lane;
  float* told_too = told + EXCHANGED * 32;
  int* any_odd = reinterpret_cast<int*>(base + Layout::kOdd) + 4 * block;
  auto meet = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(block + 1) : "memory"); };
  auto tell = [&](float* to, const float (&x)[8][4]) {
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int j = 0; j < 4; ++j) to[32 * (4 * n + j)] = x[n][j];
  };

  // the warp's part of S': columns my_column (+ 8), key coordinates 8 n + pair (+ 1) of its half
  float* s_state = a.state + static_cast<size_t>(a.request_slot[request]) * a.state_stride +
                   static_cast<size_t>(head) * a.head_stride;
  const int lanes = a.vdim * a.parts;
  const int my_column = column0 + 16 * block + row;
  const int half_column = second ? 16 * HALF : 0;
  float S[2 * HALF][4];
#pragma unroll
  for (int n = 0; n < 2 * HALF; ++n)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = my_column + 8 * (j >> 1), d = half_column + 8 * n + pair + (j & 1);
      S[n][j] = c < a.vdim && d < a.dim
                    ? s_state[static_cast<size_t>(d & 15) * lanes + c * a.parts + (d >> 4)] : 0.0f;
    }
  // offsets of the lane's rows in the operands
  const uint32_t row_lane = 2 * (((matrix >> 1) * 8 + in_matrix) * STRIDE + (matrix & 1) * 8 + half_column);
  const uint32_t key_lane = 2 * (((matrix & 1) * 8 + in_matrix) * STRIDE + (matrix >> 1) * 8 + half_column);
  const uint32_t weight_lane = 2 * (((matrix >> 1) * 8 + in_matrix) * WEIGHT_STRIDE + (matrix & 1) * 8);
  const uint32_t value_lane = 2 * (((matrix >> 1) * 8 + in_matrix) * value_stride + 16 * block + (matrix & 1) * 8);
  for (int chunk = 0; chunk < chunks; ++chunk) {
    const int stage = chunk & 1;
    if (!arrived(chunk)) {
      if (threadIdx.x == 0 && a.status != nullptr) atomicOr(a.status, HX_FLAG_WAIT_TIMEOUT);
      for (int t = chunk * CHUNK + pair / 2; second && t < count; t += 4)
        for (int c = my_column; c < min(a.vdim, my_column + 16); c += 8)
          a.o[static_cast<size_t>(start + t) * (a.heads * a.vdim) + head * a.vdim + c] = __int_as_float(0x7fc00000);
      return;
    }
    const float total = a.total[static_cast<size_t>(head) * a.rows + start + chunk * CHUNK];
    const uint32_t queries = hx_shared_address(queries_of(stage));
    const uint32_t keys = queries + 2 * CHUNK * STRIDE;
    const uint32_t weights = keys + 2 * CHUNK * STRIDE;
    const uint32_t values = weights + 2 * CHUNK * WEIGHT_STRIDE;
    const float4* factors = reinterpret_cast<const float4*>(base + stage * Layout::kStageBytes + Layout::kRowsBytes);
    const int first = start + chunk * CHUNK, live = min(CHUNK, count - chunk * CHUNK);

    // S_0' k of all tokens, [16 columns x 64 tokens], over the warp's coordinates
    float u[8][4];
    {
      float rest[8][4];
      state_product<HALF>(rest, S, keys + row_lane, STRIDE);
      if (second) tell(told, rest);
      meet();
      if (!second) {
        // R: what the values leave to be written
#pragma unroll
        for (int step = 0; step < CHUNK / 16; ++step) {
          uint32_t v[4];      // in the order of two neighbouring accumulator tiles
          hx_ldmatrix_x4_trans(v, values + value_lane + 2 * (16 * step * value_stride));
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int n = 2 * step + i;
            const float4 f0 = factors[8 * n + pair], f1 = factors[8 * n + pair + 1];
#pragma unroll
            for (int j = 0; j < 4; ++j) rest[n][j] += told[32 * (4 * n + j)];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v[2 * i + half]));
              rest[n][2 * half] = fmaf(f0.z, x.x, -f0.y * rest[n][2 * half]);
              rest[n][2 * half + 1] = fmaf(f1.z, x.y, -f1.y * rest[n][2 * half + 1]);
            }
          }
        }
        triangular_product(u, rest, weights + weight_lane);
        tell(told, u);
        meet();
        state_product<HALF>(rest, S, queries + row_lane, STRIDE);
        tell(told_too, rest);
        meet();
      }
    }
    float out[8][4];
    bool odd_here = false;
    if (second) {
      state_product<HALF>(out, S, queries + row_lane, STRIDE);
      meet();
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) u[n][j] = told[32 * (4 * n + j)];
      float written[8][4];
      triangular_product(written, u, weights + weight_lane + 2 * TERMS * CHUNK);
      meet();
      float odd = 0.0f;      // NaN with any number that is not finite (zero times it is)
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        const float by[2] = {factors[8 * n + pair].x, factors[8 * n + pair + 1].x};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          out[n][j] = fmaf(out[n][j] + told_too[32 * (4 * n + j)], by[j & 1], written[n][j]);
          odd = fmaf(out[n][j], 0.0f, odd);
        }
      }
      odd_here = odd != 0.0f;
    }
    // what the chunk adds to the state, in terms
    float odd = 0.0f;
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        u[n][j] *= factors[8 * n + pair + (j & 1)].w;
        odd = fmaf(u[n][j], 0.0f, odd);
      }
    if (second) {
      odd_here = __any_sync(0xffffffffu, odd_here || odd != 0.0f);
      if (lane == 0) *any_odd = odd_here ? 1 : 0;
    }
    uint32_t u0[CHUNK / 16][4], u1[CHUNK / 16][4], u2[CHUNK / 16][4];
#pragma unroll
    for (int step = 0; step < CHUNK / 16; ++step) operand_terms(u, step, u0[step], u1[step], u2[step]);
    meet();
    if (*any_odd != 0) {
      // the first warp goes through the tokens with all of S'
      if (second) {
#pragma unroll
        for (int n = 0; n < 2 * HALF; ++n)
#pragma unroll
          for (int j = 0; j < 4; ++j) told[32 * (4 * n + j)] = S[n][j];
      }
      meet();
      if (!second) {
        const __nv_bfloat16* staged = queries_of(stage);
        float held[2 * STEPS][4];
#pragma unroll
        for (int n = 0; n < 2 * HALF; ++n)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            held[n][j] = S[n][j];
            held[2 * HALF + n][j] = told[32 * (4 * n + j)];
          }
        tokens_in_turn<2 * STEPS>(a, held, staged, staged + CHUNK * STRIDE, STRIDE,
                                  staged + CHUNK * (2 * STRIDE + WEIGHT_STRIDE) + 16 * block + row, value_stride,
                                  first, live, head, my_column);
#pragma unroll
        for (int n = 0; n < 2 * HALF; ++n)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            S[n][j] = held[n][j];
            told[32 * (4 * n + j)] = held[2 * HALF + n][j];
          }
      }
      meet();
      if (second) {
#pragma unroll
        for (int n = 0; n < 2 * HALF; ++n)
#pragma unroll
          for (int j = 0; j < 4; ++j) S[n][j] = told[32 * (4 * n + j)];
      }
      continue;
    }
    if (second) {
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int t = 8 * n + pair + (j & 1), c = my_column + 8 * (j >> 1);
          if (t < live && c < a.vdim)
            a.o[static_cast<size_t>(first + t) * (a.heads * a.vdim) + head * a.vdim + c] = out[n][j];
        }
    }
    // The state behind the chunk.  What the chunk adds is summed by itself and meets the state in one
    // multiply-add: the tensor cores cut off what a sum of theirs cannot hold, and onto the state itself
    // they would do so a dozen times a chunk.
    constexpr int TURN = HALF % 2 == 0 ? 2 : 1;      // steps of key coordinates side by side
#pragma unroll
    for (int n0 = 0; n0 < HALF; n0 += TURN) {
      float added[2 * TURN][4];
#pragma unroll
      for (int n = 0; n < 2 * TURN; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) added[n][j] = 0.0f;
      uint32_t b[2][TURN][4];      // of a step of tokens, asked for while the products of the one before run
      auto keys_of = [&](int step, int slot) {
#pragma unroll
        for (int n = 0; n < TURN; ++n)
          hx_ldmatrix_x4_trans(b[slot][n], keys + key_lane + 2 * (16 * step * STRIDE + 16 * (n0 + n)));
      };
      auto added_by = [&](const uint32_t (&ut)[4], int slot) {
#pragma unroll
        for (int n = 0; n < TURN; ++n) {
          hx_mma_bf16(added[2 * n], ut, b[slot][n][0], b[slot][n][1]);
          hx_mma_bf16(added[2 * n + 1], ut, b[slot][n][2], b[slot][n][3]);
        }
      };
      keys_of(0, 0);
#pragma unroll
      for (int step = 0; step < CHUNK / 16; ++step) {
        keys_of((step + 1) % (CHUNK / 16), (step + 1) & 1);
        added_by(u2[step], step & 1);
        added_by(u1[step], step & 1);
      }
#pragma unroll
      for (int step = 0; step < CHUNK / 16; ++step) {
        if (step + 1 < CHUNK / 16) keys_of(step + 1, (step + 1) & 1);
        added_by(u0[step], step & 1);
      }
#pragma unroll
      for (int n = 0; n < 2 * TURN; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) S[2 * n0 + n][j] = fmaf(total, S[2 * n0 + n][j], added[n][j]);
    }
  }
#pragma unroll
  for (int n = 0; n < 2 * HALF; ++n)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = my_column + 8 * (j >> 1), d = half_column + 8 * n + pair + (j & 1);
      if (c < a.vdim && d < a.dim)
        s_state[static_cast<size_t>(d & 15) * lanes + c * a.parts + (d >> 4)] = S[n][j];
    }
}

template <int STEPS>
int launch_delta(const DeltaArgs& a, int tiles, cudaStream_t stream) {
  constexpr int shared = DeltaLayout<16 * STEPS>::kBytes;
  const int first = weights_shared(16 * STEPS);
  static std::once_flag once;
  static bool configured = false;
  std::call_once(once, [first] {
    configured = cudaFuncSetAttribute(delta_weights_kernel<STEPS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      first) == cudaSuccess &&
                 cudaFuncSetAttribute(delta_states_kernel<STEPS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      shared) == cudaSuccess;
    if (!configured) cudaGetLastError();
  });
  if (!configured) {
    hx_set_error("hx_delta_chunks: the device refuses %d bytes of shared memory", shared);
    return HX_ERR_LAUNCH;
  }
  hx_launch(delta_weights_kernel<STEPS>, dim3(tiles, a.heads), 128, first, stream, a);
  hx_launch(delta_states_kernel<STEPS>, dim3(a.portions, a.heads, (a.vdim + BLOCK_COLUMNS - 1) / BLOCK_COLUMNS),
            STATES_THREADS, shared, stream, a);
  return HX_OK;
}

}  // namespace

// 1: heads of these sizes run here (bfloat16); else they take the token-by-token scan.
HX_API int hx_delta_chunks_supports(int dim, int vdim) {
  return dim > 0 && vdim > 0 && dim % 8 == 0 && vdim % 8 == 0 && dim <= 128 ? 1 : 0;
}

// Bytes of scratch for a step of `tokens` tokens.
HX_API long long hx_delta_chunks_scratch(int heads, int tokens) {
  return static_cast<long long>(heads) * tokens * (2 * WEIGHT_COLUMNS + 16 + 4);
}

// See the head of this file.  q, k [tokens, qk_heads * dim] and v [tokens, heads * vdim] bfloat16
// rows on 16 bytes; decay_in, beta_in, a_log, dt_bias, fixed_decay_m1, the scales, the state and o
// as for hx_linear_state_scan with its delta rule and without a rotation.  scratch:
// hx_delta_chunks_scratch bytes on 16 bytes.  tiles: at least the chunks of 64 tokens in the step,
// counted request by request.
// Requests that bring fewer than min_query_len tokens are left alone (hx_linear_state_scan_below takes
// them); portions: how many bring as many, tiles: the chunks of those.  status: the device status word, or
// null; a wait for a chunk's rows that runs out (after `polls` polls) leaves NaN in the outputs from there on
// besides, and the portion's state as it was.
HX_API int hx_delta_chunks_limited(const void* q, int ld_q, const void* k, int ld_k, const void* v, int ld_v,
                                const void* decay_in, const void* beta_in, int ld_gates,
                                const float* a_log, const float* dt_bias, const float* fixed_decay_m1,
                                int unit_norm, float unit_eps, float q_scale, float k_scale,
                                void* scratch, float* state, long long state_stride, int head_stride,
                                float* o, const int* request_start, const int* request_slot,
                                int requests, int tokens, int tiles, int heads, int qk_heads, int dim,
                                int vdim, int min_query_len, int portions, int* status, unsigned polls,
                                cudaStream_t stream) {
  HX_REQUIRE(hx_delta_chunks_supports(dim, vdim), "hx_delta_chunks: heads of %d by %d are not supported",
             dim, vdim);
  HX_REQUIRE(requests >= 0 && tokens >= requests && min_query_len > 0 && portions >= 0 &&
                 portions <= requests && tiles >= portions && heads > 0 && heads <= 65535 &&
                 qk_heads > 0 && heads % qk_heads == 0,
             "hx_delta_chunks: bad sizes");
  HX_REQUIRE(ld_q % 8 == 0 && ld_k % 8 == 0 && ld_v % 8 == 0 && ld_q >= qk_heads * dim &&
                 ld_k >= qk_heads * dim && ld_v >= heads * vdim && ld_gates >= heads,
             "hx_delta_chunks: bad strides");
  HX_REQUIRE(((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) |
               reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(scratch)) & 15) == 0,
             "hx_delta_chunks: rows are not 16-byte aligned");
  HX_REQUIRE(beta_in != nullptr && scratch != nullptr &&
                 (decay_in != nullptr ? (a_log != nullptr && dt_bias != nullptr) : fixed_decay_m1 != nullptr),
             "hx_delta_chunks: gates missing");
  HX_REQUIRE(head_stride >= state_floats(vdim, dim), "hx_delta_chunks: a head's state takes %d floats, not %d",
             state_floats(vdim, dim), head_stride);
  if (portions == 0) return HX_OK;
  const size_t rows = static_cast<size_t>(heads) * tokens;
  float4* factors = static_cast<float4*>(scratch);
  __nv_bfloat16* weights = reinterpret_cast<__nv_bfloat16*>(factors + rows);
  float* total = reinterpret_cast<float*>(weights + rows * WEIGHT_COLUMNS);
  const DeltaArgs a{static_cast<const __nv_bfloat16*>(q), static_cast<const __nv_bfloat16*>(k),
                    static_cast<const __nv_bfloat16*>(v), ld_q, ld_k, ld_v,
                    static_cast<const __nv_bfloat16*>(decay_in), static_cast<const __nv_bfloat16*>(beta_in),
                    ld_gates, a_log, dt_bias, fixed_decay_m1, unit_norm, unit_eps, q_scale, k_scale, weights,
                    factors, total, tokens, state, state_stride, head_stride, o, request_start, request_slot,
                    requests, heads, qk_heads, dim, vdim, parts_for(dim), min_query_len,
                    portions, status, polls};
  int rc;
  switch ((dim + 15) / 16) {
    case 1: case 2: rc = launch_delta<2>(a, tiles, stream); break;
    case 3: case 4: rc = launch_delta<4>(a, tiles, stream); break;
    case 5: case 6: rc = launch_delta<6>(a, tiles, stream); break;
    default: rc = launch_delta<8>(a, tiles, stream); break;
  }
  if (rc != HX_OK) return rc;
  hx_count_launches(1);
  HX_CHECK_LAUNCH("hx_delta_chunks");
  return HX_OK;
}

HX_API int hx_delta_chunks_checked(const void* q, int ld_q, const void* k, int ld_k, const void* v, int ld_v,
                                const void* decay_in, const void* beta_in, int ld_gates,
                                const float* a_log, const float* dt_bias, const float* fixed_decay_m1,
                                int unit_norm, float unit_eps, float q_scale, float k_scale,
                                void* scratch, float* state, long long state_stride, int head_stride,
                                float* o, const int* request_start, const int* request_slot,
                                int requests, int tokens, int tiles, int heads, int qk_heads, int dim,
                                int vdim, int min_query_len, int portions, int* status,
                                cudaStream_t stream) {
  return hx_delta_chunks_limited(q, ld_q, k, ld_k, v, ld_v, decay_in, beta_in, ld_gates, a_log, dt_bias,
                                 fixed_decay_m1, unit_norm, unit_eps, q_scale, k_scale, scratch, state, state_stride,
                                 head_stride, o, request_start, request_slot, requests, tokens, tiles, heads,
                                 qk_heads, dim, vdim, min_query_len, portions, status, WAIT_LIMIT, stream);
}

HX_API int hx_delta_chunks_from(const void* q, int ld_q, const void* k, int ld_k, const void* v, int ld_v,
                                const void* decay_in, const void* beta_in, int ld_gates,
                                const float* a_log, const float* dt_bias, const float* fixed_decay_m1,
                                int unit_norm, float unit_eps, float q_scale, float k_scale,
                                void* scratch, float* state, long long state_stride, int head_stride,
                                float* o, const int* request_start, const int* request_slot,
                                int requests, int tokens, int tiles, int heads, int qk_heads, int dim,
                                int vdim, int min_query_len, int portions, cudaStream_t stream) {
  return hx_delta_chunks_checked(q, ld_q, k, ld_k, v, ld_v, decay_in, beta_in, ld_gates, a_log, dt_bias,
                                 fixed_decay_m1, unit_norm, unit_eps, q_scale, k_scale, scratch, state, state_stride,
                                 head_stride, o, request_start, request_slot, requests, tokens, tiles, heads,
                                 qk_heads, dim, vdim, min_query_len, portions, nullptr, stream);
}

// Every request of the step.
HX_API int hx_delta_chunks(const void* q, int ld_q, const void* k, int ld_k, const void* v, int ld_v,
                           const void* decay_in, const void* beta_in, int ld_gates,
                           const float* a_log, const float* dt_bias, const float* fixed_decay_m1,
                           int unit_norm, float unit_eps, float q_scale, float k_scale,
                           void* scratch, float* state, long long state_stride, int head_stride,
                           float* o, const int* request_start, const int* request_slot,
                           int requests, int tokens, int tiles, int heads, int qk_heads, int dim,
                           int vdim, cudaStream_t stream) {
  return hx_delta_chunks_from(q, ld_q, k, ld_k, v, ld_v, decay_in, beta_in, ld_gates, a_log, dt_bias, fixed_decay_m1,
                              unit_norm, unit_eps, q_scale, k_scale, scratch, state, state_stride, head_stride, o,
                              request_start, request_slot, requests, tokens, tiles, heads, qk_heads, dim, vdim, 1,
                              requests, stream);
}
