// The true 32-bit matrix product: float32 operands, one fused multiply-add chain per output over k ascending, on
// the CUDA cores. No tensor cores, no reduced-precision mode, no split of the reduction, so an output's bits depend
// only on its own row of A and row of W: not on M, on the tile it falls in, or on what else is in the batch.
#include "gemm_common.cuh"

namespace {
__device__ __forceinline__ void cp_async_f4(float* smem, const float* gmem, bool ok) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  int bytes = ok ? 16 : 0;  // (a copy of no bytes fills the 16 bytes with zeros)
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}

// ---- tiles of 64 x 64 and 32 x 32 outputs, 4 x 4 of them a thread ----------------------------------------------------
// For products that have too few tiles of 128 x 128 (below) for the device. Bound by reads of shared memory (a warp's
// 16-byte read takes four cycles whoever shares it, which 4 x 4 outputs a thread hide half of the multiply-adds under:
// about 37 TFLOP/s), so nothing else is put there: rows of A and W arrive as they lie (k innermost, by cp.async,
// STAGES - 1 steps of 32 values ahead), a thread reads four k of a row at a time, and its rows and columns are TILE / 4
// apart, which keeps the reads free of bank conflicts.
// Microseconds before (128 x 128 tiles, or 64 x 64 with one step of 16 values ahead for up to 64 rows) and now:
// 2048 x 576 x 576 71 -> 43, 2048 x 576 x 1536 171 -> 98, 512 x 576 x 1536 167 -> 40, 32 x 576 x 1536 104 -> 31.
constexpr int DEPTH = 32, TLD = DEPTH + 4;

template <int EPI, int TILE, int STAGES, int BLOCKS>
__global__ void __launch_bounds__(TILE * TILE / 16, BLOCKS) gemm_f32_tile_kernel(
    void* __restrict__ c, const float* __restrict__ a, const float* __restrict__ w, int M, int N, int K) {
  constexpr int PER = 4, T = TILE * TILE / (PER * PER), APART = TILE / PER, STAGE = 2 * TILE * TLD;
  constexpr int COPIES = 2 * TILE * (DEPTH / 4) / T;
  static_assert(TILE % (T / 8) == 0, "a copy is A's or W's for the whole block");
  extern __shared__ __align__(16) float ring[];  // [STAGES][rows of A, then rows of W][TLD]
  int tid = threadIdx.x, tx = tid % APART, ty = tid / APART;  // rows ty + i * APART, columns tx + j * APART
  int m0 = blockIdx.y * TILE, n0 = blockIdx.x * TILE;
  int tiles = (K + DEPTH - 1) / DEPTH;
  auto ask = [&](int t) {
    float* stage = ring + (t % STAGES) * STAGE;
    int k = t * DEPTH + (tid & 7) * 4;
#pragma unroll
    for (int i = 0; i < COPIES; ++i) {
      int r = (tid >> 3) + i * (T / 8);
      bool from_a = i * (T / 8) < TILE;
      int row = from_a ? m0 + r : n0 + r - TILE;
      bool ok = k < K && row < (from_a ? M : N);
      const float* base = from_a ? a : w;
      cp_async_f4(stage + r * TLD + (tid & 7) * 4, ok ? base + (size_t)row * K + k : base, ok);
    }
  };
  auto close = [] { asm volatile("cp.async.commit_group;\n" ::); };
  float acc[PER][PER];
#pragma unroll
  for (int i = 0; i < PER; ++i)
#pragma unroll
    for (int j = 0; j < PER; ++j) acc[i][j] = 0.f;
  for (int t = 0; t < STAGES - 1; ++t) {
    if (t < tiles) ask(t);
    close();
  }
  for (int t = 0; t < tiles; ++t) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
    __syncthreads();  // (this stage has arrived for everybody, and everybody is done with the one before it)
    if (t + STAGES - 1 < tiles) ask(t + STAGES - 1);
    close();
    const float* rows = ring + (t % STAGES) * STAGE + ty * TLD;
    const float* cols = ring + (t % STAGES) * STAGE + (TILE + tx) * TLD;
#pragma unroll
    for (int k = 0; k < DEPTH; k += 4) {
      float4 wv[PER];
#pragma unroll
      for (int j = 0; j < PER; ++j) wv[j] = *(const float4*)(cols + j * APART * TLD + k);
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        float4 av = *(const float4*)(rows + i * APART * TLD + k);
#pragma unroll
        for (int j = 0; j < PER; ++j) acc[i][j] = fmaf(av.x, wv[j].x, acc[i][j]);
#pragma unroll
        for (int j = 0; j < PER; ++j) acc[i][j] = fmaf(av.y, wv[j].y, acc[i][j]);
#pragma unroll
        for (int j = 0; j < PER; ++j) acc[i][j] = fmaf(av.z, wv[j].z, acc[i][j]);
#pragma unroll
        for (int j = 0; j < PER; ++j) acc[i][j] = fmaf(av.w, wv[j].w, acc[i][j]);
      }
    }
  }
  // (columns are stored by the lane that has the even one: neighbouring columns lie in neighbouring lanes)
#pragma unroll
  for (int i = 0; i < PER; ++i)
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      float other = __shfl_down_sync(0xffffffffu, acc[i][j], 1);
      if (!(tx & 1)) epilogue_pair<EPI, float>(c, m0 + ty + i * APART, n0 + tx + j * APART, M, N, acc[i][j], other);
    }
}

template <int EPI, int TILE, int STAGES, int BLOCKS>
int launch_tile(void* c, const float* a, const float* w, int M, int N, int K, cudaStream_t stream) {
  auto kernel = gemm_f32_tile_kernel<EPI, TILE, STAGES, BLOCKS>;
  constexpr int smem = STAGES * 2 * TILE * TLD * (int)sizeof(float);
  static std::atomic<unsigned long long> allowed{0};
  if (!dllm_allow_shared((const void*)kernel, smem, allowed)) return DLLM_LAUNCH_FAILED;
  dim3 grid((N + TILE - 1) / TILE, (M + TILE - 1) / TILE);
  if (grid.y > 65535) return DLLM_UNSUPPORTED_SIZE;
  kernel<<<grid, TILE * TILE / 16, smem, stream>>>(c, a, w, M, N, K);
  return dllm_launch_status();
}

// ---- tiles of 128 x 128 outputs, 8 x 8 of them a thread ----------------------------------------------------------------
// Two stages of shared memory; the next k tile travels from global memory into registers while this one is multiplied.
// A thread's 64 outputs are 2 x 2 groups of 4 x 4, so its shared-memory reads are four 16-byte loads per k. Every output is
// one chain over k ascending from zero here too: the same bits. Bounds for one block a multiprocessor: with bounds for two, with
// packed multiply-adds (two outputs an instruction), or both, a round of one tile each is slower. 512 x 4096 x
// 4096 (128 tiles): 396 us (43 TFLOP/s); bounds for two 458, packed 483, both 497. 2048 x 3072 x 576 (384 tiles): 176; 187,
// 198, 179. 4096 x 4096 x 2048 (1,024 tiles): 1,397; 1,468, 1,665, 1,407. Only very many tiles gain by both (49152 columns,
// 6,144 tiles: 2,437 against 2,352). 8 x 16 outputs a thread: 186 at 2048 x 3072 x 576; rows as they lie with cp.async, as
// for the smaller tiles: 240.
constexpr int WM = 128, WN = 128, WK = 16;

template <int EPI>
__global__ void __launch_bounds__(256, 1) gemm_f32_wide_kernel(
    void* __restrict__ c, const float* __restrict__ a, const float* __restrict__ w, int M, int N, int K) {
  __shared__ __align__(16) float as[2][WK][WM + 4];
  __shared__ __align__(16) float ws[2][WK][WN + 4];
  int tid = threadIdx.x;
  int tx = tid & 15, ty = tid >> 4;             // rows ty * 4 + {0..3, 64..67}, columns likewise
  int m0 = blockIdx.y * WM, n0 = blockIdx.x * WN;
  int lrow = tid >> 2, lk = (tid & 3) * 4;      // a thread fetches rows lrow and lrow + 64, k lk .. lk + 3
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  float4 va[2], vw[2];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      int r = lrow + 64 * h;
      va[h] = vw[h] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (m0 + r < M && k0 + lk < K) va[h] = *(const float4*)(a + (size_t)(m0 + r) * K + k0 + lk);
      if (n0 + r < N && k0 + lk < K) vw[h] = *(const float4*)(w + (size_t)(n0 + r) * K + k0 + lk);
    }
  };
  auto stash = [&](int buf) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      int r = lrow + 64 * h;
      as[buf][lk + 0][r] = va[h].x; as[buf][lk + 1][r] = va[h].y; as[buf][lk + 2][r] = va[h].z; as[buf][lk + 3][r] = va[h].w;
      ws[buf][lk + 0][r] = vw[h].x; ws[buf][lk + 1][r] = vw[h].y; ws[buf][lk + 2][r] = vw[h].z; ws[buf][lk + 3][r] = vw[h].w;
    }
  };
  fetch(0);
  stash(0);
  __syncthreads();
  int tiles = (K + WK - 1) / WK;
  for (int t = 0; t < tiles; ++t) {
    int buf = t & 1;
    if (t + 1 < tiles) fetch((t + 1) * WK);
#pragma unroll
    for (int k = 0; k < WK; ++k) {
      float4 a0 = *(const float4*)&as[buf][k][ty * 4], a1 = *(const float4*)&as[buf][k][64 + ty * 4];
      float4 w0 = *(const float4*)&ws[buf][k][tx * 4], w1 = *(const float4*)&ws[buf][k][64 + tx * 4];
      float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      float wv[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
    }
    if (t + 1 < tiles) {
      stash(buf ^ 1);  // (the other stage was last read before the barrier that ended the step before)
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    int m = m0 + (i >> 2) * 64 + ty * 4 + (i & 3);
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      int n = n0 + (j >> 2) * 64 + tx * 4 + (j & 3);
      epilogue_pair<EPI, float>(c, m, n, M, N, acc[i][j], acc[i][j + 1]);
    }
  }
}

template <int EPI>
int launch_wide(void* c, const float* a, const float* w, int M, int N, int K, cudaStream_t stream) {
  dim3 grid((N + WN - 1) / WN, (M + WM - 1) / WM);
  if (grid.y > 65535) return DLLM_UNSUPPORTED_SIZE;
  gemm_f32_wide_kernel<EPI><<<grid, 256, 0, stream>>>(c, a, w, M, N, K);
  return dllm_launch_status();
}

// Which tile: the fewest microseconds by rounds of one tile per multiprocessor. Whole launches of K = 576, last rounds that
// are partly empty among them, are fitted by 57 us a round of 128 x 128, 20 of 64 x 64 and, while few rounds are needed,
// 8 of 32 x 32, plus a few to begin; all grow alike with K. So full devices take the large tile, and a product too small
// for it (2048 x 576: 80 tiles of 128 x 128 for 148 multiprocessors) one that spreads over all of them.
// Launched without programmatic dependence: blocks of the next kernel that wait on a multiprocessor for this one make the
// launch after it spread unevenly (2048 x 576 x 576 back to back: 110 us instead of 72).
template <int EPI>
int launch_tiles(void* c, const float* a, const float* w, int M, int N, int K, cudaStream_t stream) {
  auto rounds = [&](int tile) {
    long long tiles = (long long)((M + tile - 1) / tile) * ((N + tile - 1) / tile);
    return (tiles + 147) / 148;
  };
  auto fits = [&](int tile) { return (M + tile - 1) / tile <= 65535; };  // (rows of tiles are the grid's second dimension)
  long long wide = 57 * rounds(128) + 4, middle = 20 * rounds(64) + 2, small = 8 * rounds(32) + 2;
  if (!fits(64) || (wide <= middle && (wide <= small || !fits(32)))) return launch_wide<EPI>(c, a, w, M, N, K, stream);
  if (!fits(32) || middle <= small) return launch_tile<EPI, 64, 4, 2>(c, a, w, M, N, K, stream);
  return launch_tile<EPI, 32, 6, 4>(c, a, w, M, N, K, stream);
}

// ---- and for a few rows (decode steps): the reduction streamed through a ring of stages -----------------------------
// One chain of fused multiply-adds per output over k ascending from zero, as above: a token's bits are the ones it gets
// in a long prompt. So a product cannot be faster than its K dependent multiply-adds (four cycles each: 3.1 us for
// K = 1536), and the split is made to come close to that: a block takes COLS columns, few enough that the columns
// spread over the whole device, a thread PER rows of one column, and W and A arrive by cp.async STAGES - 1 stages of
// DEPTH values ahead of the chain. W's first stages are asked for before the kernel in front has finished.
// Eight rows, 576 columns: K = 576 12.0 -> 3.3 us, K = 1536 27.5 -> 6.1 us (before: 32 columns a block, three stages of
// 32 values, which was 18 blocks for the device and a round trip to L2 every other stage); 49152 x 576 52 -> 28.5 us.
constexpr int SM_ROWS = 16;

template <int EPI, int COLS, int ROWS, int PER, int DEPTH, int STAGES>
__global__ void __launch_bounds__(COLS * ROWS / PER) gemm_f32_small_kernel(void* __restrict__ c, const float* __restrict__ a,
                                                                           const float* __restrict__ w, int M, int N,
                                                                           int K) {
  constexpr int T = COLS * ROWS / PER, LD = DEPTH + 4, PIECES = DEPTH / 4, STAGE = (COLS + ROWS) * LD;
  static_assert(T % 32 == 0 && (COLS * PIECES) % T == 0 && (ROWS * PIECES) % T == 0 && COLS % 2 == 0, "whole warps and copies");
  extern __shared__ __align__(16) float ring[];  // [STAGES][COLS of W, then ROWS of A][LD]
  int tid = threadIdx.x, col = tid % COLS, row0 = tid / COLS;  // rows row0 + i * (ROWS / PER)
  int n0 = blockIdx.x * COLS;
  int tiles = (K + DEPTH - 1) / DEPTH;
  auto ask_w = [&](int t) {
    float* stage = ring + (t % STAGES) * STAGE;
#pragma unroll
    for (int i = 0; i < COLS * PIECES / T; ++i) {
      int at = tid + i * T, r = at / PIECES, k = (at % PIECES) * 4;
      bool ok = n0 + r < N && t * DEPTH + k < K;
      cp_async_f4(stage + r * LD + k, ok ? w + (size_t)(n0 + r) * K + t * DEPTH + k : w, ok);
    }
  };
  auto ask_a = [&](int t) {
    float* stage = ring + (t % STAGES) * STAGE + COLS * LD;
#pragma unroll
    for (int i = 0; i < ROWS * PIECES / T; ++i) {
      int at = tid + i * T, r = at / PIECES, k = (at % PIECES) * 4;
      bool ok = r < M && t * DEPTH + k < K;
      cp_async_f4(stage + r * LD + k, ok ? a + (size_t)r * K + t * DEPTH + k : a, ok);
    }
  };
  auto close = [] { asm volatile("cp.async.commit_group;\n" ::); };
  for (int t = 0; t < min(tiles, STAGES - 1); ++t) ask_w(t);
  pdl_wait();
  // (the next kernel starts here and not with this one: those behind it would all ask for their weights and wait beside it.
  // Eight sequences of the 135M shape in float32, with the same in the attention of single tokens, 63.8 -> 56.1 ms a call)
  pdl_launch_dependents();
  for (int t = 0; t < STAGES - 1; ++t) {
    if (t < tiles) ask_a(t);
    close();
  }
  float acc[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) acc[i] = 0.f;
  for (int t = 0; t < tiles; ++t) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
    __syncthreads();  // (this stage has arrived for everybody, and everybody is done with the one before it)
    if (t + STAGES - 1 < tiles) {
      ask_w(t + STAGES - 1);
      ask_a(t + STAGES - 1);
    }
    close();
    const float* stage = ring + (t % STAGES) * STAGE;
    const float* mine = stage + col * LD;
    const float* rows = stage + (COLS + row0) * LD;
    // (the values of the next GROUP pieces are on their way from shared memory while these are multiplied; the chains of
    // a thread go side by side, since a warp issues in order)
    constexpr int GROUP = PER == 1 ? 4 : 2;
    float4 wv[2][GROUP], av[2][GROUP][PER];
    auto load = [&](int slot, int k) {
#pragma unroll
      for (int g = 0; g < GROUP; ++g) {
        wv[slot][g] = *(const float4*)(mine + k + 4 * g);
#pragma unroll
        for (int i = 0; i < PER; ++i) av[slot][g][i] = *(const float4*)(rows + i * (ROWS / PER) * LD + k + 4 * g);
      }
    };
    load(0, 0);
#pragma unroll
    for (int k = 0; k < DEPTH; k += 4 * GROUP) {
      int slot = (k / (4 * GROUP)) & 1;
      if (k + 4 * GROUP < DEPTH) load(slot ^ 1, k + 4 * GROUP);
#pragma unroll
      for (int g = 0; g < GROUP; ++g) {
#pragma unroll
        for (int i = 0; i < PER; ++i) acc[i] = fmaf(av[slot][g][i].x, wv[slot][g].x, acc[i]);
#pragma unroll
        for (int i = 0; i < PER; ++i) acc[i] = fmaf(av[slot][g][i].y, wv[slot][g].y, acc[i]);
#pragma unroll
        for (int i = 0; i < PER; ++i) acc[i] = fmaf(av[slot][g][i].z, wv[slot][g].z, acc[i]);
#pragma unroll
        for (int i = 0; i < PER; ++i) acc[i] = fmaf(av[slot][g][i].w, wv[slot][g].w, acc[i]);
      }
    }
  }
  // pairs of columns are stored by the even lane (the SwiGLU epilogue needs gate and up together)
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    float other = __shfl_down_sync(0xffffffffu, acc[i], 1);
    if (!(col & 1)) epilogue_pair<EPI, float>(c, row0 + i * (ROWS / PER), n0 + col, M, N, acc[i], other);
  }
}

template <int EPI, int COLS, int ROWS, int PER, int DEPTH, int STAGES>
int launch_small(void* c, const float* a, const float* w, int M, int N, int K, cudaStream_t stream) {
  auto kernel = gemm_f32_small_kernel<EPI, COLS, ROWS, PER, DEPTH, STAGES>;
  constexpr int smem = STAGES * (COLS + ROWS) * (DEPTH + 4) * (int)sizeof(float);
  static std::atomic<unsigned long long> allowed{0};
  if (!dllm_allow_shared((const void*)kernel, smem, allowed)) return DLLM_LAUNCH_FAILED;
  return dllm_launch_pdl(kernel, dim3((N + COLS - 1) / COLS), dim3(COLS * ROWS / PER), smem, stream, c, a, w, M, N, K);
}

// How the columns are split, by what was fastest with eight rows (all of it bounded by latency, so by how the columns
// spread and how many chains a thread keeps going, not by the bytes):
//   up to 1,184 columns   8 a block: 148 blocks and more (576 x 1536: 6.1 us; four columns 6.5, sixteen 9.0 to 11.5);
//   up to 4,736           16 a block, two rows a thread, ten short stages (3072 x 576: 5.8 us; 8 columns 8.3, 32 6.7);
//   up to 18,944          16 a block, four rows a thread (8192 x 2048: 25 us; two rows 30 to 35, 32 columns 27 to 35);
//   more                  64 a block, eight rows a thread, which reads shared memory least (49152 x 576: 28.5 us, 4.0 TB/s;
//                         16 columns 40, 32 columns 32).
template <int EPI, int ROWS>
int launch_small_by_columns(void* c, const float* a, const float* w, int M, int N, int K, cudaStream_t stream) {
  if (N <= 8 * 148) return launch_small<EPI, 8, ROWS, ROWS / 8, 128, 6>(c, a, w, M, N, K, stream);
  if (N <= 32 * 148) return launch_small<EPI, 16, ROWS, 2, 64, 10>(c, a, w, M, N, K, stream);
  if (N <= 128 * 148) return launch_small<EPI, 16, ROWS, 4, 128, 4>(c, a, w, M, N, K, stream);
  return launch_small<EPI, 64, ROWS, 8, 64, 3>(c, a, w, M, N, K, stream);
}

template <int EPI>
int launch_small_by_rows(void* c, const float* a, const float* w, int M, int N, int K, cudaStream_t stream) {
  return M <= 8 ? launch_small_by_columns<EPI, 8>(c, a, w, M, N, K, stream)
                : launch_small_by_columns<EPI, 16>(c, a, w, M, N, K, stream);
}
}  // namespace

// C = A[M,K] * W[N,K]^T in float32; K a multiple of 4 (16-byte rows); N even for the SwiGLU epilogue (column pairs).
// Up to 16 rows take the kernel that streams the reduction, more the tiles that `launch_tiles` chooses; all give an
// output the same bits.
DLLM_EXPORT int dllm_gemm_f32(void* c, const float* a, const float* w, int M, int N, int K, int epilogue,
                              cudaStream_t stream) {
  if (M <= 0 || N <= 0) return DLLM_OK;
  if (K <= 0 || (K & 3) || ((N & 1) && epilogue == EPI_SWIGLU)) return DLLM_UNSUPPORTED_SIZE;
  if (epilogue < 0 || epilogue > EPI_SWIGLU) return DLLM_BAD_ARGUMENT;
  if (epilogue == EPI_STORE_T) epilogue = EPI_STORE_F32;  // (the activation type is float32 here)
  bool few = M <= SM_ROWS;
  switch (epilogue) {
    case EPI_STORE_F32: return (few ? launch_small_by_rows<EPI_STORE_F32> : launch_tiles<EPI_STORE_F32>)(c, a, w, M, N, K, stream);
    case EPI_RESIDUAL: return (few ? launch_small_by_rows<EPI_RESIDUAL> : launch_tiles<EPI_RESIDUAL>)(c, a, w, M, N, K, stream);
    default: return (few ? launch_small_by_rows<EPI_SWIGLU> : launch_tiles<EPI_SWIGLU>)(c, a, w, M, N, K, stream);
  }
}
